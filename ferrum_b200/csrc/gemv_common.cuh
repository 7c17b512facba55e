// Pieces shared by the decode / verify projection kernels (gemv_i8.cu, gemv_nt.cu): programmatic dependent
// launch, load helpers, the warp-level integer MMAs, the 16-bit quantisation of eight activations, and the
// device side of the fused row-shard exchange.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "internal.h"

namespace fqk {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Eight codebook values of the IQ4 formats (iq4_value in blocks.cuh) for the eight 4-bit indices of `n`: nibble i of the
// low half -> byte i of .x, of the high half -> byte i of .y.  Three bits of an index select from each half of the
// codebook with a byte permute; the fourth then picks the half, again by a permute.
__device__ __forceinline__ uint2 iq4_lookup8(uint32_t n) {
    constexpr uint32_t T0 = 0xBFAD9881u, T1 = 0xF6EADDCFu, T2 = 0x26190D01u, T3 = 0x71594535u; // entries 0-3, 4-7, 8-11, 12-15
    const uint32_t low3 = n & 0x77777777u, half = ((n >> 1) & 0x44444444u) | 0x32103210u; // selector 4 + i takes byte i of the upper half's value
    auto pick = [&](uint32_t sel, uint32_t h) { return __byte_perm(__byte_perm(T0, T1, sel), __byte_perm(T2, T3, sel), h); };
    return make_uint2(pick(low3, half), pick(low3 >> 16, half >> 16)); // a permute reads the low 16 bits of its selector
}

// u8 (weights) x s8 (activations), 16 rows x 8 columns x 32 k.
__device__ __forceinline__ void mma_u8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// s8 x s8, 16 rows x 8 columns x 16 k.
__device__ __forceinline__ void mma_s8s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0));
}

// Prepared activations: written by the kernel before this one (which may still run when this grid
// starts), so ordinary coherent loads after `pdl_wait`; volatile so guarded loads are not speculated.
__device__ __forceinline__ uint4 ldx128(const void *p) {
    uint4 r;
    asm volatile("ld.global.ca.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ uint32_t ldx32(const void *p) {
    uint32_t r;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(r) : "l"(p));
    return r;
}
// Weights: immutable, read once -> read-only path, no L1 allocation.
__device__ __forceinline__ uint4 ldw128(const void *p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ uint2 ldw64(const void *p) {
    uint2 r;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ uint32_t ldw16(const void *p) {
    uint16_t r;
    asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(r) : "l"(p));
    return r;
}
// Weights of which one thread takes 4 bytes at a time: the rest of the 32-byte sector is asked for by a later
// instruction of the same warp, so the line is kept in L1.
__device__ __forceinline__ uint32_t ldw32_keep(const void *p) {
    uint32_t r;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(r) : "l"(p));
    return r;
}
__device__ __forceinline__ uint32_t lop3_select(uint32_t a, uint32_t b, uint32_t mask) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(r) : "r"(a), "r"(b), "r"(mask)); // (a & mask) | (b & ~mask)
    return r;
}
__device__ __forceinline__ uint32_t lop3_and_xor(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); // (a & b) ^ c
    return r;
}
// Byte i of w, zero- or sign-extended (one PRMT each; a selector nibble with its top bit set replicates the
// sign of the byte it names).
__device__ __forceinline__ int byte_u(uint32_t w, int i) { return (int)__byte_perm(w, 0u, 0x4440u + (uint32_t)i); }
__device__ __forceinline__ int byte_s(uint32_t w, int i) {
    int r;
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(r) : "r"(w), "r"(0x8880u + (uint32_t)i * 0x1111u));
    return r;
}
__device__ __forceinline__ uint32_t word_of(const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// Eight activations of one lane as 31-bit integers x' = round(x * 2^e) in four signed base-256 digits, p[0] the most
// significant, 2^e the largest power of two with max|x| * 2^e <= 0x7F7F7F00 over the superblock, up to 2^149: a step is at
// most 2^-30 of the superblock's largest value, and never more than fp32's own smallest, so less is dropped than the
// products and sums of an fp32 dot product round off (24 bits of the largest value were not enough: 1.3 to 7 times the
// error of the fp32 kernels on rows of 1024..2304 values, more where a superblock has an outlier).
// inv = 2^-e.  A superblock with an infinity and no NaN: inv = +infinity and p[0] holds the sign (+-1) of every infinity,
// 0 for the rest; with a NaN: inv is NaN.
struct Quant8Wide {
    uint32_t p[4][2]; // values 0-3 and 4-7, one per byte
    float inv;
};
// The scale of a group of values from amax, the largest |value| that is no NaN, and whether one is.
struct WideScale {
    float s0, s1, inv; // 2^e may be beyond fp32: two factors
    bool finite, nan;
    __device__ __forceinline__ WideScale(float amax, bool nan_) : nan(nan_) {
        finite = amax < INFINITY && !nan;
        // amax = 1.f * 2^ex: e = 30 - ex, one less where the mantissa is above that of 0x7F7F7F00; a subnormal amax ends at 149.
        const uint32_t bits = __float_as_uint(amax);
        int e = 0;
        if (amax > 0.f && finite) e = min(149, 157 - (int)(bits >> 23) - ((bits & 0x7FFFFFu) > 0x7EFEFEu));
        inv = e > 126 ? __uint_as_float(1u << (149 - e)) : __uint_as_float((uint32_t)(127 - e) << 23);
        if (!finite) inv = nan ? __int_as_float(0x7fc00000) : INFINITY;
        const int e0 = e >> 1;
        s0 = __uint_as_float((uint32_t)(127 + e0) << 23);
        s1 = __uint_as_float((uint32_t)(127 + e - e0) << 23);
    }
    // A value's digits, the most significant in the top byte (adding 0x80 to every digit makes them unsigned).
    __device__ __forceinline__ uint32_t digits(float v) const { return ((uint32_t)__float2int_rn(v * s0 * s1) + 0x80808080u) ^ 0x80808080u; }
    __device__ __forceinline__ uint32_t sign_of_infinity(float v) const { return nan || fabsf(v) < INFINITY ? 0u : v > 0.f ? 0x01000000u : 0xFF000000u; }
};
__device__ __forceinline__ Quant8Wide quantize8_wide(const float (&v)[8]) {
    Quant8Wide q;
    float amax = 0.f;
    bool nan = false;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        amax = fmaxf(amax, fabsf(v[i])); // drops a NaN
        nan |= v[i] != v[i];
    }
    nan = __any_sync(0xffffffffu, nan);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    const WideScale s(amax, nan);
    q.inv = s.inv;
    uint32_t d[8];
#pragma unroll
    for (int i = 0; i < 8; i++) d[i] = s.digits(v[i]);
    if (!s.finite)
#pragma unroll
        for (int i = 0; i < 8; i++) d[i] = s.sign_of_infinity(v[i]);
#pragma unroll
    for (int h = 0; h < 2; h++) { // bytes of four values -> one word per digit
        const uint32_t *x = d + 4 * h;
        const uint32_t low01 = __byte_perm(x[0], x[1], 0x5140), low23 = __byte_perm(x[2], x[3], 0x5140);
        const uint32_t top01 = __byte_perm(x[0], x[1], 0x7362), top23 = __byte_perm(x[2], x[3], 0x7362);
        q.p[3][h] = __byte_perm(low01, low23, 0x5410);
        q.p[2][h] = __byte_perm(low01, low23, 0x7632);
        q.p[1][h] = __byte_perm(top01, top23, 0x5410);
        q.p[0][h] = __byte_perm(top01, top23, 0x7632);
    }
    return q;
}

// Eight activations of one lane (values 8 lane .. 8 lane + 7 of a 256-value superblock handled by one warp) as
// 16-bit integers x' = round(x * s) = 256 hi + lo with both halves signed bytes; s = 2^e is the largest power of
// two with max|x| * s <= 32639 over the superblock (1 when the superblock is all zero or holds a NaN or an
// infinity, in which case `finite` is false and every x' is zero: the caller makes the superblock's factor NaN).
struct Quant8 {
    uint8_t hi[8], lo[8];
    int sum, sum_hi, sum_lo; // over the lane's eight values
    int e;
    bool finite;
};
__device__ __forceinline__ Quant8 quantize8(const float (&v)[8]) {
    Quant8 q;
    float amax = 0.f;
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        amax = fmaxf(amax, fabsf(v[i]));
        bad |= !(fabsf(v[i]) < INFINITY);
    }
    q.finite = __ballot_sync(0xffffffffu, bad) == 0u;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    int e = 0;
    if (amax > 0.f && q.finite) {
        int ex;
        frexpf(amax, &ex);
        e = 15 - ex;
        if (ldexpf(amax, e) > 32639.f) e -= 1;
        e = max(-110, min(110, e));
    }
    q.e = e;
    const float s = ldexpf(1.f, e);
    q.sum = q.sum_hi = q.sum_lo = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        int x = __float2int_rn(fminf(fmaxf(v[i] * s, -32639.f), 32639.f));
        if (!q.finite) x = 0;
        const int h = (x + 128) >> 8, l = x - (h << 8);
        q.hi[i] = (uint8_t)h;
        q.lo[i] = (uint8_t)l;
        q.sum += x;
        q.sum_hi += h;
        q.sum_lo += l;
    }
    return q;
}
// 1 / sqrt(mean(x^2) + eps) of a row of n values (a multiple of 4).  The sum is that of sixteen virtual warps: lane l
// of virtual warp w adds the float4s 32 w + l, + 512, .. in order, a butterfly adds its lanes, and the sixteen are added
// in order.  Whoever computes it -- a block of 16 warps, one of four, a single warp -- gets the same bits, so the
// standalone normalisation and the ones fused into activation preparation agree.  (One warp walking the row in a single
// chain, as this once was, took 15 us on a 5120-value row: 40 dependent loads.)
constexpr uint32_t NORM_WARPS = 16;
__device__ __forceinline__ float norm_square(float ss, const float4 &v) {
    ss = fmaf(v.x, v.x, ss);
    ss = fmaf(v.y, v.y, ss);
    ss = fmaf(v.z, v.z, ss);
    return fmaf(v.w, v.w, ss);
}
__device__ __forceinline__ float norm_butterfly(float ss) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    return ss;
}
// `parts`: the virtual warps the row reaches, where that is known (the others would add zero).
template <uint32_t parts = NORM_WARPS> __device__ __forceinline__ float norm_finish(const float *part, uint32_t n, float eps) {
    float ss = 0.f;
#pragma unroll
    for (uint32_t w = 0; w < parts; w++) ss += part[w];
    return 1.0f / sqrtf(ss / (float)n + eps);
}
// By a block of W warps; `part` holds NORM_WARPS floats of shared memory.  A warp's virtual warps run side by side, so their
// loads are in flight together.  Synchronises.
template <uint32_t W> __device__ __forceinline__ float block_inv_rms(const float *__restrict__ row, uint32_t n, float eps, float *part) {
    constexpr uint32_t PER = NORM_WARPS / W;
    static_assert(PER * W == NORM_WARPS, "virtual warps are dealt out evenly");
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float ss[PER];
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) ss[k] = 0.f;
#pragma unroll 4
    for (uint32_t i = 32 * warp + lane; i < n / 4; i += 32 * NORM_WARPS)
#pragma unroll
        for (uint32_t k = 0; k < PER; k++)
            if (i + 32 * W * k < n / 4) ss[k] = norm_square(ss[k], reinterpret_cast<const float4 *>(row)[i + 32 * W * k]);
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) {
        ss[k] = norm_butterfly(ss[k]);
        if (lane == 0) part[warp + W * k] = ss[k];
    }
    __syncthreads();
    return norm_finish(part, n, eps);
}
// By one warp.
__device__ __forceinline__ float row_inv_rms(const float *__restrict__ row, uint32_t n, float eps, uint32_t lane) {
    float part[NORM_WARPS];
#pragma unroll
    for (uint32_t w = 0; w < NORM_WARPS; w++) part[w] = 0.f;
    for (uint32_t i0 = lane; i0 < n / 4; i0 += 32 * NORM_WARPS)
#pragma unroll
        for (uint32_t w = 0; w < NORM_WARPS; w++)
            if (i0 + 32 * w < n / 4) part[w] = norm_square(part[w], reinterpret_cast<const float4 *>(row)[i0 + 32 * w]);
#pragma unroll
    for (uint32_t w = 0; w < NORM_WARPS; w++) part[w] = norm_butterfly(part[w]);
    return norm_finish(part, n, eps);
}
__device__ __forceinline__ uint32_t pack4(const uint8_t *p) { return p[0] | (p[1] << 8) | (p[2] << 16) | ((uint32_t)p[3] << 24); }

// Row-sharded launches (TpPush, internal.h).  tp_seq: the sequence number of this exchange, read by every block
// once the kernel before has finished.  tp_store: one output value to the mirror of every peer, tagged.
// tp_finish: this block's share of the incoming slots, then the bookkeeping by the last block.  A slot that has
// not arrived after P.wait_ns of wall time makes the block record FQ_ERR_TIMEOUT and stop polling for good (its
// remaining slots are looked at once each), so an absent peer costs one limit per block, not one per slot.
__device__ __forceinline__ uint32_t tp_seq(const TpPush &P) { return *(volatile uint32_t *)P.epoch + 1u; }
__device__ __forceinline__ void tp_store(const TpPush &P, uint32_t seq, const float *dst, float v) {
    const size_t off = (size_t)((const uint8_t *)dst - P.peer[P.rank]);
    for (uint32_t p = 0; p < P.world; p++)
        if (p != P.rank)
            asm volatile("st.global.v2.u32 [%0], {%1, %2};" ::"l"(P.peer[p] + P.mirror_off + 2 * off), "r"(__float_as_uint(v)), "r"(seq) : "memory");
}
__device__ __forceinline__ void tp_finish(const TpPush &P, uint32_t seq) {
    __shared__ uint32_t tp_gave_up;
    const uint32_t blocks = gridDim.x * gridDim.y * gridDim.z, block = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    if (threadIdx.x == 0) tp_gave_up = 0;
    __syncthreads();
    const size_t per_rank = P.covered_bytes / 4, incoming = per_rank * (P.world - 1);
    const size_t lo = incoming * block / blocks, hi = incoming * (block + 1) / blocks;
    uint64_t t0 = 0;
    for (size_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        uint32_t p = (uint32_t)(i / per_rank);
        const size_t j = i % per_rank;
        if (p >= P.rank) p++; // the senders, skipping this rank
        const size_t off = P.slice_off + ((size_t)p - P.rank) * P.slice_bytes + 4 * j; // wraps correctly for p < rank
        const uint8_t *slot = P.peer[P.rank] + P.mirror_off + 2 * off;
        uint32_t v = 0, tag = 0;
        bool arrived = false;
        for (uint32_t n = 0;; n++) {
            asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(v), "=r"(tag) : "l"(slot) : "memory");
            arrived = tag == seq;
            if (arrived || *(volatile uint32_t *)&tp_gave_up) break;
            if (n > 16) {
                __nanosleep(64);
                if (t0 == 0) t0 = global_ns();
                else if ((n & 15u) == 0 && global_ns() - t0 > P.wait_ns) {
                    tp_gave_up = 1u;
                    break;
                }
            }
        }
        if (arrived) *reinterpret_cast<uint32_t *>(P.peer[P.rank] + off) = v;
        else *(volatile int *)P.status = (int)FQ_ERR_TIMEOUT; // the peer never sent: report, do not hang
    }
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(P.counter, 1u) + 1u == blocks) {
        *P.counter = 0;
        *(volatile uint32_t *)P.epoch = seq; // every block has read it by now
    }
}

// ---------------------------------------------------------------- per-warp weight rings
//
// A warp streams the packed superblocks of its 16-row weight tiles through a private ring of stages in shared
// memory with 16-byte asynchronous copies: several superblocks in flight per warp, no registers held, no
// block-wide barrier.  A stage holds one superblock of 16 rows, row r at r * ROW (ROW >= the bytes of a row's
// superblock, padded so that the reads of a kernel's fragment pattern fall on different banks):
//   Q4_K / Q5_K  the 144 / 176 bytes of the block;
//   IQ4          the 128 bytes of nibbles, then the superblock's scales: IQ4_XS 8 bytes d | scales_h | scales_l, IQ4_NL
//                the eight f16 d of its blocks;
//   Q6_K         ql[128] | qh[64] | scales[16] of the device layout (blocks.cuh), and after the 16 rows 4 bytes
//                per row: the aligned word that holds the f16 d of the superblock (its high half for odd b).
// A lane copies the same pieces of every superblock, so their offsets from the tile's first row are worked out
// once per tile (`start_tile`); rows past the end of the matrix read its last row.
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void *smem_dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem_dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int FMT, uint32_t ROW> struct WeightRing {
    static constexpr bool IQ4 = FMT == FQ_IQ4_XS || FMT == FQ_IQ4_NL;
    static constexpr uint32_t SRC = FMT == FQ_Q4_K ? 144 : FMT == FQ_Q5_K ? 176 : IQ4 ? 144 : 208; // bytes copied per row and superblock
    static constexpr uint32_t PER_ROW = SRC / 16;
    static constexpr uint32_t PIECES = 16 * PER_ROW;
    static constexpr int NP = FMT == FQ_Q6_K ? 7 : IQ4 ? 5 : (int)((PIECES + 31) / 32);
    static constexpr uint32_t BYTES = 16 * ROW + (FMT == FQ_Q6_K ? 64 : 0);
    static_assert(ROW >= SRC && ROW % 16 == 0, "stage rows hold a row's superblock and stay 16-byte aligned");
    const uint8_t *base = nullptr;
    uint32_t off[NP];
    // Q6_K: pieces 0..127 are ql (row p / 8), 128..191 qh (row / 4), 192..207 the scales, 208..223 the word with d.
    // IQ4: pieces 0..127 are nibbles (row p / 8), then one piece of scales per row (lanes 0..15).
    __device__ __forceinline__ uint32_t piece_row(int i, uint32_t lane) const {
        const uint32_t p = lane + 32 * i;
        if constexpr (IQ4) return i < 4 ? p / 8 : (lane & 15);
        else if constexpr (FMT != FQ_Q6_K) return p / PER_ROW;
        return i < 4 ? p / 8 : i < 6 ? (p - 128) / 4 : (lane & 15);
    }
    // `first_row`: the tile's first weight row; `last`: index of the matrix's last row relative to it.
    __device__ __forceinline__ void start_tile(const uint8_t *first_row, uint32_t last, uint32_t pitch, uint32_t nblk, uint32_t lane) {
        base = first_row;
#pragma unroll
        for (int i = 0; i < NP; i++) {
            const uint32_t p = lane + 32 * i, r = min(piece_row(i, lane), last);
            uint32_t in_row;
            if constexpr (IQ4) in_row = i < 4 ? 16 * (p % 8) : nblk * 128;
            else if constexpr (FMT != FQ_Q6_K) in_row = 16 * (p % PER_ROW);
            else in_row = i < 4 ? 16 * (p % 8) : i < 6 ? nblk * 128 + 16 * (p % 4) : lane < 16 ? nblk * 192 : nblk * 208;
            off[i] = r * pitch + in_row;
        }
    }
    // Superblock b of the tile into the stage at `dst`.
    __device__ __forceinline__ void issue(uint8_t *dst, uint32_t b, uint32_t lane) const {
#pragma unroll
        for (int i = 0; i < NP; i++) {
            const uint32_t p = lane + 32 * i;
            if constexpr (IQ4) {
                if (i < 4) cp_async16(dst + ROW * (p / 8) + 16 * (p % 8), base + (off[i] + b * 128));
                else if (lane < 16) {
                    if constexpr (FMT == FQ_IQ4_XS) cp_async8(dst + ROW * lane + 128, base + (off[i] + b * 8));
                    else cp_async16(dst + ROW * lane + 128, base + (off[i] + b * 16));
                }
            } else if constexpr (FMT != FQ_Q6_K) {
                if (p < PIECES) cp_async16(dst + ROW * (p / PER_ROW) + 16 * (p % PER_ROW), base + (off[i] + b * SRC));
            } else {
                if (i < 4) cp_async16(dst + ROW * (p / 8) + 16 * (p % 8), base + (off[i] + b * 128));
                else if (i < 6) cp_async16(dst + ROW * ((p - 128) / 4) + 128 + 16 * (p % 4), base + (off[i] + b * 64));
                else if (lane < 16) cp_async16(dst + ROW * lane + 192, base + (off[i] + b * 16));
                else cp_async4(dst + 16 * ROW + 4 * (lane - 16), base + (off[i] + (b & ~1u) * 2)); // the aligned 4 bytes that hold d
            }
        }
    }
};

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

} // namespace fqk
