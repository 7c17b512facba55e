// Pieces shared by the kernels that multiply ONE activation row (gemv_i8.cu, moe_decode.cu): the prepared activation row,
// the packed fragments of a superblock, and the dot product of a 16-row weight tile's superblock with the row on the
// integer tensor path.  gemv_i8.cu explains the arithmetic.
#pragma once
#include "blocks.cuh"
#include "gemv_common.cuh"

namespace fqk {

// ---------------------------------------------------------------- prepared activations
//
// Per group (one activation row in expert mode, else all rows) and token:
//   plane[2][cols] s8   hi and lo bytes of x' in natural k order
//   sx32 [cols / 32] s32   sum of x' per 32 values            (Q4_K minimum term)
//   sx16 [2][cols / 16] s16  sum of hi / lo bytes per 16 values (Q6_K "- 32" term)
//   isc  [cols / 256] f32  1 / s
struct PrepI8 {
    uint32_t cols, nblk;
    uint32_t lo_off, sx32_off, sx16_off, isc_off, token_bytes;
};

__host__ __device__ inline PrepI8 prep_i8_layout(uint32_t cols) {
    PrepI8 L;
    L.cols = cols;
    L.nblk = cols / 256;
    L.lo_off = cols;
    L.sx32_off = 2 * cols;
    L.sx16_off = L.sx32_off + cols / 32 * 4;
    L.isc_off = L.sx16_off + 2 * (cols / 16) * 2;
    L.token_bytes = (L.isc_off + L.nblk * 4 + 255u) & ~255u;
    return L;
}

// Superblock b of one activation row, by one warp (lane l owns the eight values at 256 b + 8 l), written in
// the layout above at `base` (global or shared memory).
// With `urow` the activations are the gated unit silu(x) * u, x / (1 + exp(-x)) * u as `k_swiglu` computes it.
// With `norm_w` they are rmsnorm(x) * norm_w (`h_rmsnorm`, src/metal/shaders/hybrid.metal:1563-1575).
// `bsrc` is the superblock of the row that is read, `b` the slot of the layout `L` it is written to (the same
// unless `L` describes a slice of the row); `norm_scale` = row_inv_rms of the whole row when `norm_w` is given.
struct PrepLoad { // the lane's eight values of one superblock, fetched ahead of their use
    float4 v0, v1;
    __device__ __forceinline__ void fetch(const float *__restrict__ xrow, uint32_t bsrc, uint32_t lane) {
        const float4 *src = reinterpret_cast<const float4 *>(xrow + (size_t)bsrc * 256 + lane * 8);
        v0 = src[0];
        v1 = src[1];
    }
};
// `v`: the lane's eight activations of the superblock, whatever they were computed from.
__device__ __forceinline__ void prep_values(const float (&v)[8], uint32_t b, uint32_t lane, const PrepI8 &L, uint8_t *base) {
    const Quant8 q = quantize8(v);
    const bool finite = q.finite;
    const int e = q.e;
    int sum = q.sum, sum_hi = q.sum_hi, sum_lo = q.sum_lo;
    auto pack8 = [](const uint8_t *p) { return make_uint2(pack4(p), pack4(p + 4)); };
    const uint8_t *hi = q.hi, *lo = q.lo;
    reinterpret_cast<uint2 *>(base)[b * 32 + lane] = pack8(hi);
    reinterpret_cast<uint2 *>(base + L.lo_off)[b * 32 + lane] = pack8(lo);
    // 16-value sums (lane pairs) and 32-value sums (lane quads).
    sum_hi += __shfl_xor_sync(0xffffffffu, sum_hi, 1);
    sum_lo += __shfl_xor_sync(0xffffffffu, sum_lo, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if ((lane & 1) == 0) {
        int16_t *s16 = reinterpret_cast<int16_t *>(base + L.sx16_off);
        s16[b * 16 + (lane >> 1)] = (int16_t)sum_hi;
        s16[L.cols / 16 + b * 16 + (lane >> 1)] = (int16_t)sum_lo;
    }
    if ((lane & 3) == 0) reinterpret_cast<int *>(base + L.sx32_off)[b * 8 + (lane >> 2)] = sum;
    if (lane == 0) {
        // A non-finite activation anywhere in the block makes the block's factor NaN.
        reinterpret_cast<float *>(base + L.isc_off)[b] = finite ? ldexpf(1.f, -e) : __int_as_float(0x7fc00000);
    }
}
__device__ __forceinline__ void prep_superblock(const PrepLoad &in, uint32_t bsrc, uint32_t b, uint32_t lane, const PrepI8 &L, uint8_t *base,
                                                const float *__restrict__ urow, const float *__restrict__ norm_w, float norm_scale) {
    const float4 v0 = in.v0, v1 = in.v1;
    float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    if (norm_w) {
        const float scale = norm_scale;
        const float4 *ws = reinterpret_cast<const float4 *>(norm_w + (size_t)bsrc * 256 + lane * 8);
        const float4 w0 = ws[0], w1 = ws[1];
        const float g[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = v[i] * scale * g[i];
    }
    if (urow) {
        const float4 *us = reinterpret_cast<const float4 *>(urow + (size_t)bsrc * 256 + lane * 8);
        const float4 u0 = us[0], u1 = us[1];
        const float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = v[i] / (1.f + expf(-v[i])) * u[i];
    }
    prep_values(v, b, lane, L, base);
}

__device__ __forceinline__ void prep_superblock(const float *__restrict__ xrow, uint32_t bsrc, uint32_t b, uint32_t lane, const PrepI8 &L, uint8_t *base,
                                                const float *__restrict__ urow, const float *__restrict__ norm_w, float norm_scale) {
    PrepLoad in;
    in.fetch(xrow, bsrc, lane);
    prep_superblock(in, bsrc, b, lane, L, base, urow, norm_w, norm_scale);
}

// ---------------------------------------------------------------- helpers

// Q4_K: the header, 16 bytes of chunk t / 2 and 16 bytes of chunk 2 + t / 2 (bytes 16 (t % 2) .. of each
// chunk's 32), so that the four threads of a quad read 64 contiguous bytes per instruction.
struct Q4Raw {
    uint4 hdr, qa, qb;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t, uint32_t b, int t) {
        const uint8_t *blk = row + (size_t)b * 144;
        hdr = ldw128(blk);
        qa = ldw128(blk + 16 + 16 * t);
        qb = ldw128(blk + 80 + 16 * t);
    }
    // From a row of a ring stage (shared memory): the block's 144 bytes.
    __device__ __forceinline__ void load_staged(const uint8_t *r, uint32_t, int t) {
        hdr = *reinterpret_cast<const uint4 *>(r);
        qa = *reinterpret_cast<const uint4 *>(r + 16 + 16 * t);
        qb = *reinterpret_cast<const uint4 *>(r + 80 + 16 * t);
    }
};
// Q5_K: as Q4_K, plus the 16 bytes of qh under this thread's run (bit j of qh[l] = fifth bit of value l of sub-block j).
struct Q5Raw {
    uint4 hdr, qa, qb, qh;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t, uint32_t b, int t) {
        const uint8_t *blk = row + (size_t)b * 176;
        hdr = ldw128(blk);
        qh = ldw128(blk + 16 + 16 * (t & 1));
        qa = ldw128(blk + 48 + 16 * t);
        qb = ldw128(blk + 112 + 16 * t);
    }
    __device__ __forceinline__ void load_staged(const uint8_t *r, uint32_t, int t) {
        hdr = *reinterpret_cast<const uint4 *>(r);
        qh = *reinterpret_cast<const uint4 *>(r + 16 + 16 * (t & 1));
        qa = *reinterpret_cast<const uint4 *>(r + 48 + 16 * t);
        qb = *reinterpret_cast<const uint4 *>(r + 112 + 16 * t);
    }
};
struct Q6Raw;
template <int FMT> struct RawOf { using type = Q6Raw; };
template <> struct RawOf<FQ_Q4_K> { using type = Q4Raw; };
template <> struct RawOf<FQ_Q5_K> { using type = Q5Raw; };
template <int FMT> constexpr bool is_k45 = FMT == FQ_Q4_K || FMT == FQ_Q5_K;
struct Q6Raw { // device layout of blocks.cuh; thread t = (n, lh)
    uint4 q0, q1, qh; // ql of 32-groups 0|2 and 1|3 of half n, qh of half n: run lh (16 bytes each)
    uint2 sc;         // the 8 scales of half t % 2 (the half whose groups this thread sums up)
    uint32_t d;
    __device__ __forceinline__ void load(const uint8_t *row, uint32_t nblk, uint32_t b, int t) {
        const int n = t >> 1, lh = t & 1;
        const uint8_t *ql = row + (size_t)b * 128 + 64 * n + 16 * lh;
        q0 = ldw128(ql);
        q1 = ldw128(ql + 32);
        qh = ldw128(row + (size_t)nblk * 128 + (size_t)b * 64 + 32 * n + 16 * lh);
        sc = ldw64(row + (size_t)nblk * 192 + (size_t)b * 16 + 8 * (t & 1));
        d = ldw16(row + (size_t)nblk * 208 + (size_t)b * 2);
    }
    // From a row of a ring stage: ql[128] | qh[64] | scales[16]; `dword` = the stage's word that holds d.
    __device__ __forceinline__ void load_staged(const uint8_t *r, uint32_t dword, int t) {
        const int n = t >> 1, lh = t & 1;
        q0 = *reinterpret_cast<const uint4 *>(r + 64 * n + 16 * lh);
        q1 = *reinterpret_cast<const uint4 *>(r + 64 * n + 16 * lh + 32);
        qh = *reinterpret_cast<const uint4 *>(r + 128 + 32 * n + 16 * lh);
        sc = *reinterpret_cast<const uint2 *>(r + 192 + 8 * (t & 1));
        d = dword;
    }
};

// The prepared activations of one row that one thread needs for one superblock.
//   Q4_K: xb[0] / xb[1] = the 16 activation bytes under this thread's low / high nibbles of the chunk it
//         feeds (values 64 c + 16 (t % 2) + [0, 16), + 32), sx = sums of sub-blocks 4u .. 4u+3.
//   Q6_K: xb[i] = the 16 bytes under its run of 32-group i, sx = byte sums of 16-groups 8u .. 8u+7.
template <int FMT> struct Act {
    uint4 xb[is_k45<FMT> ? 2 : 4];
    uint4 sx;
    float inv;
    __device__ __forceinline__ void load(const uint8_t *tok, const PrepI8 &L, uint32_t b, int t, int g) { load_at<false>(tok, L, b, t, g); }
    // SH: `tok` is shared memory (plain loads), else global memory written by the kernel before.
    template <bool SH> __device__ __forceinline__ void load_at(const uint8_t *tok, const PrepI8 &L, uint32_t b, int t, int g) {
        auto ld128 = [](const uint8_t *p) { return SH ? *reinterpret_cast<const uint4 *>(p) : ldx128(p); };
        auto ld32 = [](const uint8_t *p) { return SH ? *reinterpret_cast<const uint32_t *>(p) : ldx32(p); };
        const int plane = g >> 2, u = t & 1;
        if constexpr (is_k45<FMT>) {
            const bool feeds = (t >> 1) == (g & 1);
            const int chunk = (((g & 3) >> 1) ? 2 : 0) + (t >> 1);
            const uint8_t *src = tok + (plane ? L.lo_off : 0) + (size_t)b * 256 + 64 * chunk + 16 * (t & 1);
#pragma unroll
            for (int i = 0; i < 2; i++) xb[i] = feeds ? ld128(src + 32 * i) : make_uint4(0, 0, 0, 0);
            sx = ld128(tok + L.sx32_off + (size_t)b * 32 + 16 * u);
        } else {
            const bool feeds = (g & 3) == t;
            const uint8_t *src = tok + (plane ? L.lo_off : 0) + (size_t)b * 256 + 128 * (t >> 1) + 16 * (t & 1);
#pragma unroll
            for (int i = 0; i < 4; i++) xb[i] = feeds ? ld128(src + 32 * i) : make_uint4(0, 0, 0, 0);
            sx = ld128(tok + L.sx16_off + ((t >> 1) ? (L.cols / 16) * 2 : 0) + (size_t)b * 32 + 16 * u);
        }
        inv = __uint_as_float(ld32(tok + L.isc_off + (size_t)b * 4));
    }
};

// One superblock of a 16-row tile against MT prepared activation rows: adds into yacc[m][r] this thread's
// share (its scale groups and plane) of rows g and g + 8.
template <int FMT, int MT, typename RawT>
__device__ __forceinline__ void superblock_dot(const RawT (&cur)[2], const Act<FMT> (&acur)[MT], int t, int g, float (&yacc)[MT][2]) {
    // This thread feeds column g of B (scale group g & 3, plane g >> 2) on its own k slots only, and
    // only if those k slots belong to that scale group; everything else it feeds is zero.
    //   Q6_K: group j = the k slots of quad thread j.
    //   Q4_K: group j = chunk j; thread t holds chunk t / 2 in its first operand word (k slots 4t ..)
    //         and chunk 2 + t / 2 in its second (k slots 16 + 4t ..).
    const bool second = is_k45<FMT> && ((g & 3) >> 1); // Q4_K / Q5_K: the group sits in the second operand word
    // It reads columns 2t, 2t+1 of the accumulators: scale groups 2 (t & 1), 2 (t & 1) + 1, plane t >> 1.
    const int u = t & 1;
    const float plane_weight = (t >> 1) ? 1.f : 256.f;
    (void)second;
    (void)u;
    if constexpr (is_k45<FMT>) {
        // The four scales and minimums of sub-blocks 4u .. 4u+3, one per byte.
        uint32_t sc4[2], mn4[2];
        float dsc[2], dmn[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint4 h = cur[r].hdr;
            sc4[r] = u ? ((h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u)) : (h.y & 0x3F3F3F3Fu);
            mn4[r] = u ? (((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u)) : (h.z & 0x3F3F3F3Fu);
            dsc[r] = f16_bits_to_f32((uint16_t)(h.x & 0xFFFFu)) * plane_weight;
            dmn[r] = (t >> 1) ? 0.f : f16_bits_to_f32((uint16_t)(h.x >> 16)); // minimum term once per plane pair
        }
        // u8 operands: low nibbles (even sub-block of the chunk) and high nibbles (odd sub-block); words
        // 0..3 from the first chunk, 4..7 from the second.
        uint32_t lo[2][8], hi[2][8];
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t wd = word_of(i < 4 ? cur[r].qa : cur[r].qb, i & 3);
                lo[r][i] = wd & 0x0F0F0F0Fu;
                hi[r][i] = (wd >> 4) & 0x0F0F0F0Fu;
                if constexpr (FMT == FQ_Q5_K) {
                    // The fifth bits: qa is chunk t / 2 (sub-blocks 2 (t / 2), + 1), qb chunk 2 + t / 2 (four bits on).
                    const uint32_t v = word_of(cur[r].qh, i & 3) >> (2 * (t >> 1) + (i < 4 ? 0 : 4));
                    lo[r][i] |= (v << 4) & 0x10101010u;
                    hi[r][i] |= (v << 3) & 0x10101010u;
                }
            }
#pragma unroll
        for (int m = 0; m < MT; m++) {
            int cl[4] = {0, 0, 0, 0}, ch[4] = {0, 0, 0, 0};
#pragma unroll
            for (int i = 0; i < 4; i++) { // word i of either chunk <-> activation bytes 4i .. 4i+3 of the run
                const uint32_t xl = word_of(acur[m].xb[0], i), xh = word_of(acur[m].xb[1], i);
                mma_u8s8(cl, lo[0][i], lo[1][i], lo[0][4 + i], lo[1][4 + i], second ? 0u : xl, second ? xl : 0u);
                mma_u8s8(ch, hi[0][i], hi[1][i], hi[0][4 + i], hi[1][4 + i], second ? 0u : xh, second ? xh : 0u);
            }
            // Columns 2t, 2t+1 = scale groups 2u, 2u+1: sub-blocks 4u (low), 4u+1 (high), 4u+2, 4u+3.
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int dot = byte_u(sc4[r], 0) * cl[2 * r] + byte_u(sc4[r], 1) * ch[2 * r] + byte_u(sc4[r], 2) * cl[2 * r + 1] +
                                byte_u(sc4[r], 3) * ch[2 * r + 1];
                const uint4 &sx = acur[m].sx;
                const int mins = byte_u(mn4[r], 0) * (int)sx.x + byte_u(mn4[r], 1) * (int)sx.y +
                                 byte_u(mn4[r], 2) * (int)sx.z + byte_u(mn4[r], 3) * (int)sx.w;
                yacc[m][r] = fmaf(acur[m].inv, dsc[r] * (float)dot - dmn[r] * (float)mins, yacc[m][r]);
            }
        }
    } else {
        // Q6_K: thread t = (n, lh) owns, for i = 0..3, the values 128 n + 32 i + 16 lh + [0, 16).
        uint32_t v4[2][4][4]; // [row][i][word]: four 6-bit quants, one per byte
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int wi = 0; wi < 4; wi++) {
                    const uint32_t lw = word_of((i & 1) ? cur[r].q1 : cur[r].q0, wi), hw = word_of(cur[r].qh, wi);
                    const uint32_t lo4 = (i < 2) ? lw : (lw >> 4);
                    const uint32_t hi4 = i == 0 ? (hw << 4) : i == 1 ? (hw << 2) : i == 2 ? hw : (hw >> 2);
                    v4[r][i][wi] = lop3_select(lo4, hi4, 0x0F0F0F0Fu) & 0x3F3F3F3Fu;
                }
        float dd[2];
#pragma unroll
        for (int r = 0; r < 2; r++) dd[r] = f16_bits_to_f32((uint16_t)cur[r].d) * plane_weight;
#pragma unroll
        for (int m = 0; m < MT; m++) {
            int dot[2] = {0, 0};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int c[4] = {0, 0, 0, 0};
                const uint4 &xv = acur[m].xb[i];
                mma_u8s8(c, v4[0][i][0], v4[1][i][0], v4[0][i][1], v4[1][i][1], xv.x, xv.y);
                mma_u8s8(c, v4[0][i][2], v4[1][i][2], v4[0][i][3], v4[1][i][3], xv.z, xv.w);
                // Columns 2t, 2t+1 = quad threads 2u, 2u+1 = (half u, runs 0 and 1): 16-groups
                // 8u + 2i and 8u + 2i + 1.  (q - 32) is applied as  dot - 32 * sum(x bytes).
                const uint32_t spair = word_of(acur[m].sx, i);
                const int s0 = (int)(int16_t)(spair & 0xFFFFu), s1 = (int)(int16_t)(spair >> 16);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const uint32_t scw = (i < 2) ? cur[r].sc.x : cur[r].sc.y;
                    dot[r] += byte_s(scw, 2 * (i & 1)) * (c[2 * r] - 32 * s0) + byte_s(scw, 2 * (i & 1) + 1) * (c[2 * r + 1] - 32 * s1);
                }
            }
#pragma unroll
            for (int r = 0; r < 2; r++) yacc[m][r] = fmaf(acur[m].inv * dd[r], (float)dot[r], yacc[m][r]);
        }
    }
}

} // namespace fqk
