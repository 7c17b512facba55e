// IQ4_NL / IQ4_XS per-route expert projections (`project_id`, F32 in, F32 out): the reference's `h_mv_id_iq4_*`
// (src/metal/shaders/hybrid.metal:2390-2428 over :900-1000), and dense projections of one short row
// (`h_mv_iq4_*`, :900-1000, 1317-1323); the other dense projections of 1..16 rows run in gemv_nt.cu.  The 4-bit indices
// go through the 16-entry codebook to signed bytes with byte permutes (no memory lookup), and from there the arithmetic
// is that of the Q8_0 kernel (gemv_q8.cu): dp4a against the byte planes of activations rounded per block of 32 -- the
// granularity of both formats' scales -- to 16 bits (routes) or, as in gemv_nt.cu, 31 (dense), then one conversion and FMA
// with d (ls - 32) / s per sub-block and pair of planes.
//
// Device layout of a row (blocks.cuh): the nibbles of all blocks first (cols / 2 bytes, natural order), then per
// block the f16 d (IQ4_NL) or the 8 bytes d | scales_h | scales_l (IQ4_XS).  Byte j of a 16-byte run holds values
// j and j + 16 of its 32.
#include <algorithm>
#include <cstdlib>

#include "blocks.cuh"
#include "gemv_common.cuh"
#include "internal.h"

namespace {

constexpr int WARPS = 8;
constexpr uint32_t MAX_COLS_IQ4 = 16384; // wider rows run on the exact fp32 kernel
// One dense row: k_nt spends most of a short row on its ring, the preparation of a slice and the exchange of partial sums
// (1024 x 1024 5.0 us against 4.2-4.4, 512 x 512 4.7 against 3.3-3.6; 4096 x 1024 5.5 against 6.4, 64 x 512 2.8 against
// 3.3).
constexpr uint32_t DENSE_COLS = 1024, DENSE_MIN_ROWS = 128, DENSE_MAX_ROWS = 2048;

// What a block of 32 with infinities and no NaN contributes, as fp32 products have it.  `q`: the weights' nibbles, `sign`:
// the block of the first plane (below).
__device__ __noinline__ float iq4_block_infinite(uint4 q, float d, const int8_t *sign) {
    float sum = 0.f;
    for (int i = 0; i < 32; i++) { // byte i of the plane: nibble byte i / 2, its high half for odd i
        const uint32_t byte = (fqk::word_of(q, i >> 3) >> (8 * ((i >> 1) & 3))) & 0xFFu;
        if (sign[i]) sum += d * iq4_value((i & 1) ? byte >> 4 : byte & 15u) * (sign[i] > 0 ? INFINITY : -INFINITY);
    }
    return sum;
}

// Shared memory: PLANES planes of [cols] signed bytes, the most significant first, then isc[cols / 32] (1 / s).
// BLOCKS: per SM at least (0: as the compiler has it).  ROUTES: blockIdx.y is a route, two planes; else one row, four planes: digits, scale and what stands for a block that is
// not finite as in Quant8Wide (gemv_common.cuh).
template <int FMT, bool ROUTES, int BLOCKS>
__global__ void __launch_bounds__(WARPS * 32, BLOCKS)
k_gemv_iq4(const uint8_t *__restrict__ w, uint32_t rows, uint32_t cols, uint32_t pitch, const float *x, float *y, const uint32_t *ids, uint32_t x_div,
           uint32_t experts) {
    constexpr int PLANES = ROUTES ? 2 : 4;
    extern __shared__ __align__(16) uint8_t iq4_smem[];
    int8_t *plane = reinterpret_cast<int8_t *>(iq4_smem);
    float *isc = reinterpret_cast<float *>(plane + (size_t)PLANES * cols);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nb32 = cols / 32;
    fqk::pdl_trigger();
    fqk::pdl_wait(); // x (and the routing) may be the output of the kernel before this one
    if constexpr (ROUTES) {
        // Route blockIdx.y uses expert ids[route] (`rows` rows each), activation row route / x_div, output row route.
        const uint32_t route = blockIdx.y, expert = ids[route];
        if (expert >= experts) return;
        w += (size_t)expert * rows * pitch;
        x += (size_t)(route / x_div) * cols;
        y += (size_t)route * rows;
    }

    // 1. Activations -> integers, one warp per block of 32, lane = value (as in gemv_q8.cu).
    for (uint32_t b = warp; b < nb32; b += WARPS) {
        const float v = x[32 * b + lane];
        float amax = fabsf(v);
        // Within a run the bytes sit where the permuted codebook values of the weights fall: a byte pair (2p, 2p + 1)
        // of nibbles decodes to values 2p, 2p + 16, 2p + 1, 2p + 17 in that order.
        int8_t *at = plane + 32 * b + 2 * (lane & 15u) + (lane >> 4);
        if constexpr (ROUTES) {
            const bool finite = __ballot_sync(0xffffffffu, !(fabsf(v) < INFINITY)) == 0u;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
            int e = 0;
            if (amax > 0.f && finite) {
                const int ex = (int)(__float_as_uint(amax) >> 23) - 126;
                e = max(-110, min(110, 15 - ex));
                if (amax * __uint_as_float((uint32_t)(127 + e) << 23) > 32639.f) e -= 1;
            }
            int q = __float2int_rn(fminf(fmaxf(v * __uint_as_float((uint32_t)(127 + e) << 23), -32639.f), 32639.f));
            if (!finite) q = 0; // the block's factor below is NaN in that case
            const int h = (q + 128) >> 8;
            at[0] = (int8_t)h;
            at[cols] = (int8_t)(q - (h << 8));
            if (lane == 0) isc[b] = finite ? __uint_as_float((uint32_t)(127 - e) << 23) : __int_as_float(0x7fc00000);
        } else {
            const bool nan = __any_sync(0xffffffffu, v != v);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
            const fqk::WideScale s(amax, nan);
            const uint32_t d = s.finite ? s.digits(v) : s.sign_of_infinity(v);
#pragma unroll
            for (int p = 0; p < 4; p++) at[(size_t)p * cols] = (int8_t)(d >> (24 - 8 * p));
            if (lane == 0) isc[b] = s.inv;
        }
    }
    __syncthreads();

    // 2. Rows.  A warp takes RPW weight rows at a time, strided over the grid, the loads of all of them in flight
    // together; lane l reads 16 bytes = one run of 32 values (an IQ4_NL block, an IQ4_XS sub-block) of every
    // 1024-value chunk.
    constexpr int RPW = 4;
    const uint32_t chunks = (cols + 1023) / 1024, groups = (rows + RPW - 1) / RPW;
    for (uint32_t g = blockIdx.x * WARPS + warp; g < groups; g += gridDim.x * WARPS) {
        const uint32_t row0 = g * RPW;
        const uint8_t *rp[RPW];
#pragma unroll
        for (int r = 0; r < RPW; r++) rp[r] = w + (size_t)min(row0 + r, rows - 1) * pitch;
        float acc[RPW] = {};
        for (uint32_t c = 0; c < chunks; c++) {
            const uint32_t run = 32 * c + lane; // index of the 32-value run
            const bool live = run < nb32;
            const uint32_t rr = live ? run : 0;
            uint4 q[RPW];
            float d[RPW];
#pragma unroll
            for (int r = 0; r < RPW; r++) q[r] = fqk::ldw128(rp[r] + (size_t)rr * 16);
#pragma unroll
            for (int r = 0; r < RPW; r++) {
                const uint8_t *hdr = rp[r] + cols / 2;
                if constexpr (FMT == FQ_IQ4_XS) {
                    const uint8_t *h8 = hdr + (size_t)(rr / 8) * 8;
                    d[r] = load_f16(h8) * (float)iq4xs_scale(h8, (int)(rr % 8));
                } else {
                    d[r] = load_f16(hdr + (size_t)rr * 2);
                }
            }
#pragma unroll
            for (int r = 0; r < RPW; r++) {
                // byte pairs of nibbles -> four signed bytes each, in the order the activations were laid down
                const uint32_t qw[4] = {q[r].x, q[r].y, q[r].z, q[r].w};
                int4 a[PLANES][2];
                int dot[PLANES];
#pragma unroll
                for (int p = 0; p < PLANES; p++) {
                    const int4 *run_p = reinterpret_cast<const int4 *>(plane + (size_t)p * cols + (size_t)rr * 32);
                    a[p][0] = run_p[0], a[p][1] = run_p[1];
                    dot[p] = 0;
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint2 v = fqk::iq4_lookup8(qw[i]);
#pragma unroll
                    for (int p = 0; p < PLANES; p++) {
                        const int4 &b = a[p][i >> 1];
                        dot[p] = __dp4a((int)v.y, (i & 1) ? b.w : b.y, __dp4a((int)v.x, (i & 1) ? b.z : b.x, dot[p]));
                    }
                }
                const float s = live ? isc[rr] : 0.f; // lanes past the row's end contribute nothing
                if constexpr (ROUTES) acc[r] = fmaf((float)(dot[0] * 256 + dot[1]), d[r] * s, acc[r]);
                else if (s < INFINITY) acc[r] = fmaf(s, d[r] * fmaf(65536.f, (float)(dot[0] * 256 + dot[1]), (float)(dot[2] * 256 + dot[3])), acc[r]);
                else acc[r] += s != s ? s : iq4_block_infinite(q[r], d[r], plane + (size_t)rr * 32);
            }
        }
#pragma unroll
        for (int r = 0; r < RPW; r++) {
            float v = acc[r];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (lane == 0 && row0 + r < rows) y[row0 + r] = v;
        }
    }
}

template <int FMT, bool ROUTES, int BLOCKS> cudaError_t launch_as(fq_device *dev, const ProjectArgs &a, uint32_t grid) {
    const size_t smem = (size_t)(ROUTES ? 2 : 4) * a.cols + (size_t)(a.cols / 32) * sizeof(float);
    static size_t configured = 48 * 1024;
    if (smem > configured) {
        const size_t most = (size_t)2 * MAX_COLS_IQ4 + MAX_COLS_IQ4 / 8;
        cudaError_t e = cudaFuncSetAttribute(k_gemv_iq4<FMT, ROUTES, BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e != cudaSuccess) return e;
        configured = most;
    }
    return fqk::launch_pdl(k_gemv_iq4<FMT, ROUTES, BLOCKS>, dim3(grid, ROUTES ? a.m : 1), dim3(WARPS * 32), smem, dev->stream, a.w, a.rows, a.cols, a.row_bytes,
                           (const float *)a.x, (float *)a.y, a.ids, a.x_div, a.experts);
}
// IQ4_NL takes 71 registers where it may, three blocks per SM; with more blocks than that holds at once, a fourth in 64
// registers is worth more (512 x 2048, 32 routes 14.3 -> 12.0 us, eight 8.3 -> 9.1; 2048 x 512, eight 6.9 -> 6.3).
template <int FMT, bool ROUTES> cudaError_t launch(fq_device *dev, const ProjectArgs &a) {
    const uint32_t need = (a.rows + WARPS * 4 - 1) / (WARPS * 4), sms = (uint32_t)dev->sm_count, grid = std::min(need, sms * 4);
    if constexpr (FMT == FQ_IQ4_NL && ROUTES)
        if ((uint64_t)grid * a.m > 3 * sms) return launch_as<FMT, ROUTES, 4>(dev, a, grid);
    return launch_as<FMT, ROUTES, 0>(dev, a, grid);
}

} // namespace

// IQ4_NL / IQ4_XS, F32 in / F32 out, routes (`a.ids`: one activation row per route, `a.m` routes, `a.rows` rows per
// expert) or one dense row of up to DENSE_COLS values against DENSE_MIN_ROWS..DENSE_MAX_ROWS weight rows; FQ_ERR_UNSUPPORTED otherwise.
int fq_launch_gemv_iq4(fq_device *dev, const ProjectArgs &a) {
    if ((a.format != FQ_IQ4_NL && a.format != FQ_IQ4_XS) || a.x_dtype != FQ_F32 || a.y_dtype != FQ_F32 || a.offsets || a.norm_w || a.x_up)
        return FQ_ERR_UNSUPPORTED;
    if (a.m == 0 || a.m > 65535 || a.x_div == 0 || a.cols > MAX_COLS_IQ4 || a.cols % 256 || a.row_bytes % 16) return FQ_ERR_UNSUPPORTED;
    if (!a.ids && (a.m > 1 || a.cols > DENSE_COLS || a.rows < DENSE_MIN_ROWS || a.rows > DENSE_MAX_ROWS)) return FQ_ERR_UNSUPPORTED;
    const bool xs = a.format == FQ_IQ4_XS;
    const cudaError_t e = a.ids ? (xs ? launch<FQ_IQ4_XS, true>(dev, a) : launch<FQ_IQ4_NL, true>(dev, a))
                                : (xs ? launch<FQ_IQ4_XS, false>(dev, a) : launch<FQ_IQ4_NL, false>(dev, a));
    if (int rc = fq_check_cuda(dev, e, "gemv_iq4 launch")) return rc;
    return fq_end_enqueue(dev, "gemv_iq4", 1);
}
