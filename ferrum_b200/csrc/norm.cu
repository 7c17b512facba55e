// The steps on either side of a projection: the row normalisation that produces its input and the reductions
// that consume the output head's logits.  Counterparts of `h_rmsnorm` / `h_add_rmsnorm`
// (src/metal/shaders/hybrid.metal:1563-1595; `HybridModel::rmsnorm` / `add_rmsnorm`, src/hybrid/engine.rs:3301-3345),
// `h_argmax` (:2214-2243) and `h_topk_blocks` (:3616-3657).  The normalisation is also available inside the
// activation preparation of the decode / verify projections (ProjectArgs::norm_w), with the same arithmetic.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>
#include <utility>

#include "gemv_common.cuh"
#include "internal.h"

namespace {
using namespace fqk;

// WPR warps per row.  A row's values stay in registers between the sum and the scaling (CACHED float4s a thread; longer
// rows are read again), every load of a thread is in flight at once, and the launch overlaps the end of the kernel before
// it.  The sum is that of sixteen virtual warps (gemv_common.cuh) whatever WPR, so the bits do not depend on it.
template <int WPR, int CACHED> constexpr int NORM_BLOCK = WPR == 16 ? 16 : WPR == 8 || CACHED <= 2 ? 8 : 4; // warps
template <int WPR, int CACHED>
__global__ void __launch_bounds__(NORM_BLOCK<WPR, CACHED> * 32)
k_rmsnorm(const float *x, const float *r, const float *w, uint32_t n, float eps, uint32_t rows, float *h, float *y) {
    pdl_trigger();
    // x, r and w may be the outputs of kernels that still run when this grid starts: coherent loads after the wait (through
    // L1 for the weights, which every row reads).  h may be
    // x, and y may be x or r: every value of a row is read before the first of its y is written, and a value's h by the
    // thread that read it.
    pdl_wait();
    // Warps of a block; virtual warps of a warp, as far as the row reaches (a row that is all cached may be shorter).
    constexpr uint32_t W = NORM_BLOCK<WPR, CACHED>, PER = CACHED < NORM_WARPS / WPR ? CACHED : NORM_WARPS / WPR;
    constexpr bool TAIL = CACHED >= NORM_WARPS / WPR;
    __shared__ float part[W / WPR][NORM_WARPS];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n4 = n / 4, slot = warp / WPR;
    const uint32_t row = blockIdx.x * (W / WPR) + slot;
    const bool live = row < rows;
    const size_t base = (size_t)(live ? row : 0) * n4;
    const uint32_t first = 32 * (warp % WPR) + lane, end = live ? n4 : 0;
    const float4 *xr = reinterpret_cast<const float4 *>(x) + base, *rr = r ? reinterpret_cast<const float4 *>(r) + base : nullptr;
    float4 *hr = r ? reinterpret_cast<float4 *>(h) + base : nullptr, *yr = reinterpret_cast<float4 *>(y) + base;
    const float4 *g = reinterpret_cast<const float4 *>(w);
    auto sum = [](const float4 &a, const float4 &b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); };
    float4 v[CACHED]; // value j is the thread's j-th float4 of the row: virtual warp j % PER, its step j / PER
#pragma unroll
    for (int j = 0; j < CACHED; j++) {
        const uint32_t i = first + 32 * WPR * j;
        if (i < end) v[j] = __ldcg(xr + i);
    }
    if (r) { // h = x + r first; the norm is taken of h
#pragma unroll
        for (int j = 0; j < CACHED; j++) {
            const uint32_t i = first + 32 * WPR * j;
            if (i < end) v[j] = sum(v[j], __ldcg(rr + i));
        }
    }
    float4 gv[CACHED]; // the weights are on their way while the sum is taken
#pragma unroll
    for (int j = 0; j < CACHED; j++) {
        const uint32_t i = first + 32 * WPR * j;
        if (i < end) gv[j] = g[i];
    }
    float ss[PER];
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) ss[k] = 0.f;
#pragma unroll
    for (int j = 0; j < CACHED; j++) {
        const uint32_t i = first + 32 * WPR * j;
        if (i < end) {
            if (r) hr[i] = v[j];
            ss[j % PER] = norm_square(ss[j % PER], v[j]);
        }
    }
    static_assert(!TAIL || CACHED % PER == 0, "the tail starts with virtual warp 0 of the warp");
    if constexpr (TAIL)
        for (uint32_t i0 = first + 32 * WPR * CACHED; i0 < end; i0 += 32 * NORM_WARPS)
#pragma unroll
            for (uint32_t k = 0; k < PER; k++) {
                const uint32_t i = i0 + 32 * WPR * k;
                if (i < end) {
                    float4 a = __ldcg(xr + i);
                    if (r) hr[i] = a = sum(a, __ldcg(rr + i));
                    ss[k] = norm_square(ss[k], a);
                }
            }
    float scale;
    if constexpr (WPR == 1) {
        // The sums of all virtual warps at once: the same butterfly steps, but at each a lane keeps only the half of the
        // sums that its bit picks, so that sum k ends in the lanes from k * 32 / PER on.
        uint32_t off = 16;
#pragma unroll
        for (uint32_t half = PER / 2; half > 0; half /= 2, off /= 2)
#pragma unroll
            for (uint32_t k = 0; k < half; k++) {
                const float give = (lane & off) ? ss[k] : ss[k + half], keep = (lane & off) ? ss[k + half] : ss[k];
                ss[k] = keep + __shfl_xor_sync(0xffffffffu, give, off);
            }
#pragma unroll
        for (; off > 0; off /= 2) ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], off);
        float sums[PER];
#pragma unroll
        for (uint32_t k = 0; k < PER; k++) sums[k] = __shfl_sync(0xffffffffu, ss[0], k * (32 / PER));
        scale = norm_finish<PER>(sums, n, eps);
    } else {
#pragma unroll
        for (uint32_t k = 0; k < PER; k++) ss[k] = norm_butterfly(ss[k]);
        if (lane == 0)
#pragma unroll
            for (uint32_t k = 0; k < PER; k++) part[slot][warp % WPR + WPR * k] = ss[k];
        __syncthreads();
        scale = norm_finish(part[slot], n, eps);
    }
    auto scaled = [scale](const float4 &a, const float4 &b) {
        return make_float4(a.x * scale * b.x, a.y * scale * b.y, a.z * scale * b.z, a.w * scale * b.w);
    };
#pragma unroll
    for (int j = 0; j < CACHED; j++) {
        const uint32_t i = first + 32 * WPR * j;
        if (i < end) yr[i] = scaled(v[j], gv[j]);
    }
    if constexpr (TAIL)
        for (uint32_t i = first + 32 * WPR * CACHED; i < end; i += 32 * WPR) yr[i] = scaled(__ldcg((r ? hr : xr) + i), g[i]);
}

cudaError_t launch_norm(fq_device *dev, const float *x, const float *r, const float *w, uint32_t n, float eps, uint32_t rows, float *h, float *y) {
    auto go = [&](auto wpr, auto cached) {
        constexpr int WPR = decltype(wpr)::value, C = decltype(cached)::value, W = NORM_BLOCK<WPR, C>;
        return launch_pdl(k_rmsnorm<WPR, C>, dim3((rows + W / WPR - 1) / (W / WPR)), dim3(W * 32), 0, dev->stream, x, r, w, n, eps, rows, h, y);
    };
    using std::integral_constant;
    constexpr integral_constant<int, 1> one;
    constexpr integral_constant<int, 2> two;
    constexpr integral_constant<int, 4> four;
    constexpr integral_constant<int, 8> eight;
    // A few rows, a decode step's, are bound by latency: sixteen warps a row (1 x 5120 1.9 us; one warp 11).  With more rows
    // than two per SM the machine is full anyway and a row takes the warps its values keep busy: us with that many against
    // sixteen, 16384 x 128 4.7 / 78, 1024 x 2048 3.9 / 6.5, 2048 x 4096 8.9 / 13.0, 1024 x 5120 6.9 / 10.5.
    if (rows <= 2 * (uint32_t)dev->sm_count || n > 8192) return go(integral_constant<int, 16>{}, eight);
    if (n > 4096) return go(eight, eight);
    if (n > 2048) return go(four, eight);
    if (n > 1024) return go(two, eight);
    return n > 512 ? go(one, eight) : n > 256 ? go(one, four) : n > 128 ? go(one, two) : go(one, one);
}

__device__ __forceinline__ void better(float &bv, uint32_t &bi, float ov, uint32_t oi) {
    if (ov > bv || (ov == bv && oi < bi)) {
        bv = ov;
        bi = oi;
    }
}

// Float groups first, first + step, .. below `groups` of a row: the first maximum of a thread's share so far.
template <int VEC>
__device__ __forceinline__ void argmax_scan(const float *x, uint32_t first, uint32_t groups, uint32_t step, float &bv, uint32_t &bi) {
    auto take = [&](float v, uint32_t i) {
        if (v > bv) {
            bv = v;
            bi = i;
        }
    };
#pragma unroll 4
    for (uint32_t i = first; i < groups; i += step) {
        if constexpr (VEC == 4) {
            const float4 v = reinterpret_cast<const float4 *>(x)[i];
            take(v.x, 4 * i);
            take(v.y, 4 * i + 1);
            take(v.z, 4 * i + 2);
            take(v.w, 4 * i + 3);
        } else {
            take(x[i], i);
        }
    }
}
template <int LANES> __device__ __forceinline__ void argmax_reduce(float &bv, uint32_t &bi) {
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) better(bv, bi, __shfl_down_sync(0xffffffffu, bv, off), __shfl_down_sync(0xffffffffu, bi, off));
}

// The index of the first maximum of a row, by a cluster of eight blocks: each takes a contiguous part of the row and
// block 0 collects the parts' winners through distributed shared memory (a 151,936-value row of logits: 7.8 us with
// one block, whose single SM is what bounds it).  VEC: values per load (4 where rows start on 16-byte boundaries).
constexpr int ARGMAX_CLUSTER = 8;
template <int VEC>
__global__ void __cluster_dims__(ARGMAX_CLUSTER, 1, 1) __launch_bounds__(512)
k_argmax(const float *x, uint32_t n, uint32_t *out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float best_v[16];
    __shared__ uint32_t best_i[16];
    __shared__ float part_v[ARGMAX_CLUSTER];
    __shared__ uint32_t part_i[ARGMAX_CLUSTER];
    // Block 0's shared memory may be written once every block of the cluster is known to run: arrived here, waited for
    // just before the first remote store, so that the scan of the row hides it.
    cg::cluster_group::arrival_token running = cluster.barrier_arrive();
    pdl_trigger();
    pdl_wait(); // the logits are the output of a kernel that may still run when this grid starts: coherent loads from here on
    const uint32_t tid = threadIdx.x, rank = cluster.block_rank();
    x += (size_t)blockIdx.y * n;
    const uint32_t groups = (n + VEC - 1) / VEC, per = (groups + ARGMAX_CLUSTER - 1) / ARGMAX_CLUSTER;
    const uint32_t end = min(groups, (rank + 1) * per);
    float bv = -INFINITY;
    uint32_t bi = 0;
    argmax_scan<VEC>(x, rank * per + tid, end, 512, bv, bi);
    argmax_reduce<32>(bv, bi);
    if ((tid & 31) == 0) {
        best_v[tid >> 5] = bv;
        best_i[tid >> 5] = bi;
    }
    __syncthreads();
    cluster.barrier_wait(std::move(running));
    if (tid < 32) {
        bv = best_v[tid & 15];
        bi = best_i[tid & 15];
        argmax_reduce<16>(bv, bi);
        if (tid == 0) {
            cluster.map_shared_rank(part_v, 0)[rank] = bv;
            cluster.map_shared_rank(part_i, 0)[rank] = bi;
        }
    }
    cluster.sync();
    if (rank == 0 && tid < 32) {
        bv = part_v[tid & 7];
        bi = part_i[tid & 7];
        argmax_reduce<8>(bv, bi);
        if (tid == 0) out[blockIdx.y] = bi;
    }
}

// The same by WPR warps per row, without a cluster.
template <int VEC, int WPR>
__global__ void __launch_bounds__(WPR == 32 ? 1024 : 256)
k_argmax_rows(const float *x, uint32_t n, uint32_t rows, uint32_t *out) {
    pdl_trigger();
    pdl_wait(); // as above
    constexpr uint32_t W = WPR == 32 ? 32 : 8;
    __shared__ float best_v[W];
    __shared__ uint32_t best_i[W];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = blockIdx.x * (W / WPR) + warp / WPR;
    if (row >= rows) return; // whole warps, and with several per row whole blocks
    x += (size_t)row * n;
    float bv = -INFINITY;
    uint32_t bi = 0;
    argmax_scan<VEC>(x, 32 * (warp % WPR) + lane, (n + VEC - 1) / VEC, 32 * WPR, bv, bi);
    argmax_reduce<32>(bv, bi);
    if constexpr (WPR > 1) {
        if (lane == 0) {
            best_v[warp] = bv;
            best_i[warp] = bi;
        }
        __syncthreads();
        if (warp != 0) return;
        bv = best_v[lane % WPR];
        bi = best_i[lane % WPR];
        argmax_reduce<WPR>(bv, bi);
    }
    if (lane == 0) out[row] = bi;
}

// grid (ceil(n / 1024), rows), 256 threads: per 1024-value block the 32 largest (value, index) pairs in descending
// order, ties to the lower index; out[(row * blocks + block) * 32 + k] = {value, index bits}.
__global__ void __launch_bounds__(256)
k_topk_blocks(const float *__restrict__ x, uint32_t n, float2 *__restrict__ out) {
    __shared__ float sv[8];
    __shared__ uint32_t si[8];
    const uint32_t tid = threadIdx.x, block = blockIdx.x;
    x += (size_t)blockIdx.y * n;
    out += (size_t)blockIdx.y * ((n + 1023) / 1024) * 32;
    float v[4];
    uint32_t idx[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        idx[j] = block * 1024 + j * 256 + tid;
        v[j] = idx[j] < n ? x[idx[j]] : -INFINITY;
    }
    for (int k = 0; k < 32; k++) {
        float best = v[0];
        uint32_t bidx = idx[0];
        int slot = 0;
#pragma unroll
        for (int j = 1; j < 4; j++)
            if (v[j] > best || (v[j] == best && idx[j] < bidx)) {
                best = v[j];
                bidx = idx[j];
                slot = j;
            }
        float wv = best;
        uint32_t wi = bidx;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) better(wv, wi, __shfl_down_sync(0xffffffffu, wv, off), __shfl_down_sync(0xffffffffu, wi, off));
        if ((tid & 31) == 0) {
            sv[tid >> 5] = wv;
            si[tid >> 5] = wi;
        }
        __syncthreads();
        float gv = sv[0];
        uint32_t gi = si[0];
#pragma unroll
        for (int s = 1; s < 8; s++) better(gv, gi, sv[s], si[s]);
        __syncthreads();
        if (tid == 0) out[block * 32 + k] = make_float2(gv, __uint_as_float(gi));
        if (bidx == gi && best == gv) v[slot] = -INFINITY;
    }
}

int check_norm(fq_device *dev, const float *x, const float *w, uint32_t n, uint32_t rows, const float *y) {
    if (n == 0 || n % 4 || rows == 0) return fq_fail(dev, FQ_ERR_SHAPE, "normalisation of %u rows of %u values (a multiple of 4)", rows, n);
    if (int rc = fq_check_binding(dev, x, (size_t)rows * n * 4, "x")) return rc;
    if (int rc = fq_check_binding(dev, w, (size_t)n * 4, "w")) return rc;
    return fq_check_binding(dev, y, (size_t)rows * n * 4, "y");
}

} // namespace

extern "C" int fq_rmsnorm(fq_device *dev, const float *x, const float *w, uint32_t n, float eps, uint32_t rows, float *y) {
    if (int rc = fq_begin_enqueue(dev)) return rc;
    if (int rc = check_norm(dev, x, w, n, rows, y)) return rc;
    if (int rc = fq_check_cuda(dev, launch_norm(dev, x, nullptr, w, n, eps, rows, nullptr, y), "rmsnorm launch")) return rc;
    return fq_end_enqueue(dev, "rmsnorm", 1);
}

extern "C" int fq_add_rmsnorm(fq_device *dev, const float *x, const float *r, const float *w, uint32_t n, float eps, uint32_t rows, float *h,
                              float *y) {
    if (int rc = fq_begin_enqueue(dev)) return rc;
    if (int rc = check_norm(dev, x, w, n, rows, y)) return rc;
    if (int rc = fq_check_binding(dev, r, (size_t)rows * n * 4, "r")) return rc;
    if (int rc = fq_check_binding(dev, h, (size_t)rows * n * 4, "h")) return rc;
    if (int rc = fq_check_no_alias(dev, y, (size_t)rows * n * 4, h, (size_t)rows * n * 4, "y")) return rc;
    if (int rc = fq_check_cuda(dev, launch_norm(dev, x, r, w, n, eps, rows, h, y), "add_rmsnorm launch")) return rc;
    return fq_end_enqueue(dev, "add_rmsnorm", 1);
}

extern "C" int fq_argmax(fq_device *dev, const float *x, uint32_t n, uint32_t rows, uint32_t *out) {
    if (int rc = fq_begin_enqueue(dev)) return rc;
    if (n == 0 || rows == 0) return fq_fail(dev, FQ_ERR_SHAPE, "argmax of %u rows of %u values", rows, n);
    if (int rc = fq_check_binding(dev, x, (size_t)rows * n * 4, "x")) return rc;
    if (int rc = fq_check_binding(dev, out, (size_t)rows * 4, "out")) return rc;
    // us with a cluster / one / eight / 32 warps: 1 x 151936 2.7 / 70 / 10 / 4.9, 64 x 151936 5.1 / 72 / 11 / 7.2, 32 x 32000
    // 2.8 / 16 / 3.7 / 2.6, 148 x 8192 6.3 / 5.0 / 1.9 / 2.1, 1024 x 1024 31 / 1.8 / 2.3 / 5.2, 64 x 256 2.5 / 1.4 / 1.4 / 1.6.
    const bool cluster = (n >= 16384 && rows <= 16) || (n >= 65536 && rows <= 64);
    if (!cluster) {
        const int shape = n <= 128 || (n <= 2048 && rows >= 1024) ? 1 : n < 12288 ? 8 : 32; // warps per row
        auto go = [&](auto vec) {
            constexpr int VEC = decltype(vec)::value;
            return shape == 1   ? launch_pdl(k_argmax_rows<VEC, 1>, dim3((rows + 7) / 8), dim3(256), 0, dev->stream, x, n, rows, out)
                   : shape == 8 ? launch_pdl(k_argmax_rows<VEC, 8>, dim3(rows), dim3(256), 0, dev->stream, x, n, rows, out)
                                : launch_pdl(k_argmax_rows<VEC, 32>, dim3(rows), dim3(1024), 0, dev->stream, x, n, rows, out);
        };
        const cudaError_t e = n % 4 == 0 ? go(std::integral_constant<int, 4>{}) : go(std::integral_constant<int, 1>{});
        if (int rc = fq_check_cuda(dev, e, "argmax launch")) return rc;
        return fq_end_enqueue(dev, "argmax", 1);
    }
    for (uint32_t r0 = 0; r0 < rows; r0 += 65535) { // rows sit in the grid's y extent
        const dim3 grid(ARGMAX_CLUSTER, std::min(rows - r0, 65535u));
        const float *xr = x + (size_t)r0 * n;
        const cudaError_t e = n % 4 == 0 ? launch_pdl(k_argmax<4>, grid, dim3(512), 0, dev->stream, xr, n, out + r0)
                                         : launch_pdl(k_argmax<1>, grid, dim3(512), 0, dev->stream, xr, n, out + r0);
        if (int rc = fq_check_cuda(dev, e, "argmax launch")) return rc;
    }
    return fq_end_enqueue(dev, "argmax", 1);
}

extern "C" int fq_topk_blocks(fq_device *dev, const float *x, uint32_t n, uint32_t rows, float *out) {
    if (int rc = fq_begin_enqueue(dev)) return rc;
    if (n == 0 || rows == 0) return fq_fail(dev, FQ_ERR_SHAPE, "top-k of %u rows of %u values", rows, n);
    const uint32_t blocks = (n + 1023) / 1024;
    if (int rc = fq_check_binding(dev, x, (size_t)rows * n * 4, "x")) return rc;
    if (int rc = fq_check_binding(dev, out, (size_t)rows * blocks * 32 * 8, "out")) return rc;
    k_topk_blocks<<<dim3(blocks, rows), 256, 0, dev->stream>>>(x, n, reinterpret_cast<float2 *>(out));
    return fq_end_enqueue(dev, "topk_blocks", 1);
}
