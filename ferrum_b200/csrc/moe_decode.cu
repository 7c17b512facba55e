// The mixture-of-experts block of ONE token as one launch: router, routing, shared expert, routed experts and the
// weighted sum (`HybridModel::moe_ffn` at decode, src/hybrid/engine.rs:2881-3092).
//
// A token of the 35B-A3B-class block reads 18.9 MB of weights, 3 us of HBM time; as a chain of six kernels the block
// took 37 us, nearly all of it launch and dependency latency (router 6, routing 8, gate|up 7, the join with the shared
// expert's stream and the down projection 13).  Here one cooperative launch, a block of 16 warps per SM, goes through
// three phases with a grid-wide barrier between them:
//
//   0  every block prepares the token's activations for itself; router logits (a warp per row) and the shared expert's
//      gate and up projections (a block per 16-row tile, its warps splitting K);
//   1  every block routes the token for itself (256 logits: cheaper than another barrier), then the routed experts' gate
//      and up projections; the tiles of the next phase are known now and are fetched into L2 meanwhile;
//   2  every block prepares the gated units of all routes for itself; a block per 16-row tile of the output multiplies
//      them by their experts' down projections, one warp per route, and adds the routes in order and the shared expert.
//
// The arithmetic and the order of every sum are those of the kernels the block is otherwise made of (k_gemv_q8,
// k_gemv_i8s, k_gemv_i8 with its combine): `*_slices` and `*_split` are their ways of cutting K, so the result has the
// same bits as theirs -- what an expert-parallel block on several ranks, which uses those, is compared with.
//
// The barriers are bounded waits: a block that has waited for two seconds records FQ_ERR_TIMEOUT, waits no more and
// runs to its end.
#include <algorithm>

#include "blocks.cuh"
#include "gemv_common.cuh"
#include "gemv_i8.cuh"
#include "gemv_q8.cuh"
#include "internal.h"
#include "moe_route.cuh"

namespace {
using namespace fqk;

constexpr uint32_t WARPS = 16;
constexpr uint32_t MAX_USED = 12;    // warps of the last phase: one per route, the rest on the shared expert
constexpr uint32_t MAX_PARTS = 64;   // partial results of a tile held in shared memory
constexpr uint64_t WAIT_NS = 2000000000ull, TEST_WAIT_NS = 20000000ull;

struct MoeDecodeJob {
    const float *x, *shared_w; // shared_w null: no gate on the shared expert
    float *out;
    const uint8_t *router, *sg, *su, *sd, *ge, *ue, *de; // shared gate / up / down, the experts' gate / up / down stacks
    uint32_t router_pitch, gu_pitch, sd_pitch, dn_pitch;
    uint32_t hidden, ffn, shared_ffn, experts, used;
    int sigmoid, norm;
    uint32_t sg_slices, sd_slices, gu_split, dn_split;
    float *logits, *g, *u, *shared_g, *shared_u; // [experts], [used][ffn] x 2, [shared_ffn] x 2
    uint32_t *barrier;                           // three words, zero between launches
    uint32_t arrivals;                           // that a barrier waits for: the blocks (a test: one more, so that the wait runs out)
    uint64_t wait_ns;
    int *status;
};

__device__ __forceinline__ void prefetch_l2(const uint8_t *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Every block has arrived at `counter` when this returns (or the wait ran out: `gave_up`, for the whole block).
__device__ __forceinline__ void grid_barrier(const MoeDecodeJob &J, uint32_t *counter, uint32_t &gave_up) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(counter, 1u);
        if (!gave_up) {
            uint64_t t0 = 0;
            for (uint32_t n = 0;; n++) {
                uint32_t v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
                if (v >= J.arrivals) break;
                if ((n & 255u) == 255u) {
                    if (t0 == 0) t0 = global_ns();
                    else if (global_ns() - t0 > J.wait_ns) {
                        *(volatile int *)J.status = (int)FQ_ERR_TIMEOUT;
                        gave_up = 1u;
                        break;
                    }
                }
            }
        }
        __threadfence();
    }
    __syncthreads();
}

// A 16-row tile (first row `w`, `last` = index of the last row it may read) against superblocks first, first + step, ..
// below `end` of the prepared row, by one warp: afterwards the quad's four threads hold the sums of rows g and g + 8.
template <int FMT>
__device__ __forceinline__ void tile_dot(const uint8_t *w, uint32_t last, uint32_t pitch, uint32_t nblk, const uint8_t *act, const PrepI8 &L, uint32_t first,
                                         uint32_t step, uint32_t end, int g, int t, float (&v)[2]) {
    using Raw = typename RawOf<FMT>::type;
    const uint8_t *r0 = w + (size_t)min((uint32_t)g, last) * pitch, *r1 = w + (size_t)min((uint32_t)g + 8, last) * pitch;
    float yacc[1][2] = {{0.f, 0.f}};
    Raw cur[2], nxt[2];
    if (first < end) {
        cur[0].load(r0, nblk, first, t);
        cur[1].load(r1, nblk, first, t);
    }
    for (uint32_t b = first; b < end; b += step) {
        if (b + step < end) {
            nxt[0].load(r0, nblk, b + step, t);
            nxt[1].load(r1, nblk, b + step, t);
        }
        Act<FMT> a[1];
        a[0].template load_at<true>(act, L, b, t, g);
        superblock_dot<FMT, 1>(cur, a, t, g, yacc);
        cur[0] = nxt[0];
        cur[1] = nxt[1];
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        v[r] = yacc[0][r];
        v[r] += __shfl_xor_sync(0xffffffffu, v[r], 1);
        v[r] += __shfl_xor_sync(0xffffffffu, v[r], 2);
    }
}

// silu(g) * u of one superblock, written by other blocks of this launch, prepared into `act`.
__device__ __forceinline__ void prep_gated(const float *g, const float *u, uint32_t b, uint32_t lane, const PrepI8 &L, uint8_t *act) {
    const float4 *gp = reinterpret_cast<const float4 *>(g + (size_t)b * 256 + lane * 8), *up = reinterpret_cast<const float4 *>(u + (size_t)b * 256 + lane * 8);
    const float4 g0 = __ldcg(gp), g1 = __ldcg(gp + 1), u0 = __ldcg(up), u1 = __ldcg(up + 1);
    float v[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
    const float w[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = v[i] / (1.f + expf(-v[i])) * w[i];
    prep_values(v, b, lane, L, act);
}

struct MoeDecodeSmem { // offsets in dynamic shared memory
    uint32_t act_x, q8_hi, q8_lo, q8_isc, act_s, act_f, total;
};
__host__ __device__ inline MoeDecodeSmem moe_decode_smem(uint32_t hidden, uint32_t ffn, uint32_t shared_ffn, uint32_t used) {
    MoeDecodeSmem S;
    S.act_x = 0;
    S.q8_hi = S.act_x + prep_i8_layout(hidden).token_bytes;
    S.q8_lo = S.q8_hi + hidden;
    S.q8_isc = S.q8_lo + hidden;
    S.act_s = S.q8_isc + (hidden / 32 * 4 + 255u) / 256u * 256u;
    S.act_f = S.act_s + prep_i8_layout(shared_ffn).token_bytes;
    S.total = S.act_f + used * prep_i8_layout(ffn).token_bytes;
    return S;
}

template <int GU, int DN>
__global__ void __launch_bounds__(WARPS * 32, 1)
k_moe_decode(const __grid_constant__ MoeDecodeJob J) {
    extern __shared__ __align__(256) uint8_t md_smem[];
    __shared__ float part[MAX_PARTS][16];
    __shared__ uint32_t ids[MAX_USED];
    __shared__ float weights[MAX_USED];
    __shared__ float gate;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blocks = gridDim.x;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t H = J.hidden, F = J.ffn, SF = J.shared_ffn, hblk = H / 256, fblk = F / 256, sblk = SF / 256;
    const PrepI8 LX = prep_i8_layout(H), LF = prep_i8_layout(F), LS = prep_i8_layout(SF);
    const MoeDecodeSmem S = moe_decode_smem(H, F, SF, J.used);
    uint8_t *act_x = md_smem + S.act_x, *act_s = md_smem + S.act_s, *act_f = md_smem + S.act_f;
    int8_t *q8_hi = reinterpret_cast<int8_t *>(md_smem + S.q8_hi), *q8_lo = reinterpret_cast<int8_t *>(md_smem + S.q8_lo);
    float *q8_isc = reinterpret_cast<float *>(md_smem + S.q8_isc);
    uint32_t gave_up = 0;

    // ---- phase 0
    const uint32_t s_tiles = SF / 16; // of gate, and as many of up
    auto shared_tile = [&](uint32_t tile) { return (tile < s_tiles ? J.sg + (size_t)tile * 16 * J.gu_pitch : J.su + (size_t)(tile - s_tiles) * 16 * J.gu_pitch); };
    // The first weights of the block are on their way to L2 while it prepares the activations.
    if (blockIdx.x < 2 * s_tiles)
        for (uint32_t o = tid * 128; o < 16 * J.gu_pitch; o += WARPS * 32 * 128) prefetch_l2(shared_tile(blockIdx.x) + o);
    {
        const uint32_t row = blockIdx.x + blocks * (WARPS - 1 - warp);
        if (row < J.experts)
            for (uint32_t o = lane * 128; o < J.router_pitch; o += 32 * 128) prefetch_l2(J.router + (size_t)row * J.router_pitch + o);
    }
    for (uint32_t b = warp; b < hblk; b += WARPS) prep_superblock(J.x, b, b, lane, LX, act_x, nullptr, nullptr, 0.f);
#pragma unroll 4
    for (uint32_t b = warp; b < H / 32; b += WARPS) q8_quantize_block(J.x[32 * b + lane], lane, q8_hi + 32 * b, q8_lo + 32 * b, q8_isc + b);
    __syncthreads();
    for (uint32_t row = blockIdx.x + blocks * (WARPS - 1 - warp); row < J.experts; row += blocks * WARPS) { // a warp per row, as k_gemv_q8<1, 1>
        const uint8_t *rp = J.router + (size_t)row * J.router_pitch;
        float acc = 0.f;
#pragma unroll 4
        for (uint32_t c = 0; c < (H + 511) / 512; c++) {
            const uint32_t k = 512 * c + 16 * lane;
            const bool live = k < H;
            const uint32_t kk = live ? k : 0, b = kk / 32;
            const uint4 q = ldw128(rp + kk);
            const float d = load_f16(rp + H + 2 * b), s = live ? q8_isc[b] : 0.f;
            acc = fmaf((float)q8_dot16(q, *reinterpret_cast<const int4 *>(q8_hi + kk), *reinterpret_cast<const int4 *>(q8_lo + kk)), d * s, acc);
        }
        acc = route_warp_sum(acc);
        if (lane == 0) J.logits[row] = acc;
    }
    for (uint32_t tile = blockIdx.x; tile < 2 * s_tiles; tile += blocks) {
        for (uint32_t s = warp; s < J.sg_slices; s += WARPS) {
            float v[2];
            tile_dot<GU>(shared_tile(tile), 15, J.gu_pitch, hblk, act_x, LX, s * hblk / J.sg_slices, 1, (s + 1) * hblk / J.sg_slices, g, t, v);
            if (t == 0) part[s][g] = v[0], part[s][g + 8] = v[1];
        }
        __syncthreads();
        if (tid < 16) {
            float v = part[0][tid];
            if (J.sg_slices > 1) {
                v = 0.f;
                for (uint32_t s = 0; s < J.sg_slices; s++) v += part[s][tid];
            }
            (tile < s_tiles ? J.shared_g + tile * 16 : J.shared_u + (tile - s_tiles) * 16)[tid] = v;
        }
        __syncthreads();
    }
    grid_barrier(J, J.barrier, gave_up);

    // ---- phase 1
    if (warp == 0) {
        uint32_t id = 0;
        float weight = 0.f;
        const bool good = J.experts <= 256   ? route_row<8>(J.logits, J.experts, J.used, J.sigmoid, J.norm, lane, id, weight)
                          : J.experts <= 512 ? route_row<16>(J.logits, J.experts, J.used, J.sigmoid, J.norm, lane, id, weight)
                                             : route_row<32>(J.logits, J.experts, J.used, J.sigmoid, J.norm, lane, id, weight);
        if (lane < J.used) { // a row of logits without a ranking: reported, and the token gets weight zero
            ids[lane] = good ? id : lane;
            weights[lane] = good ? weight : 0.f;
        }
        if (!good && lane == 0) {
            gate = 0.f;
            if (blockIdx.x == 0) *(volatile int *)J.status = (int)FQ_ERR_WEIGHT;
        }
        if (good && !J.shared_w && lane == 0) gate = 1.f;
        part[0][0] = good ? 1.f : 0.f;
    } else if (warp == 1) {
        if (J.shared_w) {
            const float v = route_gate(J.x, J.shared_w, H, lane);
            if (lane == 0) part[1][0] = v;
        }
    } else {
        for (uint32_t b = warp - 2; b < sblk; b += WARPS - 2) prep_gated(J.shared_g, J.shared_u, b, lane, LS, act_s);
    }
    __syncthreads();
    if (tid == 0 && J.shared_w && part[0][0] != 0.f) gate = part[1][0];
    const uint32_t f_tiles = F / 16, h_tiles = H / 16;
    // The next phase's first tile: the routes' rows of it, and the shared expert's.
    if (blockIdx.x < h_tiles)
        for (uint32_t i = warp; i <= J.used; i += WARPS) {
            const uint32_t pitch = i < J.used ? J.dn_pitch : J.sd_pitch;
            const uint8_t *p = i < J.used ? J.de + ((size_t)ids[i] * H + blockIdx.x * 16) * pitch : J.sd + (size_t)blockIdx.x * 16 * pitch;
            for (uint32_t o = lane * 128; o < 16 * pitch; o += 32 * 128) prefetch_l2(p + o);
        }
    __syncthreads(); // `part` is free again
    {
        const uint32_t split = J.gu_split, groups = WARPS / split, group = warp / split, seg = warp % split, units = J.used * 2 * f_tiles;
        for (uint32_t base = blockIdx.x * groups; base < units; base += blocks * groups) {
            const uint32_t q = base + group;
            const bool valid = group < groups && q < units;
            const uint32_t route = q / (2 * f_tiles), in_route = q - route * 2 * f_tiles, up = in_route >= f_tiles, tile = in_route - up * f_tiles;
            float v[2];
            if (valid) {
                tile_dot<GU>((up ? J.ue : J.ge) + ((size_t)ids[route] * F + tile * 16) * J.gu_pitch, 15, J.gu_pitch, hblk, act_x, LX, seg, split, hblk, g, t, v);
                if (t == 0) part[warp][g] = v[0], part[warp][g + 8] = v[1];
            }
            __syncthreads();
            if (valid && seg == 0 && lane < 16) {
                float sum = part[warp][lane];
                for (uint32_t w = 1; w < split; w++) sum += part[warp + w][lane];
                (up ? J.u : J.g)[(size_t)route * F + tile * 16 + lane] = sum;
            }
            __syncthreads();
        }
    }
    grid_barrier(J, J.barrier + 1, gave_up);

    // ---- phase 2
    for (uint32_t i = warp; i < J.used * fblk; i += WARPS) {
        const uint32_t r = i / fblk, b = i - r * fblk;
        prep_gated(J.g + (size_t)r * F, J.u + (size_t)r * F, b, lane, LF, act_f + (size_t)r * LF.token_bytes);
    }
    __syncthreads();
    for (uint32_t tile = blockIdx.x; tile < h_tiles; tile += blocks) {
        for (uint32_t i = warp; i < J.used + J.sd_slices; i += WARPS) {
            float v[2];
            if (i < J.used) {
                const uint8_t *w = J.de + ((size_t)ids[i] * H + tile * 16) * J.dn_pitch;
                for (uint32_t seg = 0; seg < J.dn_split; seg++) {
                    float p[2];
                    tile_dot<DN>(w, 15, J.dn_pitch, fblk, act_f + (size_t)i * LF.token_bytes, LF, seg, J.dn_split, fblk, g, t, p);
                    v[0] = seg ? v[0] + p[0] : p[0];
                    v[1] = seg ? v[1] + p[1] : p[1];
                }
            } else {
                const uint32_t s = i - J.used;
                tile_dot<DN>(J.sd + (size_t)tile * 16 * J.sd_pitch, 15, J.sd_pitch, sblk, act_s, LS, s * sblk / J.sd_slices, 1, (s + 1) * sblk / J.sd_slices, g, t, v);
            }
            if (t == 0) part[i][g] = v[0], part[i][g + 8] = v[1];
        }
        __syncthreads();
        if (tid < 16) {
            float acc = 0.f;
            for (uint32_t r = 0; r < J.used; r++) acc = fmaf(weights[r], part[r][tid], acc);
            float shared = part[J.used][tid];
            if (J.sd_slices > 1) {
                shared = 0.f;
                for (uint32_t s = 0; s < J.sd_slices; s++) shared += part[J.used + s][tid];
            }
            J.out[tile * 16 + tid] = fmaf(gate, shared, acc);
        }
        __syncthreads();
    }
    // Everybody is past both barriers: the last block to leave puts the counters back to zero.
    if (tid == 0 && atomicAdd(J.barrier + 2, 1u) + 1u == blocks) J.barrier[0] = J.barrier[1] = J.barrier[2] = 0;
}

template <int GU, int DN> cudaError_t launch(fq_device *dev, const MoeDecodeJob &J, size_t smem) {
    auto kernel = k_moe_decode<GU, DN>;
    static size_t configured = 32 * 1024;
    if (smem > configured) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(200 * 1024));
        if (e != cudaSuccess) return e;
        configured = 200 * 1024;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)dev->sm_count);
    cfg.blockDim = dim3(WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = dev->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative; // the blocks wait for one another
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, J);
}

} // namespace

// One token on the shapes and formats above (the experts' and the shared expert's matrices of one format per role, a
// Q8_0 router, widths a whole number of superblocks); FQ_ERR_UNSUPPORTED otherwise, nothing enqueued.  `logits` ..
// `shared_u`: parts of `scratch`, of experts, used * ffn (twice) and shared_ffn (twice) floats; x, out and the gate's
// weight lie outside `scratch`.
int fq_launch_moe_decode(fq_device *dev, const fq_moe_ffn_desc *f, const float *x, float *scratch, size_t scratch_elems, float *logits, float *g, float *u,
                         float *shared_g, float *shared_u, float *out) {
    const int gu = f->gate_exps->format, dn = f->down_exps->format;
    const uint32_t H = f->hidden, F = f->expert_ffn, SF = f->shared_ffn;
    if (f->router->format != FQ_Q8_0 || f->up_exps->format != gu || f->shared_gate->format != gu || f->shared_up->format != gu || f->shared_down->format != dn)
        return FQ_ERR_UNSUPPORTED;
    if (H % 256 || F % 256 || SF % 256 || H == 0 || F == 0 || SF == 0 || H > 16384 || f->used == 0 || f->used > MAX_USED || f->experts > 1024 || f->used > f->experts)
        return FQ_ERR_UNSUPPORTED;
    // In the last phase a warp walks a route's row alone, F / 256 superblocks, and a tile of the shared expert's gate or up
    // has no more warps than k_gemv_i8s cuts K into slices; the chain deals both out over all SMs.  Wide blocks are its:
    // one launch against chain, us, Q4_K / Q6_K, 16 experts: H 2048, two routes, F 1024 20.9 / 34.3, 3072 33.6 / 38.7,
    // 4096 37.7 / 41.4, 8192 66.9 / 52.5; four routes, F 3072 41.2 / 48.7, 4096 51.7 / 51.8; H 4096, one route, F 2048
    // 35.4 / 40.6, 3072 47.2 / 42.7, eight routes, F 3072 88.2 / 93.1, 4096 113 / 108; shared expert at H 2048, F 1024:
    // 4096 30.9 / 40.2, 8192 51.0 / 43.5.
    const uint32_t used = f->used;
    const uint32_t most_ffn = H <= 2048 ? (used <= 2 ? 4096u : used <= 4 || H > 1024 ? 3072u : 2048u)
                                        : (used >= 12 ? 4096u : used >= 8 || (used >= 4 && H <= 4096) ? 3072u : 2048u);
    const uint32_t most_shared = F > 2048 ? 2048u : H <= 2048 ? (used >= 4 ? 6144u : 4096u) : H <= 4096 && F >= 512 ? 4096u : 2048u;
    if (F > most_ffn || SF > most_shared) return FQ_ERR_UNSUPPORTED;
    if (f->shared_up->rows != SF || f->shared_gate->cols != H || f->shared_up->cols != H || f->shared_down->cols != SF || f->up_exps->cols != H)
        return FQ_ERR_UNSUPPORTED;
    MoeDecodeJob J{};
    J.x = x;
    J.shared_w = f->shared_gate_inp;
    J.out = out;
    J.router = f->router->data;
    J.sg = f->shared_gate->data;
    J.su = f->shared_up->data;
    J.sd = f->shared_down->data;
    J.ge = f->gate_exps->data;
    J.ue = f->up_exps->data;
    J.de = f->down_exps->data;
    J.router_pitch = (uint32_t)f->router->pitch;
    J.gu_pitch = (uint32_t)f->gate_exps->pitch;
    J.sd_pitch = (uint32_t)f->shared_down->pitch;
    J.dn_pitch = (uint32_t)f->down_exps->pitch;
    J.hidden = H;
    J.ffn = F;
    J.shared_ffn = SF;
    J.experts = f->experts;
    J.used = f->used;
    J.sigmoid = f->sigmoid;
    J.norm = f->norm_weights;
    J.sg_slices = fq_gemv_i8_slices(dev, 2 * (SF / 16), H / 256);
    J.sd_slices = fq_gemv_i8_slices(dev, H / 16, SF / 256);
    J.gu_split = fq_gemv_i8_split(dev, 2 * (F / 16), f->used, H / 256);
    J.dn_split = fq_gemv_i8_split(dev, H / 16, f->used, F / 256);
    if (J.sg_slices > MAX_PARTS || J.used + J.sd_slices > MAX_PARTS || J.gu_split > WARPS) return FQ_ERR_UNSUPPORTED;
    J.logits = logits;
    J.g = g;
    J.u = u;
    J.shared_g = shared_g;
    J.shared_u = shared_u;
    J.barrier = dev->combine_counters + FQ_COMBINE_COUNTERS;
    J.arrivals = (uint32_t)dev->sm_count + (dev->test_moe_wait ? 1 : 0);
    J.wait_ns = dev->test_moe_wait ? TEST_WAIT_NS : WAIT_NS;
    J.status = dev->status_dev;
    const size_t smem = moe_decode_smem(H, F, SF, f->used).total;
    if (smem > 200 * 1024) return FQ_ERR_UNSUPPORTED;
    auto kernel = gu == FQ_Q4_K && dn == FQ_Q6_K   ? launch<FQ_Q4_K, FQ_Q6_K>
                  : gu == FQ_Q4_K && dn == FQ_Q4_K ? launch<FQ_Q4_K, FQ_Q4_K>
                  : gu == FQ_Q5_K && dn == FQ_Q6_K ? launch<FQ_Q5_K, FQ_Q6_K>
                  : gu == FQ_Q5_K && dn == FQ_Q5_K ? launch<FQ_Q5_K, FQ_Q5_K>
                  : gu == FQ_Q6_K && dn == FQ_Q6_K ? launch<FQ_Q6_K, FQ_Q6_K>
                                                   : nullptr;
    if (!kernel) return FQ_ERR_UNSUPPORTED;
    if (int rc = fq_begin_enqueue(dev)) return rc;
    if (int rc = fq_check_binding(dev, x, (size_t)H * 4, "x")) return rc;
    if (int rc = fq_check_binding(dev, scratch, scratch_elems * 4, "scratch")) return rc;
    if (int rc = fq_check_binding(dev, out, (size_t)H * 4, "out")) return rc;
    if (f->shared_gate_inp)
        if (int rc = fq_check_binding(dev, f->shared_gate_inp, (size_t)H * 4, "shared gate weight")) return rc;
    if (int rc = fq_check_no_alias(dev, scratch, scratch_elems * 4, x, (size_t)H * 4, "scratch")) return rc;
    dev->test_moe_wait = false;
    if (int rc = fq_check_cuda(dev, kernel(dev, J, smem), "moe decode launch")) return rc;
    fq_note_write(dev, out, (size_t)H * 4);
    return fq_end_enqueue(dev, "moe_decode", 1);
}
