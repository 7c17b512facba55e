// Routing of one token by one warp, shared by the routing kernel (moe.cu) and the fused decode block (moe_decode.cu).
#pragma once
#include <stdint.h>

namespace fqk {

__device__ __forceinline__ float route_warp_sum(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Scores (softmax: max, exp, sum, divide; or a logistic per logit) and the `used` <= 32 best of `experts` <= 32 NPL,
// ties to the lower index; lane l owns experts l, l + 32, .. in registers, so a round of the arg-max is two warp-wide
// integer reductions (scores are non-negative: their bits order like the scores) and a scan of the owner's registers.
// Lane k < used returns the k-th expert in `id` and its weight, divided by the picked sum when `norm`.  False when a
// logit is not finite (such a row has no ranking).
template <int NPL>
__device__ __forceinline__ bool route_row(const float *__restrict__ row, uint32_t experts, uint32_t used, int sigmoid, int norm, uint32_t lane, uint32_t &id,
                                          float &weight) {
    float p[NPL];
    int bad = 0;
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < NPL; i++) {
        const uint32_t e = lane + 32 * i;
        p[i] = e < experts ? __ldcg(row + e) : 0.f;
        bad |= !(fabsf(p[i]) < INFINITY);
        if (e < experts) mx = fmaxf(mx, p[i]);
    }
    if (__any_sync(0xffffffffu, bad)) return false;
    if (sigmoid) {
#pragma unroll
        for (int i = 0; i < NPL; i++) p[i] = 1.f / (1.f + expf(-p[i]));
    } else {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        float part = 0.f;
#pragma unroll
        for (int i = 0; i < NPL; i++)
            if (lane + 32 * i < experts) {
                p[i] = expf(p[i] - mx);
                part += p[i];
            }
        const float total = route_warp_sum(part);
#pragma unroll
        for (int i = 0; i < NPL; i++) p[i] = p[i] / total;
    }
    uint32_t key[NPL]; // bits + 1; 0 once taken (or no expert)
#pragma unroll
    for (int i = 0; i < NPL; i++) key[i] = lane + 32 * i < experts ? __float_as_uint(p[i]) + 1u : 0u;
    float picked_sum = 0.f, mine = 0.f;
    for (uint32_t k = 0; k < used; k++) {
        uint32_t bk = 0, be = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < NPL; i++)
            if (key[i] > bk) { // ascending expert: ties keep the lower index
                bk = key[i];
                be = lane + 32 * i;
            }
        const uint32_t top = __reduce_max_sync(0xffffffffu, bk), win = __reduce_min_sync(0xffffffffu, bk == top ? be : 0xffffffffu);
        const float v = __uint_as_float(top - 1u);
        picked_sum += v;
        if (lane == k) {
            id = win;
            mine = v;
        }
#pragma unroll
        for (int i = 0; i < NPL; i++)
            if (win == lane + 32 * i) key[i] = 0u;
    }
    weight = norm ? mine / picked_sum : mine;
    return true;
}

// The shared expert's gate: logistic(x . w) of `hidden` values, by one warp.
__device__ __forceinline__ float route_gate(const float *__restrict__ x, const float *__restrict__ w, uint32_t hidden, uint32_t lane) {
    float dot = 0.f;
    if (hidden % 4 == 0) {
#pragma unroll 8
        for (uint32_t i = lane; i < hidden / 4; i += 32) {
            const float4 a = reinterpret_cast<const float4 *>(x)[i], b = reinterpret_cast<const float4 *>(w)[i];
            dot = fmaf(a.x, b.x, dot);
            dot = fmaf(a.y, b.y, dot);
            dot = fmaf(a.z, b.z, dot);
            dot = fmaf(a.w, b.w, dot);
        }
    } else {
        for (uint32_t i = lane; i < hidden; i += 32) dot = fmaf(x[i], w[i], dot);
    }
    dot = route_warp_sum(dot);
    return 1.f / (1.f + expf(-dot));
}

} // namespace fqk
