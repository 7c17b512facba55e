// Pieces of the Q8_0 integer dot product shared by gemv_q8.cu and moe_decode.cu.
#pragma once
#include "blocks.cuh"

namespace fqk {

// One block of 32 activations by one warp, lane = value: x' = round(v * s) = 256 hi + lo, both halves signed bytes,
// s = 2^e the largest power of two with amax * s <= 32639: amax = f * 2^ex with f in [0.5, 1), so e = 15 - ex, one less
// when f * 2^15 > 32639.  Exponents straight from the float's bits.  `hi`, `lo`: the block's 32 bytes; `isc`: 1 / s, or
// NaN when a value of the block is not finite.
__device__ __forceinline__ void q8_quantize_block(float v, uint32_t lane, int8_t *hi, int8_t *lo, float *isc) {
    float amax = fabsf(v);
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
    if (!finite) q = 0; // the block's factor is NaN in that case
    const int h = (q + 128) >> 8;
    hi[lane] = (int8_t)h;
    lo[lane] = (int8_t)(q - (h << 8));
    if (lane == 0) *isc = finite ? __uint_as_float((uint32_t)(127 - e) << 23) : __int_as_float(0x7fc00000);
}

// Sixteen weights against the two planes of sixteen activations.
__device__ __forceinline__ int q8_dot16(const uint4 &q, const int4 &xh, const int4 &xl) {
    int dh = __dp4a((int)q.x, xh.x, 0), dl = __dp4a((int)q.x, xl.x, 0);
    dh = __dp4a((int)q.y, xh.y, dh), dl = __dp4a((int)q.y, xl.y, dl);
    dh = __dp4a((int)q.z, xh.z, dh), dl = __dp4a((int)q.z, xl.z, dl);
    dh = __dp4a((int)q.w, xh.w, dh), dl = __dp4a((int)q.w, xl.w, dl);
    return dh * 256 + dl;
}

} // namespace fqk
