// bvh_quant_lanes.cuh — tlas_quantise (bvh_quant.h) by eight lanes, a child
// slot's box per lane, with the same bytes.  A thread that quantises a whole node
// evaluates 48 planes in double precision one after the other; here a lane
// evaluates the six of its own child and the frame's axes are lanes 0 to 2.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bvh_layout.h"

namespace bsm {

constexpr uint32_t kWideLanes = 8;

__device__ __forceinline__ double pow2d(int e) { return __hiloint2double((e + 1023) << 20, 0); }

// quant_exponent_hd: the smallest e with 253 * 2^e >= extent, biased and clamped.
__device__ __forceinline__ int quant_exponent_dev(float extent) {
    const double ext = (double)extent > 1e-30 ? (double)extent : 1e-30;
    int e = ((__double2hiint(ext) >> 20) & 0x7ff) - 1023 - 7;
    while (253.0 * pow2d(e - 1) >= ext) --e;
    while (253.0 * pow2d(e) < ext) ++e;
    const int biased = e + 127;
    return biased < 1 ? 1 : (biased > 254 ? 254 : biased);
}

// Reductions over a group of eight lanes; all lanes of the warp take part.
__device__ __forceinline__ float wide_min(float x) {
    for (int o = 1; o < (int)kWideLanes; o <<= 1) x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}
__device__ __forceinline__ float wide_max(float x) {
    for (int o = 1; o < (int)kWideLanes; o <<= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}
__device__ __forceinline__ uint32_t wide_or(uint32_t x) {
    for (int o = 1; o < (int)kWideLanes; o <<= 1) x |= __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Writes the frame (origin and exponents) and the planes of the valid lanes'
// children into the node image at `image` (80 bytes, shared or global memory);
// [nlo, nhi] is the union of the valid boxes, `any` whether there is one.
__device__ __forceinline__ void quantise_lanes(uint8_t* image, bool valid, uint32_t slot, bool any, const float* lo,
                                               const float* hi, const float* nlo, const float* nhi) {
    const uint32_t lane = threadIdx.x & 31u, sub = lane % kWideLanes, shift = lane - sub;
    int e = 0;
    float org = 0.0f;
    if (sub < 3u && any) {
        const float l = sub == 0 ? nlo[0] : sub == 1 ? nlo[1] : nlo[2], h = sub == 0 ? nhi[0] : sub == 1 ? nhi[1] : nhi[2];
        e = quant_exponent_dev(h - l);
        const double at = (double)l - pow2d(e - 127);
        org = (float)at;
        while ((double)org > at) org = nextafterf(org, -INFINITY);
        reinterpret_cast<float*>(image)[sub] = org;
        image[12 + sub] = (uint8_t)e;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int ek = __shfl_sync(0xffffffffu, e, (int)shift + k);
        const float ok = __shfl_sync(0xffffffffu, org, (int)shift + k);
        if (!valid) continue;
        const double sc = pow2d(ek - 127), inv = pow2d(127 - ek), o = (double)ok;
        double l = floor(((double)lo[k] - o) * inv) - 1.0;
        double h = ceil(((double)hi[k] - o) * inv) + 1.0;
        l = l < 0.0 ? 0.0 : (l > 255.0 ? 255.0 : l);
        h = h < 0.0 ? 0.0 : (h > 255.0 ? 255.0 : h);
        while (l > 0.0 && o + l * sc > (double)lo[k]) l -= 1.0;
        while (h < 255.0 && o + h * sc < (double)hi[k]) h += 1.0;
        image[32 + 8 * k + slot] = (uint8_t)l;
        image[56 + 8 * k + slot] = (uint8_t)h;
    }
}

}  // namespace bsm
