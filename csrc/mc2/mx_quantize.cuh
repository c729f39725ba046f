// One 1 x 32 block of bf16 values -> e4m3 values and the e8m0 scale (OCP MX v1.0: scale = 2^(floor(log2(amax)) - 8), round to nearest even, saturating). The quantiser and
// the products that quantise their activations themselves share it.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>

namespace hccl {
namespace mc2 {

__device__ __forceinline__ uint8_t QuantizeBlock(const uint4 (&raw)[4], uint4 (&out)[2])
{
    float v[32];
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 *h = (const __nv_bfloat162 *)&raw[i];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float2 f = __bfloat1622float2(h[j]);
            v[i * 8 + 2 * j] = f.x; v[i * 8 + 2 * j + 1] = f.y;
            amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
        }
    }
    // biased exponent of amax (finite inputs assumed; NaN / Inf saturate through the conversion below)
    int e = (int)((__float_as_uint(amax) >> 23) & 0xff);         // floor(log2(amax)) + 127 for normal amax; 0 for zero / denormal
    int se = e - 8;                                              // scale exponent, biased
    if (se < 0) se = 0;
    if (se > 254) se = 254;
    const float inv = __uint_as_float((uint32_t)(254 - se) << 23);    // 2^(127 - se): exact reciprocal of the scale (se = 0 gives 2^127)
    uint32_t packed[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[i * 4] * inv, v[i * 4 + 1] * inv), __NV_SATFINITE, __NV_E4M3);
        __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[i * 4 + 2] * inv, v[i * 4 + 3] * inv), __NV_SATFINITE, __NV_E4M3);
        packed[i] = (uint32_t)lo | ((uint32_t)hi << 16);
    }
    out[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    out[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
    return (uint8_t)se;
}

}  // namespace mc2
}  // namespace hccl
