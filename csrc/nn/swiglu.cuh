// Arithmetic of SwiGLU on eight bf16 values at a time, for the element-wise kernels and the epilogues that do the same: one place, so that they give the same bits.
#pragma once
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>

namespace hccl {
namespace nn {

__device__ __forceinline__ void Unpack8(const uint4 &r, float (&f)[8])
{
    const __nv_bfloat162 *h = (const __nv_bfloat162 *)&r;
#pragma unroll
    for (int j = 0; j < 4; ++j) { const float2 p = __bfloat1622float2(h[j]); f[2 * j] = p.x; f[2 * j + 1] = p.y; }
}
__device__ __forceinline__ uint4 Pack8(const float (&f)[8])
{
    uint4 o;
    __nv_bfloat162 t0 = __floats2bfloat162_rn(f[0], f[1]), t1 = __floats2bfloat162_rn(f[2], f[3]);
    __nv_bfloat162 t2 = __floats2bfloat162_rn(f[4], f[5]), t3 = __floats2bfloat162_rn(f[6], f[7]);
    o.x = *(uint32_t *)&t0; o.y = *(uint32_t *)&t1; o.z = *(uint32_t *)&t2; o.w = *(uint32_t *)&t3;
    return o;
}

// a / b for a finite a and 1 <= b < 2^100: Newton's iteration on the reciprocal and one correction by the residual (P. W. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990). No branch, so that the divisions of several values overlap; the general division has one per value.
__device__ __forceinline__ float Quotient(float a, float b)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    r = __fmaf_rn(__fmaf_rn(-b, r, 1.f), r, r);
    const float q = __fmul_rn(a, r);
    return copysignf(__fmaf_rn(__fmaf_rn(-b, q, a), r, q), a);         // a zero keeps its sign
}
// The same for any value of x, out of line: a / (1 + exp(-x)).
static __device__ __noinline__ float OverOnePlusExp(float a, float x) { return __fdiv_rn(a, __fadd_rn(1.f, expf(-x))); }

// Whether all eight magnitudes are below 64: then 1 + exp(-x) is below 2^100. Infinities and NaN are not.
__device__ __forceinline__ bool Below64(const uint4 &v)
{
    const uint32_t m = __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu));
    return (m & 0xffffu) < 0x4280u && m >> 16 < 0x4280u;
}

// silu(gate) * up. silu is rounded to bf16 before the product, as two separate operations round it. The product of two bf16 values is exact in 32 bits, so
// a packed multiplication rounds it the same way.
__device__ __forceinline__ uint4 SwiGlu8(const uint4 &gate, const uint4 &up)
{
    float g[8];
    Unpack8(gate, g);
    const __nv_bfloat162 *u = (const __nv_bfloat162 *)&up;
    uint4 o;
    __nv_bfloat162 *ov = (__nv_bfloat162 *)&o;
    if (Below64(gate)) {
#pragma unroll
        for (int x = 0; x < 8; ++x) g[x] = Quotient(g[x], __fadd_rn(1.f, expf(-g[x])));
    } else {
#pragma unroll
        for (int x = 0; x < 8; ++x) g[x] = OverOnePlusExp(g[x], g[x]);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) ov[x] = __hmul2_rn(__floats2bfloat162_rn(g[2 * x], g[2 * x + 1]), u[x]);
    return o;
}

// d = gradient of silu(gate) * up -> gradients of gate and up. OVERLAP: divisions that overlap, for the few warps of an epilogue (2048 x 14336 x 4096 backward 285 us
// with general ones, 224 so; with eight warps 214); a kernel with many warps has nothing to gain (51.5 us, 53.5 for the registers). Products and sums are spelled out, so that no compilation contracts them differently.
template <bool OVERLAP> __device__ __forceinline__ void SwiGluGrad8(const uint4 &d8, const uint4 &gate, const uint4 &up, uint4 *dGate, uint4 *dUp)
{
    float g[8], u[8], d[8], sg[8];
    Unpack8(gate, g);
    Unpack8(up, u);
    Unpack8(d8, d);
    if (!OVERLAP) {
#pragma unroll
        for (int x = 0; x < 8; ++x) sg[x] = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-g[x])));
    } else if (Below64(gate)) {
#pragma unroll
        for (int x = 0; x < 8; ++x) sg[x] = Quotient(1.f, __fadd_rn(1.f, expf(-g[x])));
    } else {
#pragma unroll
        for (int x = 0; x < 8; ++x) sg[x] = OverOnePlusExp(1.f, g[x]);
    }
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const float si = __fmul_rn(g[x], sg[x]);
        const float dg = __fmul_rn(__fmul_rn(__fmul_rn(d[x], u[x]), sg[x]), __fmaf_rn(g[x], __fsub_rn(1.f, sg[x]), 1.f));
        u[x] = __fmul_rn(d[x], si);
        g[x] = dg;
    }
    *dGate = Pack8(g);
    *dUp = Pack8(u);
}

}  // namespace nn
}  // namespace hccl
