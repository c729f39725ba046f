// Element-wise parts of a decoder block (RMSNorm, rotary embedding of a packed QKV projection, SwiGLU, vocabulary-parallel cross
// entropy), forward and backward, bf16 in and out with fp32 arithmetic. All are bound by memory: each reads its inputs once and
// writes its outputs once, 16 bytes per thread and load, in place of chains of element-wise framework kernels that write every
// intermediate (most of them in fp32) back to memory. A Llama-3-8B block, 2048 tokens, forward and backward on one B200: 4791 us with those
// chains, 3508 with these kernels. HCCL has no counterpart; the decoder exists for the end-to-end benchmarks.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <algorithm>
#include "../common/launch_count.h"
#include "../common/log.h"
#include "hccl/hccl_nn.h"
#include "swiglu.cuh"

namespace hccl {
namespace nn {

namespace {

constexpr int kThreads = 256;

// Every kernel here is launched to start while the one before it drains (programmatic stream serialization): its blocks take the places that become free, and wait here before
// they touch memory. The next kernel may do the same. Us a sequence among others on one B200, without / with it: SwiGLU and its gradient at 1000 x 7168 24.6 / 19.6, norm, product and norm
// gradient at 1000 x 2048 28.1 / 22.5, at 2048 x 4096 70.1 / 67.7. In a graph 20.1 / 19.0, 21.4 / 21.4 and 71 / 74: there the launches follow one another closely anyway.
__device__ __forceinline__ void WaitForOthers()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// a + b, each sum rounded to bf16
__device__ __forceinline__ uint4 Add8(const uint4 &a, const uint4 &b)
{
    float f[8], g[8];
    Unpack8(a, f);
    Unpack8(b, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] += g[j];
    return Pack8(f);
}

// Sum over the TPR threads that share a row: a warp (TPR = 32) or the whole block.
template <int TPR> __device__ __forceinline__ float RowSum(float v, float *red)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (TPR == 32) return v;
    __syncthreads();                                     // red may still be read from the previous sum
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < TPR / 32; ++w) s += red[w];
    return s;
}

// y = x * rsqrt(mean(x^2) + eps) * w. A row is shared by TPR threads. Up to two vectors per thread (NV) stay in registers between the sum and the
// result; wider rows (NV = 0) are read again from L1 / L2, which leaves the registers to more rows in flight. KEEP: x and w are copied on the
// way for a backward pass that may come after they were changed. ADD: the row is x + d, rounded to bf16 as an addition by itself rounds it, and its copy is
// the sum (the residual stream of a decoder goes on with it). Bound by memory: 2048 x 4096 with copies (48 MB) on one B200 14.3 us from a cold L2,
// 16.4 with a second load of the row; 1000 x 8192 without copies 12.3 with it, 14.2 from registers.
template <int TPR, int NV, bool KEEP, bool ADD = false>
__global__ void __launch_bounds__(kThreads) RmsNormKernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ d, const __nv_bfloat16 *__restrict__ w,
                                                         __nv_bfloat16 *__restrict__ y, float *__restrict__ rstd, __nv_bfloat16 *xKept, __nv_bfloat16 *__restrict__ wKept, uint32_t T,
                                                         uint32_t H, float eps)
{
    WaitForOthers();
    __shared__ float red[kThreads / 32];
    const uint32_t row = blockIdx.x * (kThreads / TPR) + threadIdx.x / TPR, lane = threadIdx.x % TPR;
    if (row >= T) return;                                // whole warps (TPR = 32) or no thread at all (one row per block)
    const uint4 *xr = (const uint4 *)(x + (size_t)row * H), *dr = (const uint4 *)(d + (size_t)row * H), *wr = (const uint4 *)w;
    uint4 xv[NV ? NV : 1], dv[NV ? NV : 1];
    float s = 0.f;
    auto square = [&](uint32_t v, const uint4 &raw) {
        if (KEEP) ((uint4 *)(xKept + (size_t)row * H))[v] = raw;
        float f[8];
        Unpack8(raw, f);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += f[j] * f[j];
    };
    if (NV) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (lane + i * TPR < H / 8) {
                xv[i] = xr[lane + i * TPR];
                if (ADD) dv[i] = dr[lane + i * TPR];
            }
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (lane + i * TPR < H / 8) {
                if (ADD) xv[i] = Add8(xv[i], dv[i]);
                square(lane + i * TPR, xv[i]);
            }
    } else {
        for (uint32_t v = lane; v < H / 8; v += TPR) {
            const uint4 raw = ADD ? Add8(xr[v], dr[v]) : xr[v];   // a value: 9000 x 8192 without copies 45.4 us, 55.6 with a reference to memory handed on
            square(v, raw);
        }
    }
    const float r = rsqrtf(RowSum<TPR>(s, red) / (float)H + eps);
    if (lane == 0) rstd[row] = r;
    uint4 *yr = (uint4 *)(y + (size_t)row * H);
    auto scale = [&](uint32_t v, const uint4 &raw) {
        const uint4 wv = wr[v];
        if (KEEP && wKept && row == 0) ((uint4 *)wKept)[v] = wv;
        float f[8], g[8];
        Unpack8(raw, f);
        Unpack8(wv, g);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * r * g[j];
        yr[v] = Pack8(f);
    };
    if (NV) {
#pragma unroll
        for (int i = 0; i < NV; ++i) if (lane + i * TPR < H / 8) scale(lane + i * TPR, xv[i]);
    } else {
        for (uint32_t v = lane; v < H / 8; v += TPR) {
            const uint4 raw = ADD ? ((const uint4 *)(xKept + (size_t)row * H))[v] : xr[v];       // its own store of the first pass
            scale(v, raw);
        }
    }
}

// dx = r * (dy * w - xhat * mean(dy * w * xhat)), xhat = x * r; dw = sum over rows of dy * xhat. A thread owns NV vectors of columns of
// every row its block walks over (with a stride of the grid): x, dy and w of a row are loaded once and stay in registers between the
// row sum and the result, and so does the thread's part of dw, which goes to partial[block] at the end; the next row is on its way
// meanwhile. ADD: dx + res, the gradient that reached x by another way, rounded as an addition by itself rounds it. A second kernel adds the blocks in a fixed order: the same bits on every run. 2048 x 4096 on one B200, both kernels from a cold L2:
// 23.3 us, 31.6 without the early loads, with three blocks per SM and the sums below at one column per thread.
template <int TPR, int NV, bool ADD>
__global__ void __launch_bounds__(kThreads) RmsNormBwdKernel(const __nv_bfloat16 *__restrict__ dy, const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ w,
                                                            const float *__restrict__ rstd, const __nv_bfloat16 *__restrict__ res, __nv_bfloat16 *__restrict__ dx, float *__restrict__ partial, uint32_t T,
                                                            uint32_t H)
{
    WaitForOthers();
    __shared__ float red[kThreads / 32];
    constexpr uint32_t kRows = kThreads / TPR;
    __shared__ float acc[TPR == 32 ? kRows * NV * 256 : 1];   // warps of a block that share the columns: their parts of dw
    const uint32_t group = threadIdx.x / TPR, lane = threadIdx.x % TPR;
    uint4 wv[NV];
    float part[NV][8];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint32_t v = lane + i * TPR;
        wv[i] = v < H / 8 ? ((const uint4 *)w)[v] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int j = 0; j < 8; ++j) part[i][j] = 0.f;
    }
    uint4 nx[NV], nd[NV];
    float nr = 0.f;
    auto fetch = [&](uint32_t row) {
        const uint4 *xr = (const uint4 *)(x + (size_t)row * H), *dr = (const uint4 *)(dy + (size_t)row * H);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t v = lane + i * TPR;
            nx[i] = v < H / 8 ? xr[v] : make_uint4(0, 0, 0, 0);
            nd[i] = v < H / 8 ? dr[v] : make_uint4(0, 0, 0, 0);
        }
        nr = rstd[row];
    };
    constexpr bool kEarly = NV <= 4;                     // more would not fit the registers
    const uint32_t step = gridDim.x * kRows;
    uint32_t row = blockIdx.x * kRows + group;
    if (kEarly && row < T) fetch(row);
    for (; row < T; row += step) {
        uint4 xv[NV], dv[NV];
        if (!kEarly) fetch(row);
        const float r = nr;
#pragma unroll
        for (int i = 0; i < NV; ++i) { xv[i] = nx[i]; dv[i] = nd[i]; }
        uint4 rv[NV];
        if (ADD) {
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (lane + i * TPR < H / 8) rv[i] = ((const uint4 *)(res + (size_t)row * H))[lane + i * TPR];
        }
        if (kEarly && row + step < T) fetch(row + step);
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            float f[8], g[8], d[8];
            Unpack8(xv[i], f);
            Unpack8(wv[i], g);
            Unpack8(dv[i], d);
#pragma unroll
            for (int j = 0; j < 8; ++j) s += d[j] * g[j] * (f[j] * r);
        }
        const float m = RowSum<TPR>(s, red) / (float)H;
        uint4 *o = (uint4 *)(dx + (size_t)row * H);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            float f[8], g[8], d[8];
            Unpack8(xv[i], f);
            Unpack8(wv[i], g);
            Unpack8(dv[i], d);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float xh = f[j] * r;
                f[j] = r * (d[j] * g[j] - xh * m);
                part[i][j] += d[j] * xh;
            }
            if (lane + i * TPR < H / 8) o[lane + i * TPR] = ADD ? Add8(Pack8(f), rv[i]) : Pack8(f);
        }
    }
    float *out = partial + (size_t)blockIdx.x * H;
    if (TPR == kThreads) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t v = lane + i * TPR;
            if (v >= H / 8) continue;
            ((float4 *)out)[v * 2] = make_float4(part[i][0], part[i][1], part[i][2], part[i][3]);
            ((float4 *)out)[v * 2 + 1] = make_float4(part[i][4], part[i][5], part[i][6], part[i][7]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[((group * NV + i) * 8 + j) * 32 + lane] = part[i][j];
        __syncthreads();
        for (uint32_t c = threadIdx.x; c < H; c += kThreads) {
            const uint32_t v = c / 8, at = ((v / 32) * 8 + c % 8) * 32 + v % 32;
            float s = 0.f;
            for (uint32_t g = 0; g < kRows; ++g) s += acc[g * NV * 256 + at];
            out[c] = s;
        }
    }
}

// out[c] = sum over parts of partial[part][c]: 32 columns per block, four per load (VEC: 16-byte aligned) or turn, 32 threads per column group, added up in a
// fixed order.
template <bool VEC> __global__ void __launch_bounds__(kThreads) SumPartsKernel(const float *__restrict__ partial, __nv_bfloat16 *__restrict__ out, uint32_t parts, uint32_t H)
{
    WaitForOthers();
    __shared__ float4 sm[32][8];
    const uint32_t g = threadIdx.x & 7, q = threadIdx.x >> 3, c = blockIdx.x * 32 + g * 4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < H) {                                         // H is a multiple of 8: whole groups
#pragma unroll 4
        for (uint32_t p = q; p < parts; p += 32) {
            const float *at = partial + (size_t)p * H + c;
            const float4 v = VEC ? *(const float4 *)at : make_float4(at[0], at[1], at[2], at[3]);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
    }
    sm[q][g] = s;
    __syncthreads();
    if (threadIdx.x < 32 && blockIdx.x * 32 + threadIdx.x < H) {
        float t = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) t += ((const float *)sm[j])[threadIdx.x];
        out[blockIdx.x * 32 + threadIdx.x] = __float2bfloat16(t);
    }
}

// Packed projection [T, (hq + 2 hk) * D] -> rotated q [T, hq, D], rotated k [T, hk, D], v [T, hk, D]; BWD runs the other way with the
// transposed rotation. A thread takes 8 elements of the first half of a head and the 8 they are paired with in the second half.
template <bool BWD>
__global__ void __launch_bounds__(kThreads) RopeQkvKernel(__nv_bfloat16 *__restrict__ qkv, __nv_bfloat16 *__restrict__ q, __nv_bfloat16 *__restrict__ k,
                                                         __nv_bfloat16 *__restrict__ v, const float *__restrict__ cosT, const float *__restrict__ sinT, uint32_t T,
                                                         uint32_t seq, uint32_t hq, uint32_t hk, uint32_t D)
{
    WaitForOthers();
    const uint32_t half = D / 2, perHead = half / 8, heads = hq + 2 * hk, perTok = heads * perHead;
    const uint64_t idx = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (idx >= (uint64_t)T * perTok) return;
    const uint32_t t = (uint32_t)(idx / perTok), in = (uint32_t)(idx % perTok), h = in / perHead, j = (in % perHead) * 8;
    __nv_bfloat16 *pk = qkv + ((size_t)t * heads + h) * D + j;
    __nv_bfloat16 *un = (h < hq ? q + ((size_t)t * hq + h) * D : h < hq + hk ? k + ((size_t)t * hk + (h - hq)) * D : v + ((size_t)t * hk + (h - hq - hk)) * D) + j;
    const __nv_bfloat16 *src = BWD ? un : pk;
    __nv_bfloat16 *dst = BWD ? pk : un;
    const uint4 r1 = *(const uint4 *)src, r2 = *(const uint4 *)(src + half);
    if (h >= hq + hk) {
        *(uint4 *)dst = r1;
        *(uint4 *)(dst + half) = r2;
        return;
    }
    float a[8], b[8], c[8], s[8];
    Unpack8(r1, a);
    Unpack8(r2, b);
    const size_t at = (size_t)(t % seq) * half + j;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const float4 cc = *(const float4 *)(cosT + at + 4 * x), ss = *(const float4 *)(sinT + at + 4 * x);
        c[4 * x] = cc.x; c[4 * x + 1] = cc.y; c[4 * x + 2] = cc.z; c[4 * x + 3] = cc.w;
        s[4 * x] = ss.x; s[4 * x + 1] = ss.y; s[4 * x + 2] = ss.z; s[4 * x + 3] = ss.w;
    }
    float o1[8], o2[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const float sn = BWD ? -s[x] : s[x];
        // products rounded before the sum, as the element-wise form does it
        o1[x] = __fsub_rn(__fmul_rn(a[x], c[x]), __fmul_rn(b[x], sn));
        o2[x] = __fadd_rn(__fmul_rn(b[x], c[x]), __fmul_rn(a[x], sn));
    }
    *(uint4 *)dst = Pack8(o1);
    *(uint4 *)(dst + half) = Pack8(o2);
}

// gu = [T, 2F] (gate | up): h = silu(gate) * up, the bits of the plain form. What bounds it is instructions: 2048 x 14336 on one B200 33.1 us, 35.1 with a general division per value (memory
// alone 27); 4096 x 28672 120, 131. Index divisions in 64 bits cost another fifth. Index is 64 bits wide where the vectors need it.
template <class Index>
__global__ void __launch_bounds__(kThreads) SwiGluKernel(const __nv_bfloat16 *__restrict__ gu, __nv_bfloat16 *__restrict__ h, uint64_t vecs, uint32_t F)
{
    WaitForOthers();
    const Index idx = (Index)blockIdx.x * kThreads + threadIdx.x;
    if (idx >= vecs) return;
    const uint32_t per = F / 8;
    const Index t = idx / per, j = idx - t * per;
    const uint4 *row = (const uint4 *)gu + (uint64_t)t * 2 * per;
    const uint4 gv = row[j], uv = row[per + j];
    ((uint4 *)h)[idx] = SwiGlu8(gv, uv);
}

__global__ void __launch_bounds__(kThreads) SwiGluBwdKernel(const __nv_bfloat16 *__restrict__ dh, const __nv_bfloat16 *__restrict__ gu, __nv_bfloat16 *__restrict__ dgu,
                                                           uint64_t vecs, uint32_t F)
{
    WaitForOthers();
    const uint64_t idx = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (idx >= vecs) return;
    const uint32_t per = F / 8;
    const uint64_t t = idx / per, j = idx % per;
    const uint4 *row = (const uint4 *)(gu + t * 2 * F);
    uint4 *out = (uint4 *)(dgu + t * 2 * F);
    SwiGluGrad8<false>(((const uint4 *)dh)[idx], row[j], row[per + j], &out[j], &out[per + j]);
}

// Cross entropy over vocabulary shards, one block per row. STEP 0: row maximum. STEP 1: sum of exp(l - max) and the target's
// logit - max (0 on ranks that do not own it). STEP 2: gradient. The collectives over the shards run between the steps.
template <int STEP, bool VEC>
__global__ void __launch_bounds__(kThreads) XentKernel(const __nv_bfloat16 *__restrict__ logits, const int64_t *__restrict__ targets, int64_t vocabStart, float *__restrict__ mx,
                                                      float *__restrict__ packed, const float *__restrict__ gOut, __nv_bfloat16 *__restrict__ grad, uint32_t T, uint32_t V)
{
    WaitForOthers();
    __shared__ float red[kThreads / 32];
    const uint32_t t = blockIdx.x;
    const __nv_bfloat16 *row = logits + (size_t)t * V;
    if (STEP == 0) {
        float m = -INFINITY;
        bool nan = false;                                // a NaN logit makes the maximum NaN, as a plain maximum over the row does
        auto take = [&](float f) { nan |= isnan(f); m = fmaxf(m, f); };
        if (VEC) {
            for (uint32_t v = threadIdx.x; v < V / 8; v += kThreads) {
                float f[8];
                Unpack8(((const uint4 *)row)[v], f);
#pragma unroll
                for (int j = 0; j < 8; ++j) take(f[j]);
            }
        } else {
            for (uint32_t v = threadIdx.x; v < V; v += kThreads) take(__bfloat162float(row[v]));
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        const int anyNan = __syncthreads_or(nan ? 1 : 0);
        if (threadIdx.x == 0) {
            for (int w = 1; w < kThreads / 32; ++w) m = fmaxf(m, red[w]);
            mx[t] = anyNan ? NAN : m;
        }
        return;
    }
    const float m = mx[t];
    const int64_t target = targets[t] - vocabStart;
    if (STEP == 1) {
        float s = 0.f;
        if (VEC) {
            for (uint32_t v = threadIdx.x; v < V / 8; v += kThreads) {
                float f[8];
                Unpack8(((const uint4 *)row)[v], f);
#pragma unroll
                for (int j = 0; j < 8; ++j) s += expf(f[j] - m);
            }
        } else {
            for (uint32_t v = threadIdx.x; v < V; v += kThreads) s += expf(__bfloat162float(row[v]) - m);
        }
        s = RowSum<kThreads>(s, red);
        if (threadIdx.x == 0) {
            packed[t] = s;
            packed[T + t] = target >= 0 && target < (int64_t)V ? __bfloat162float(row[target]) - m : 0.f;
        }
        return;
    }
    const float denom = packed[t], scale = gOut[0] / (float)T;
    __nv_bfloat16 *out = grad + (size_t)t * V;
    if (VEC) {
        for (uint32_t v = threadIdx.x; v < V / 8; v += kThreads) {
            float f[8];
            Unpack8(((const uint4 *)row)[v], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = (expf(f[j] - m) / denom - ((int64_t)(v * 8 + j) == target ? 1.f : 0.f)) * scale;
            ((uint4 *)out)[v] = Pack8(f);
        }
    } else {
        for (uint32_t v = threadIdx.x; v < V; v += kThreads)
            out[v] = __float2bfloat16((expf(__bfloat162float(row[v]) - m) / denom - ((int64_t)v == target ? 1.f : 0.f)) * scale);
    }
}

// The cross entropy of one rank up to the loss of every row: what steps 0 and 1 compute, the rows' losses, and copies of logits and targets for a backward pass that may come after
// they were changed. The second walk over a row finds it in L2. 2048 x 128256 logits: the copy alone, as an operation of its own, reads and writes 1 GB.
template <bool VEC>
__global__ void __launch_bounds__(kThreads) XentLossKernel(const __nv_bfloat16 *__restrict__ logits, const int64_t *__restrict__ targets, int64_t vocabStart, float *__restrict__ mx,
                                                          float *__restrict__ packed, float *__restrict__ rowLoss, __nv_bfloat16 *__restrict__ kept, int64_t *__restrict__ keptTargets,
                                                          uint32_t T, uint32_t V)
{
    WaitForOthers();
    __shared__ float red[kThreads / 32];
    const uint32_t t = blockIdx.x;
    const __nv_bfloat16 *row = logits + (size_t)t * V;
    float m = -INFINITY;
    bool nan = false;                                    // a NaN logit makes the maximum NaN, as a plain maximum over the row does
    auto take = [&](float f) { nan |= isnan(f); m = fmaxf(m, f); };
    if (VEC) {
        for (uint32_t v = threadIdx.x; v < V / 8; v += kThreads) {
            const uint4 raw = ((const uint4 *)row)[v];
            if (kept) ((uint4 *)(kept + (size_t)t * V))[v] = raw;
            float f[8];
            Unpack8(raw, f);
#pragma unroll
            for (int j = 0; j < 8; ++j) take(f[j]);
        }
    } else {
        for (uint32_t v = threadIdx.x; v < V; v += kThreads) {
            const __nv_bfloat16 raw = row[v];
            if (kept) kept[(size_t)t * V + v] = raw;
            take(__bfloat162float(raw));
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    const int anyNan = __syncthreads_or(nan ? 1 : 0);
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) m = fmaxf(m, red[w]);
    if (anyNan) m = NAN;
    float s = 0.f;
    if (VEC) {
        for (uint32_t v = threadIdx.x; v < V / 8; v += kThreads) {
            float f[8];
            Unpack8(((const uint4 *)row)[v], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) s += expf(f[j] - m);
        }
    } else {
        for (uint32_t v = threadIdx.x; v < V; v += kThreads) s += expf(__bfloat162float(row[v]) - m);
    }
    s = RowSum<kThreads>(s, red);
    if (threadIdx.x == 0) {
        const int64_t target = targets[t] - vocabStart;
        const float at = target >= 0 && target < (int64_t)V ? __bfloat162float(row[target]) - m : 0.f;
        mx[t] = m;
        packed[t] = s;
        packed[T + t] = at;
        rowLoss[t] = logf(s) - at;
        if (keptTargets) keptTargets[t] = targets[t];
    }
}

// The mean over the rows, in a fixed order.
__global__ void __launch_bounds__(1024) MeanKernel(const float *__restrict__ rows, float *__restrict__ mean, uint32_t T)
{
    WaitForOthers();
    __shared__ float red[32];
    float s = 0.f;
    for (uint32_t t = threadIdx.x; t < T; t += 1024) s += rows[t];
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    s = red[threadIdx.x];
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *mean = s / (float)T;
}

// Gradient of an embedding by its few tokens: the block of a token that is the first of its id adds up the rows of all tokens with that id, in their order and in 32 bits.
// Every block looks at all ids (16 KB at most), where the general way sorts them in some ten launches. A common id is one block's walk over its rows, a load at a time: us a backward pass among others on
// one B200, general / this, 2048 tokens of hidden 256 random 92 / 47, half of them one id 658 / 220, all 1288 / 438; hidden 4096 118 / 69, 1288 / 563, 2469 / 1063.
constexpr uint32_t kEmbedTokens = 2048;
__global__ void __launch_bounds__(kThreads) EmbeddingGradKernel(const int64_t *__restrict__ ids, const __nv_bfloat16 *__restrict__ dy, __nv_bfloat16 *__restrict__ grad, uint32_t T,
                                                               uint32_t H, int64_t V)
{
    WaitForOthers();
    __shared__ uint32_t same[kEmbedTokens / 32];
    const uint32_t i = blockIdx.x;
    auto idOf = [&](uint32_t t) { const int64_t id = ids[t]; return id < 0 ? id + V : id; };      // as an index from the end
    const int64_t mine = idOf(i);
    if (mine < 0 || mine >= V) return;
    for (uint32_t t0 = 0; t0 < T; t0 += kThreads) {
        const uint32_t t = t0 + threadIdx.x, word = __ballot_sync(0xffffffffu, t < T && idOf(t) == mine);
        if ((threadIdx.x & 31) == 0 && t / 32 < kEmbedTokens / 32) same[t / 32] = word;
    }
    __syncthreads();
    for (uint32_t w = 0; w <= i / 32; ++w)
        if (w < i / 32 ? same[w] != 0 : (same[w] & ((1u << (i % 32)) - 1)) != 0) return;          // an earlier token does it
    const uint32_t v = blockIdx.y * kThreads + threadIdx.x;
    if (v >= H / 8) return;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (uint32_t w = i / 32; w < (T + 31) / 32; ++w)
        for (uint32_t bits = same[w]; bits; bits &= bits - 1) {
            float f[8];
            Unpack8(((const uint4 *)(dy + (size_t)(w * 32 + __ffs(bits) - 1) * H))[v], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] += f[j];
        }
    ((uint4 *)(grad + (size_t)mine * H))[v] = Pack8(acc);
}

bool Aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

template <class... Params, class... Args>
HcclResult Launch(const char *what, void (*kern)(Params...), dim3 grid, uint32_t threads, cudaStream_t stream, Args... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, (Params)args...);
    CountLaunch();
    if (e != cudaSuccess) { HCCL_ERROR("%s launch failed: %s", what, cudaGetErrorString(e)); (void)cudaGetLastError(); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

int Sms()
{
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
}

constexpr uint64_t kWarpRowMax = 1024;     // rows up to this wide are handled by a warp, wider ones by a block
constexpr uint64_t kNormMax = 12288;       // widest row: six vectors per thread of a block

template <int TPR, int NV>
HcclResult LaunchRmsNormBwd(const void *dy, const void *x, const void *w, const float *rstd, const void *res, void *dx, float *partial, uint32_t T, uint32_t H, uint32_t parts, cudaStream_t s)
{
    auto kern = res ? RmsNormBwdKernel<TPR, NV, true> : RmsNormBwdKernel<TPR, NV, false>;
    return Launch("RMSNorm backward", kern, parts, kThreads, s, (const __nv_bfloat16 *)dy, (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)w, rstd, (const __nv_bfloat16 *)res,
                  (__nv_bfloat16 *)dx, partial, T, H);
}

// 16-byte vectors of a row per thread
uint32_t NormVecs(uint32_t H)
{
    const uint32_t threads = H <= kWarpRowMax ? 32 : kThreads;
    return (H / 8 + threads - 1) / threads;
}

bool NormShapeOk(uint64_t T, uint64_t H) { return T > 0 && T <= 0x7fffffff && H > 0 && H % 8 == 0 && H <= kNormMax; }

// d: what is added to x first, or null
HcclResult LaunchRmsNorm(const void *x, const void *d, const void *w, void *y, float *rstd, void *xKept, void *wKept, uint64_t rows, uint64_t hidden, float eps, cudaStream_t stream)
{
    if (!x || !w || !y || !rstd) return HCCL_E_PTR;
    if (!NormShapeOk(rows, hidden) || !Aligned16(x) || !Aligned16(d) || !Aligned16(w) || !Aligned16(y) || !Aligned16(xKept) || !Aligned16(wKept)) return HCCL_E_PARA;
    const uint32_t T = (uint32_t)rows, H = (uint32_t)hidden;
    const bool warp = hidden <= kWarpRowMax;
    auto launch = [&](auto plain, auto keep, auto add) {
        auto kern = d ? add : xKept ? keep : plain;
        return Launch("RMSNorm", kern, warp ? (T + 7) / 8 : T, kThreads, stream, (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)d, (const __nv_bfloat16 *)w, (__nv_bfloat16 *)y, rstd,
                      (__nv_bfloat16 *)xKept, (__nv_bfloat16 *)wKept, T, H, eps);
    };
    const uint32_t nv = NormVecs(H);
    if (warp && nv == 1) return launch(RmsNormKernel<32, 1, false>, RmsNormKernel<32, 1, true>, RmsNormKernel<32, 1, true, true>);
    if (warp && nv == 2) return launch(RmsNormKernel<32, 2, false>, RmsNormKernel<32, 2, true>, RmsNormKernel<32, 2, true, true>);
    if (warp) return launch(RmsNormKernel<32, 0, false>, RmsNormKernel<32, 0, true>, RmsNormKernel<32, 0, true, true>);
    if (nv == 1) return launch(RmsNormKernel<kThreads, 1, false>, RmsNormKernel<kThreads, 1, true>, RmsNormKernel<kThreads, 1, true, true>);
    if (nv == 2) return launch(RmsNormKernel<kThreads, 2, false>, RmsNormKernel<kThreads, 2, true>, RmsNormKernel<kThreads, 2, true, true>);
    return launch(RmsNormKernel<kThreads, 0, false>, RmsNormKernel<kThreads, 0, true>, RmsNormKernel<kThreads, 0, true, true>);
}

}  // namespace
}  // namespace nn
}  // namespace hccl

using namespace hccl;
using namespace hccl::nn;

extern "C" {

HcclResult HcclRmsNorm(const void *x, const void *w, void *y, float *rstd, uint64_t rows, uint64_t hidden, float eps, cudaStream_t stream)
{
    return LaunchRmsNorm(x, nullptr, w, y, rstd, nullptr, nullptr, rows, hidden, eps, stream);
}

HcclResult HcclRmsNormKeep(const void *x, const void *w, void *y, float *rstd, void *xKept, void *wKept, uint64_t rows, uint64_t hidden, float eps, cudaStream_t stream)
{
    if (!xKept || !wKept) return HCCL_E_PTR;
    return LaunchRmsNorm(x, nullptr, w, y, rstd, xKept, wKept, rows, hidden, eps, stream);
}

HcclResult HcclRmsNormAdd(const void *x, const void *d, const void *w, void *sum, void *y, float *rstd, void *wKept, uint64_t rows, uint64_t hidden, float eps, cudaStream_t stream)
{
    if (!d || !sum) return HCCL_E_PTR;
    return LaunchRmsNorm(x, d, w, y, rstd, sum, wKept, rows, hidden, eps, stream);
}

uint64_t HcclRmsNormBwdParts(uint64_t rows, uint64_t hidden)
{
    const uint64_t perBlock = hidden <= kWarpRowMax ? kThreads / 32 : 1, nv = hidden ? NormVecs((uint32_t)hidden) : 1;
    return std::min<uint64_t>((rows + perBlock - 1) / perBlock, (uint64_t)Sms() * (nv == 1 ? 3 : nv == 2 ? 2 : 1));   // what the registers let an SM hold
}

HcclResult HcclRmsNormBwd(const void *dy, const void *x, const void *w, const float *rstd, void *dx, void *dw, float *partial, uint64_t rows, uint64_t hidden,
                          cudaStream_t stream)
{
    return HcclRmsNormBwdAdd(dy, x, w, rstd, nullptr, dx, dw, partial, rows, hidden, stream);
}

HcclResult HcclRmsNormBwdAdd(const void *dy, const void *x, const void *w, const float *rstd, const void *dSum, void *dx, void *dw, float *partial, uint64_t rows,
                             uint64_t hidden, cudaStream_t stream)
{
    if (!dy || !x || !w || !rstd || !dx || !dw || !partial) return HCCL_E_PTR;
    if (!NormShapeOk(rows, hidden) || !Aligned16(dy) || !Aligned16(x) || !Aligned16(w) || !Aligned16(dSum) || !Aligned16(dx)) return HCCL_E_PARA;
    const bool vec = Aligned16(partial);                 // rows up to kWarpRowMax are also taken with a workspace that is aligned to its elements alone
    if (((uintptr_t)partial & 3u) || (!vec && hidden > kWarpRowMax)) return HCCL_E_PARA;
    const uint32_t T = (uint32_t)rows, H = (uint32_t)hidden, parts = (uint32_t)HcclRmsNormBwdParts(rows, hidden);
    auto launch = [&](auto kern) { return kern(dy, x, w, rstd, dSum, dx, partial, T, H, parts, stream); };
    const uint32_t nv = NormVecs(H);
    if (hidden <= kWarpRowMax) CHK_RET(launch(nv == 1 ? LaunchRmsNormBwd<32, 1> : nv == 2 ? LaunchRmsNormBwd<32, 2> : LaunchRmsNormBwd<32, 4>));
    else CHK_RET(launch(nv == 1 ? LaunchRmsNormBwd<kThreads, 1> : nv == 2 ? LaunchRmsNormBwd<kThreads, 2> : nv <= 4 ? LaunchRmsNormBwd<kThreads, 4> : LaunchRmsNormBwd<kThreads, 6>));
    return Launch("RMSNorm weight gradient", vec ? SumPartsKernel<true> : SumPartsKernel<false>, (H + 31) / 32, kThreads, stream, partial, (__nv_bfloat16 *)dw, parts, H);
}

HcclResult HcclRopeQkv(void *qkv, void *q, void *k, void *v, const float *cosT, const float *sinT, uint64_t tokens, uint64_t seq, uint32_t qHeads, uint32_t kvHeads,
                       uint32_t headDim, int backward, cudaStream_t stream)
{
    if (!qkv || !q || !k || !v || !cosT || !sinT) return HCCL_E_PTR;
    if (tokens == 0 || tokens > 0x7fffffff || seq == 0 || seq > tokens || qHeads == 0 || kvHeads == 0 || headDim == 0 || headDim % 16) return HCCL_E_PARA;
    if (!Aligned16(qkv) || !Aligned16(q) || !Aligned16(k) || !Aligned16(v) || !Aligned16(cosT) || !Aligned16(sinT)) return HCCL_E_PARA;
    const uint64_t items = tokens * (qHeads + 2 * kvHeads) * (headDim / 16), blocks = (items + kThreads - 1) / kThreads;
    if (blocks > 0x7fffffff) return HCCL_E_PARA;
    auto kern = backward ? RopeQkvKernel<true> : RopeQkvKernel<false>;
    return Launch("rotary embedding", kern, (uint32_t)blocks, kThreads, stream, (__nv_bfloat16 *)qkv, (__nv_bfloat16 *)q, (__nv_bfloat16 *)k, (__nv_bfloat16 *)v, cosT, sinT,
                  (uint32_t)tokens, (uint32_t)seq, qHeads, kvHeads, headDim);
}

HcclResult HcclSwiGlu(const void *gateUp, void *h, uint64_t rows, uint64_t ffn, cudaStream_t stream)
{
    if (!gateUp || !h) return HCCL_E_PTR;
    const uint64_t vecs = rows * (ffn / 8), blocks = (vecs + kThreads - 1) / kThreads;
    if (rows == 0 || ffn == 0 || ffn % 8 || ffn > 0x7fffffff || blocks > 0x7fffffff || !Aligned16(gateUp) || !Aligned16(h)) return HCCL_E_PARA;
    auto kern = (blocks + 1) * kThreads <= 0xffffffffull ? SwiGluKernel<uint32_t> : SwiGluKernel<uint64_t>;
    return Launch("SwiGLU", kern, (uint32_t)blocks, kThreads, stream, (const __nv_bfloat16 *)gateUp, (__nv_bfloat16 *)h, vecs, (uint32_t)ffn);
}

HcclResult HcclSwiGluBwd(const void *dh, const void *gateUp, void *dGateUp, uint64_t rows, uint64_t ffn, cudaStream_t stream)
{
    if (!dh || !gateUp || !dGateUp) return HCCL_E_PTR;
    const uint64_t vecs = rows * (ffn / 8), blocks = (vecs + kThreads - 1) / kThreads;
    if (rows == 0 || ffn == 0 || ffn % 8 || ffn > 0x7fffffff || blocks > 0x7fffffff || !Aligned16(dh) || !Aligned16(gateUp) || !Aligned16(dGateUp)) return HCCL_E_PARA;
    return Launch("SwiGLU backward", SwiGluBwdKernel, (uint32_t)blocks, kThreads, stream, (const __nv_bfloat16 *)dh, (const __nv_bfloat16 *)gateUp, (__nv_bfloat16 *)dGateUp, vecs,
                  (uint32_t)ffn);
}

HcclResult HcclXent(int step, const void *logits, const int64_t *targets, int64_t vocabStart, float *rowMax, float *packed, const float *gradOut, void *grad, uint64_t rows,
                    uint64_t vocab, cudaStream_t stream)
{
    if (!logits || !rowMax || (step > 0 && (!targets || !packed)) || (step == 2 && (!gradOut || !grad))) return HCCL_E_PTR;
    if (step < 0 || step > 2 || rows == 0 || rows > 0x7fffffff || vocab == 0 || vocab > 0x7fffffff) return HCCL_E_PARA;
    const bool vec = vocab % 8 == 0 && Aligned16(logits) && (step != 2 || Aligned16(grad));
    auto kern = step == 0 ? (vec ? XentKernel<0, true> : XentKernel<0, false>) : step == 1 ? (vec ? XentKernel<1, true> : XentKernel<1, false>)
                                                                                         : (vec ? XentKernel<2, true> : XentKernel<2, false>);
    return Launch("cross entropy", kern, (uint32_t)rows, kThreads, stream, (const __nv_bfloat16 *)logits, targets, vocabStart, rowMax, packed, gradOut,
                  (__nv_bfloat16 *)grad, (uint32_t)rows, (uint32_t)vocab);
}

HcclResult HcclXentLoss(const void *logits, const int64_t *targets, int64_t vocabStart, float *rowMax, float *packed, float *rowLoss, void *keptLogits, int64_t *keptTargets, float *loss,
                        uint64_t rows, uint64_t vocab, cudaStream_t stream)
{
    if (!logits || !targets || !rowMax || !packed || !rowLoss || !loss) return HCCL_E_PTR;
    if (rows == 0 || rows > 0x7fffffff || vocab == 0 || vocab > 0x7fffffff) return HCCL_E_PARA;
    auto kern = vocab % 8 == 0 && Aligned16(logits) && Aligned16(keptLogits) ? XentLossKernel<true> : XentLossKernel<false>;
    CHK_RET(Launch("cross entropy", kern, (uint32_t)rows, kThreads, stream, (const __nv_bfloat16 *)logits, targets, vocabStart, rowMax, packed, rowLoss,
                   (__nv_bfloat16 *)keptLogits, keptTargets, (uint32_t)rows, (uint32_t)vocab));
    return Launch("cross entropy mean", MeanKernel, 1, 1024, stream, rowLoss, loss, (uint32_t)rows);
}

uint64_t HcclEmbeddingGradTokens(void) { return kEmbedTokens; }

HcclResult HcclEmbeddingGrad(const int64_t *ids, const void *dy, void *grad, uint64_t tokens, uint64_t hidden, uint64_t vocab, cudaStream_t stream)
{
    if (!ids || !dy || !grad) return HCCL_E_PTR;
    if (tokens == 0 || tokens > kEmbedTokens || hidden == 0 || hidden % 8 || hidden > (1u << 24) || vocab == 0 || vocab > 0x7fffffff || !Aligned16(dy) || !Aligned16(grad)) return HCCL_E_PARA;
    if (cudaMemsetAsync(grad, 0, vocab * hidden * 2, stream) != cudaSuccess) return HCCL_E_RUNTIME;
    return Launch("embedding gradient", EmbeddingGradKernel, dim3((uint32_t)tokens, (uint32_t)((hidden / 8 + kThreads - 1) / kThreads)), kThreads, stream,
                  ids, (const __nv_bfloat16 *)dy, (__nv_bfloat16 *)grad, (uint32_t)tokens, (uint32_t)hidden, (int64_t)vocab);
}

}  // extern "C"
