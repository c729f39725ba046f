// Gradient of causal attention over short sequences, from the packed QKV projection to the packed gradient of it: rotary embedding and its transpose, grouped queries and the
// five products in one kernel. A small decoder is bound by launches and by what the host does around them: the library's backward pass, the transposed
// rotary embedding and the views between them are six kernels and 130 us of host time per layer, this is one launch.
//
// Tiles of 64 queries and 64 keys, products by mma.sync (m16n8k16, bf16, 32-bit sums): at these sizes latency counts, not the tensor cores' rate (2 x 128 tokens of 8 heads: 48 CTAs, the tensor pipe 10 %
// of the time on their SMs). Scores,
// probabilities, their gradients' sums and all results stay in 32 bits; what an MMA reads is rounded to bf16 first, the rotated queries and keys as the rotary kernel
// rounds them. No CTA waits for another and nothing is added by atomics: the gradient of a block of queries and that of a block of keys are found by
// different CTAs of the launch, each of which computes its probabilities again from the forward pass's log-sums.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <atomic>
#include "../common/launch_count.h"
#include "../common/log.h"
#include "hccl/hccl_nn.h"
#include "swiglu.cuh"

namespace hccl {
namespace nn {

namespace {

constexpr int kTile = 64, kAttThreads = 128;
constexpr float kLog2e = 1.4426950408889634f;

struct AttArgs {
    const __nv_bfloat16 *qkv, *o, *dO;      // [tokens, (hq + 2 hk) D], [tokens, hq D], [tokens, hq D]
    __nv_bfloat16 *out;                     // the gradient of qkv
    const float *lse;                       // [batch, hq, seq]
    const float *cosT, *sinT;               // [seq, D / 2]
    uint32_t seq, hq, hk;
    float scale;                            // of the scores
};

__device__ __forceinline__ uint32_t Smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void LdMatrix(uint32_t (&r)[4], const __nv_bfloat16 *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(Smem(p)) : "memory");
}
__device__ __forceinline__ void LdMatrixT(uint32_t (&r)[4], const __nv_bfloat16 *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(Smem(p)) : "memory");
}
__device__ __forceinline__ void Mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t Pack2(float lo, float hi)
{
    const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *(const uint32_t *)&t;
}

// A tile in shared memory: 64 rows of D values, 16 bytes apart beyond that so that the eight rows of a matrix load meet different banks.
template <int D> constexpr int kPitch = D + 8;
template <int D> constexpr int kTileElems = kTile * kPitch<D>;

// Rows row0 ... of a matrix with `pitch` elements per row, from column 0 of src; zeros from row `seq` on. All loads of a thread are on their way before the first
// store: a tile costs one round trip. (t of kAttThreads threads take part.)
template <int D> struct Rows {
    static constexpr int N = kTile * (D / 8) / kAttThreads;
    uint4 v[N];
    __device__ __forceinline__ void Load(const __nv_bfloat16 *src, size_t pitch, uint32_t row0, uint32_t seq, uint32_t t)
    {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t i = t + k * kAttThreads, r = i / (D / 8), c = i % (D / 8) * 8;
            v[k] = row0 + r < seq ? *(const uint4 *)(src + (size_t)(row0 + r) * pitch + c) : make_uint4(0, 0, 0, 0);
        }
    }
    __device__ __forceinline__ void Store(__nv_bfloat16 *tile, uint32_t t) const
    {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t i = t + k * kAttThreads;
            *(uint4 *)(tile + i / (D / 8) * kPitch<D> + i % (D / 8) * 8) = v[k];
        }
    }
};
// The same, rotated on their way into the tile, in the rounding of the rotary kernel.
template <int D> struct RotatedRows {
    static constexpr int N = kTile * (D / 16) / kAttThreads;
    uint4 lo[N], hi[N];
    __device__ __forceinline__ void Load(const __nv_bfloat16 *src, size_t pitch, uint32_t row0, const AttArgs &A, uint32_t t)
    {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t i = t + k * kAttThreads, s = row0 + i / (D / 16), j = i % (D / 16) * 8;
            const uint4 *at = (const uint4 *)(src + (size_t)s * pitch + j);
            lo[k] = s < A.seq ? at[0] : make_uint4(0, 0, 0, 0);
            hi[k] = s < A.seq ? at[D / 16] : make_uint4(0, 0, 0, 0);
        }
    }
    __device__ __forceinline__ void Store(__nv_bfloat16 *tile, uint32_t row0, const AttArgs &A, uint32_t t) const
    {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t i = t + k * kAttThreads, r = i / (D / 16), j = i % (D / 16) * 8, s = min(row0 + r, A.seq - 1);
            const float4 *ct = (const float4 *)(A.cosT + (size_t)s * (D / 2) + j), *st = (const float4 *)(A.sinT + (size_t)s * (D / 2) + j);
            float a[8], b[8], o1[8], o2[8];
            Unpack8(lo[k], a);
            Unpack8(hi[k], b);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float4 c4 = ct[x], s4 = st[x];
                const float c[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const int z = 4 * x + y;
                    o1[z] = __fsub_rn(__fmul_rn(a[z], c[y]), __fmul_rn(b[z], sn[y]));
                    o2[z] = __fadd_rn(__fmul_rn(b[z], c[y]), __fmul_rn(a[z], sn[y]));
                }
            }
            *(uint4 *)(tile + r * kPitch<D> + j) = Pack8(o1);
            *(uint4 *)(tile + r * kPitch<D> + j + D / 2) = Pack8(o2);
        }
    }
};

// acc[16 rows of this warp][64] += rows of X (16 per warp, from row x0) times the rows of Y, over D.
template <int D> __device__ __forceinline__ void RowsTimesRows(float (&acc)[8][4], const __nv_bfloat16 *x, uint32_t x0, const __nv_bfloat16 *y)
{
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
        uint32_t a[4];
        LdMatrix(a, x + (x0 + (lane & 15)) * kPitch<D> + kk * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            uint32_t b[4];
            LdMatrix(b, y + (n * 16 + (lane & 7) + (lane >> 4) * 8) * kPitch<D> + kk * 16 + (lane >> 3 & 1) * 8);
            Mma(acc[2 * n], a, b[0], b[1]);
            Mma(acc[2 * n + 1], a, b[2], b[3]);
        }
    }
}
// acc[16 rows of this warp][D] += P (16 x 64, in the layout of a result) times Y[64][D], P rounded to bf16.
template <int D> __device__ __forceinline__ void ResultTimesTile(float (&acc)[D / 8][4], const float (&p)[8][4], const __nv_bfloat16 *y)
{
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        const uint32_t a[4] = {Pack2(p[2 * kk][0], p[2 * kk][1]), Pack2(p[2 * kk][2], p[2 * kk][3]), Pack2(p[2 * kk + 1][0], p[2 * kk + 1][1]),
                               Pack2(p[2 * kk + 1][2], p[2 * kk + 1][3])};
#pragma unroll
        for (int n = 0; n < D / 16; ++n) {
            uint32_t b[4];
            LdMatrixT(b, y + (kk * 16 + (lane & 15)) * kPitch<D> + n * 16 + (lane >> 4) * 8);
            Mma(acc[2 * n], a, b[0], b[1]);
            Mma(acc[2 * n + 1], a, b[2], b[3]);
        }
    }
}

// A gradient of rotated rows, times the scores' scale, turned back and stored: this thread's two rows, whose two halves it holds.
template <int D> __device__ __forceinline__ void StoreTurnedBack(const float (&g)[D / 8][4], const AttArgs &A, __nv_bfloat16 *dst, size_t pitch, uint32_t row0)
{
    const uint32_t lane = threadIdx.x & 31, c0 = (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t s = row0 + (lane >> 2) + i * 8;
        if (s >= A.seq) continue;
#pragma unroll
        for (int n = 0; n < D / 16; ++n) {
            const float2 c = *(const float2 *)(A.cosT + (size_t)s * (D / 2) + n * 8 + c0), sn = *(const float2 *)(A.sinT + (size_t)s * (D / 2) + n * 8 + c0);
            const float a0 = g[n][2 * i] * A.scale, a1 = g[n][2 * i + 1] * A.scale, b0 = g[n + D / 16][2 * i] * A.scale, b1 = g[n + D / 16][2 * i + 1] * A.scale;
            __nv_bfloat16 *at = dst + (size_t)s * pitch + n * 8 + c0;
            *(uint32_t *)at = Pack2(a0 * c.x + b0 * sn.x, a1 * c.y + b1 * sn.y);
            *(uint32_t *)(at + D / 2) = Pack2(b0 * c.x - a0 * sn.x, b1 * c.y - a1 * sn.y);
        }
    }
}

// Queries of one block and head with what their gradient brings: rotated queries and dO for shared memory, and per query the log-sum in base 2 (infinite past the end, which makes
// every probability 0) and the sum of dO * O, which the D / 8 threads that load a row find together.
template <int D> struct QueryBlock {
    static constexpr int N = Rows<D>::N, kPerRow = D / 8;
    RotatedRows<D> q;
    Rows<D> g, o;
    float lse[N];
    uint32_t row0;
    __device__ __forceinline__ void Load(const AttArgs &A, const __nv_bfloat16 *base, size_t pitch, uint32_t b, uint32_t h, uint32_t qb, uint32_t t)
    {
        row0 = qb * kTile;
        const size_t at = (size_t)b * A.seq * A.hq * D + h * D;
        q.Load(base + h * D, pitch, row0, A, t);
        g.Load(A.dO + at, (size_t)A.hq * D, row0, A.seq, t);
        o.Load(A.o + at, (size_t)A.hq * D, row0, A.seq, t);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t s = row0 + (t + k * kAttThreads) / kPerRow;
            lse[k] = s < A.seq ? A.lse[((size_t)b * A.hq + h) * A.seq + s] * kLog2e : INFINITY;
        }
    }
    __device__ __forceinline__ void Store(const AttArgs &A, __nv_bfloat16 *sQ, __nv_bfloat16 *sG, float *sLse, float *sDot, uint32_t t) const
    {
        q.Store(sQ, row0, A, t);
        g.Store(sG, t);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            float x[8], y[8], dot = 0.f;
            Unpack8(g.v[k], x);
            Unpack8(o.v[k], y);
#pragma unroll
            for (int j = 0; j < 8; ++j) dot += x[j] * y[j];
#pragma unroll
            for (int w = 1; w < kPerRow; w <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, w);
            const uint32_t r = (t + k * kAttThreads) / kPerRow;
            if (t % kPerRow == 0) {
                sDot[r] = dot;
                sLse[r] = lse[k];
            }
        }
    }
};

// A warp alone on its scheduler takes 4.4 cycles per instruction (ncu: fixed latencies, shared memory, MMA results), so several groups of four warps share the blocks that a
// CTA meets, each with tiles of its own, and add up their parts at the end in a fixed order.
template <int D> constexpr int kGroups = D == 32 ? 4 : 2;
template <int D> constexpr uint32_t kBwdBytes = (2 + 2 * kGroups<D>) * kTileElems<D> * 2;

__device__ __forceinline__ void GroupSync(uint32_t group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }

// Adds the groups' parts of a result to the first group's, through shared memory that nothing else uses any more.
template <int D, int N> __device__ __forceinline__ void AddGroups(float (&acc)[N][4], float *scratch, uint32_t group, uint32_t t)
{
    __syncthreads();
    if (group > 0)
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) scratch[(((group - 1) * N + n) * 4 + e) * kAttThreads + t] = acc[n][e];
    __syncthreads();
    if (group > 0) return;
#pragma unroll 1
    for (int g = 0; g < kGroups<D> - 1; ++g)
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] += scratch[((g * N + n) * 4 + e) * kAttThreads + t];
}

template <int D> __global__ void __launch_bounds__(kAttThreads * kGroups<D>) AttentionBwdKernel(const __grid_constant__ AttArgs A)
{
    extern __shared__ __align__(16) __nv_bfloat16 sm[];
    __shared__ float sLse[kGroups<D>][kTile], sDot[kGroups<D>][kTile];
    static_assert((kGroups<D> - 1) * (D / 8) * 4 * kAttThreads * 4 <= kBwdBytes<D>, "the groups' parts fit");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");      // started while the kernel before drains: nothing touches memory before its end
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t grp = threadIdx.x / kAttThreads, tid = threadIdx.x % kAttThreads, warp = tid >> 5, lane = tid & 31;
    __nv_bfloat16 *own0 = sm, *own1 = sm + kTileElems<D>, *met0 = sm + (2 + 2 * grp) * kTileElems<D>, *met1 = met0 + kTileElems<D>;
    const uint32_t blocks = (A.seq + kTile - 1) / kTile, b = blockIdx.y, heads = A.hq / A.hk;
    const uint32_t r0 = warp * 16 + (lane >> 2), c0 = (lane & 3) * 2;
    const size_t pitch = (size_t)(A.hq + 2 * A.hk) * D;
    const __nv_bfloat16 *base = A.qkv + (size_t)b * A.seq * pitch;
    __nv_bfloat16 *out = A.out + (size_t)b * A.seq * pitch;
    const float scale = A.scale * kLog2e;
    if (blockIdx.x < blocks * A.hk) {
        // keys and values of one block and head: rows of the tiles below are keys, columns queries
        const uint32_t kb = blockIdx.x / A.hk, kh = blockIdx.x % A.hk, met = blocks - kb;
        if (grp == 0) {
            RotatedRows<D> k;
            Rows<D> v;
            k.Load(base + (A.hq + kh) * D, pitch, kb * kTile, A, tid);
            v.Load(base + (A.hq + A.hk + kh) * D, pitch, kb * kTile, A.seq, tid);
            k.Store(own0, kb * kTile, A, tid);
            v.Store(own1, tid);
        }
        __syncthreads();
        float dk[D / 8][4] = {}, dv[D / 8][4] = {};
        for (uint32_t i = grp; i < heads * met; i += kGroups<D>) {
            const uint32_t h = kh * heads + i / met, qb = kb + i % met;
            {
                QueryBlock<D> x;
                x.Load(A, base, pitch, b, h, qb, tid);
                GroupSync(grp);
                x.Store(A, met0, met1, sLse[grp], sDot[grp], tid);
                GroupSync(grp);
            }
            float p[8][4] = {}, dp[8][4] = {};
            RowsTimesRows<D>(p, own0, warp * 16, met0);
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t q = n * 8 + c0 + (e & 1);
                    p[n][e] = qb == kb && q < r0 + (e >> 1) * 8 ? 0.f : exp2f(p[n][e] * scale - sLse[grp][q]);
                }
            ResultTimesTile<D>(dv, p, met1);
            RowsTimesRows<D>(dp, own1, warp * 16, met1);
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) p[n][e] *= dp[n][e] - sDot[grp][n * 8 + c0 + (e & 1)];
            ResultTimesTile<D>(dk, p, met0);
        }
        AddGroups<D>(dk, (float *)sm, grp, tid);
        AddGroups<D>(dv, (float *)sm, grp, tid);
        if (grp > 0) return;
        StoreTurnedBack<D>(dk, A, out + (A.hq + kh) * D, pitch, kb * kTile + warp * 16);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t s = kb * kTile + r0 + i * 8;
            if (s >= A.seq) continue;
            __nv_bfloat16 *at = out + (size_t)s * pitch + (A.hq + A.hk + kh) * D + c0;
#pragma unroll
            for (int n = 0; n < D / 8; ++n) *(uint32_t *)(at + n * 8) = Pack2(dv[n][2 * i], dv[n][2 * i + 1]);
        }
        return;
    }
    // queries of one block and head
    const uint32_t item = blockIdx.x - blocks * A.hk, qb = blocks - 1 - item / A.hq, h = item % A.hq, kh = h / heads;
    const __nv_bfloat16 *keys = base + (A.hq + kh) * D, *values = keys + A.hk * D;
    if (grp == 0) {
        QueryBlock<D> x;
        x.Load(A, base, pitch, b, h, qb, tid);
        x.Store(A, own0, own1, sLse[0], sDot[0], tid);
    }
    __syncthreads();
    float dq[D / 8][4] = {};
    for (uint32_t kb = grp; kb <= qb; kb += kGroups<D>) {
        {
            RotatedRows<D> k;
            Rows<D> v;
            k.Load(keys, pitch, kb * kTile, A, tid);
            v.Load(values, pitch, kb * kTile, A.seq, tid);
            GroupSync(grp);
            k.Store(met0, kb * kTile, A, tid);
            v.Store(met1, tid);
            GroupSync(grp);
        }
        float p[8][4] = {}, dp[8][4] = {};
        RowsTimesRows<D>(p, own0, warp * 16, met0);
        RowsTimesRows<D>(dp, own1, warp * 16, met1);
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t r = r0 + (e >> 1) * 8;
                const float v = kb == qb && n * 8 + c0 + (e & 1) > r ? 0.f : exp2f(p[n][e] * scale - sLse[0][r]);
                p[n][e] = v * (dp[n][e] - sDot[0][r]);
            }
        ResultTimesTile<D>(dq, p, met0);
    }
    AddGroups<D>(dq, (float *)sm, grp, tid);
    if (grp == 0) StoreTurnedBack<D>(dq, A, out + h * D, pitch, qb * kTile + warp * 16);
}

bool Aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

template <int D> HcclResult LaunchBwd(const AttArgs &A, uint32_t batch, cudaStream_t stream)
{
    const uint32_t blocks = (A.seq + kTile - 1) / kTile;
    static std::atomic<uint64_t> allowed{0};                         // devices whose kernel may use that much shared memory
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (dev > 63 || !(allowed.load() & bit)) {
        if (cudaFuncSetAttribute(AttentionBwdKernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwdBytes<D>) != cudaSuccess) return HCCL_E_RUNTIME;
        allowed.fetch_or(bit);
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks * (A.hq + A.hk), batch);
    cfg.blockDim = dim3(kAttThreads * kGroups<D>);
    cfg.dynamicSmemBytes = kBwdBytes<D>;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, AttentionBwdKernel<D>, A);
    CountLaunch();
    if (e != cudaSuccess) { HCCL_ERROR("attention backward launch failed: %s", cudaGetErrorString(e)); (void)cudaGetLastError(); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

}  // namespace
}  // namespace nn
}  // namespace hccl

using namespace hccl;
using namespace hccl::nn;

extern "C" {

// Where this kernel takes no longer than the library's backward pass and the transposed rotary embedding. Us on one B200, those / this, batch x seq x query heads / key
// heads x width: 2 x 128 x 8 / 4 x 32 18.6 / 7.2, 1 x 286 23.0 / 13.1, 2 x 512 22.1 / 18.6, 32 x 128 38 / 26, 64 x 64 32 / 23; beyond 3 x 512 22.8 / 24.4, 16 x 256 25.8 / 33.5, 1 x 768 24.4 / 25.3
// (one CTA walks over 24 blocks). Width 64: 1 x 128 x 16 / 4 23.1 / 18.7, 8 x 128 x 16 / 8 27.0 / 21.8; beyond 1 x 256 x 16 / 4 20.2 / 33.9. Width 128 would take 52 us where the
// library takes 24 (1 x 128 x 32 / 8): its tiles leave no registers.
int HcclAttentionBwdSuits(uint64_t batch, uint64_t seq, uint32_t qHeads, uint32_t kvHeads, uint32_t headDim)
{
    if (batch == 0 || seq == 0 || qHeads == 0 || kvHeads == 0 || qHeads % kvHeads || (headDim != 32 && headDim != 64) || batch > 65535 || seq > 4096 || qHeads > 1024) return 0;
    const uint64_t walk = qHeads / kvHeads * ((seq + kTile - 1) / kTile), scores = batch * qHeads * seq * seq;
    return headDim == 32 ? walk <= 16 && scores <= 4200000 : walk <= 8 && scores <= 2100000;
}

HcclResult HcclAttentionBwd(const void *dO, const void *qkv, const void *o, const float *lse, void *dQkv, const float *cosT, const float *sinT, uint64_t batch, uint64_t seq,
                            uint32_t qHeads, uint32_t kvHeads, uint32_t headDim, cudaStream_t stream)
{
    if (!dO || !qkv || !o || !lse || !dQkv || !cosT || !sinT) return HCCL_E_PTR;
    if (batch == 0 || batch > 65535 || seq == 0 || seq > (1u << 20) || qHeads == 0 || kvHeads == 0 || qHeads % kvHeads || qHeads > 1024) return HCCL_E_PARA;
    if (!Aligned16(dO) || !Aligned16(qkv) || !Aligned16(o) || !Aligned16(dQkv) || !Aligned16(cosT) || !Aligned16(sinT)) return HCCL_E_PARA;
    AttArgs A{};
    A.qkv = (const __nv_bfloat16 *)qkv; A.o = (const __nv_bfloat16 *)o; A.dO = (const __nv_bfloat16 *)dO; A.out = (__nv_bfloat16 *)dQkv;
    A.lse = lse; A.cosT = cosT; A.sinT = sinT;
    A.seq = (uint32_t)seq; A.hq = qHeads; A.hk = kvHeads;
    A.scale = 1.f / sqrtf((float)headDim);
    if (headDim == 32) return LaunchBwd<32>(A, (uint32_t)batch, stream);
    if (headDim == 64) return LaunchBwd<64>(A, (uint32_t)batch, stream);
    return HCCL_E_PARA;
}

}  // extern "C"
