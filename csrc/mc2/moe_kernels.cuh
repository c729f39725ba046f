// MoE dispatch / combine kernels (sm_100a). One cooperative launch per direction; see include/hccl/hccl_moe.h.
#pragma once
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include "../kernels/primitives.cuh"
#include "sm100_ptx.cuh"

namespace hccl {
namespace moe {

namespace cg = cooperative_groups;
using namespace dev;

constexpr int kMoeThreads = 512;
constexpr int kMaxExperts = 320;

// Offsets (bytes) inside the per-rank symmetric workspace.
struct MoeLayout {
    uint64_t recvX, recvScales, recvSrc, yBuf, recvCounts, slotMap, total;
};

struct MoeArgs {
    const void *x;             // [T, H] bf16
    const int32_t *topkIdx;    // [T, K]
    const float *weights;      // [T, K] (combine)
    void *out;                 // [T, H] bf16 (combine)
    uint32_t T, K, H, E, cap, mxfp8;
    uint64_t wsOff;            // workspace offset in every heap
    MoeLayout L;
    uint32_t segVecs;          // combine: 16-byte vectors of an output row per warp (a multiple of 32)
    uint32_t identity;         // emulation: copy recvX -> yBuf at the end of dispatch
};

__device__ __forceinline__ KCtx MoeEnter(const DevComm *c, uint32_t chan)
{
    KCtx k;
#ifdef HCCL_DEBUG_BOUNDS
    if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) g_boundsComm = c;
#endif
    k.c = c; k.rank = c->rank; k.nranks = c->nranks; k.heap = c->heap[c->rank];
    k.ctrl = CtrlOf(k.heap); k.flags = FlagsOf(k.heap);
    k.half = 0; k.chan = chan; k.syncs = 0; k.ok = true; k.vGrid = gridDim.x; k.vBlock = blockIdx.x; k.cclShift = 0; k.seq = 0xffffffffu;   // not counted by the op counter: no trace record
    k.epoch = LdVolatile(&k.ctrl->chanEpoch[chan]);
    return k;
}
__device__ __forceinline__ void MoeLeave(KCtx &k)
{
    __syncthreads();
    if (threadIdx.x == 0) *((volatile uint32_t *)&k.ctrl->chanEpoch[k.chan]) = k.epoch + k.syncs;
}

// e8m0 scale for a block with absolute maximum `amax`: the smallest power of two s with amax / s <= 448
__device__ __forceinline__ uint8_t E8m0For(float amax)
{
    if (amax <= 0.f) return 127 - 8;
    int e;
    float m = frexpf(amax / 448.f, &e);     // amax/448 = m * 2^e, m in [0.5, 1)
    if (m == 0.5f) e -= 1;
    int biased = e + 127;
    return (uint8_t)(biased < 0 ? 0 : biased > 254 ? 254 : biased);
}
__device__ __forceinline__ uint8_t ToE4m3(float v)
{
    return (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}

// Eight bf16 values of a 1 x 32 block that four neighbouring lanes share -> e4m3 values and the block's scale. Called by whole warps.
__device__ __forceinline__ uint2 QuantizeVec(const uint4 &raw, uint8_t *scale)
{
    const __nv_bfloat162 *h = (const __nv_bfloat162 *)&raw;
    float f[8], amax = 0.f;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const float2 p = __bfloat1622float2(h[x]);
        f[2 * x] = p.x; f[2 * x + 1] = p.y;
        amax = fmaxf(amax, fmaxf(fabsf(p.x), fabsf(p.y)));
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    *scale = E8m0For(amax);
    const float inv = exp2f((float)(127 - (int)*scale));
    uint32_t b[2];
#pragma unroll
    for (int x = 0; x < 2; ++x)
        b[x] = (uint32_t)ToE4m3(f[4 * x] * inv) | (uint32_t)ToE4m3(f[4 * x + 1] * inv) << 8 | (uint32_t)ToE4m3(f[4 * x + 2] * inv) << 16 |
               (uint32_t)ToE4m3(f[4 * x + 3] * inv) << 24;
    return make_uint2(b[0], b[1]);
}

// Slot of an entry that has no row (its expert id lies outside [0, numExperts), or nothing was sent because a receive buffer is too small):
// a row of zeros behind the own expert-output rows, so that the combine needs no test (one per load: 4096 tokens, top-8 106 us
// for 90; 2048 tokens, top-16 58 us for 53).
__device__ __forceinline__ uint64_t NoSlot(uint32_t me, uint32_t cap) { return (uint64_t)me << 32 | cap; }

constexpr int kMoeWarps = kMoeThreads / 32;
constexpr uint32_t kSegVecs = 128;                    // 16-byte vectors of a token row that one warp moves at a time (2 KB)
constexpr uint32_t kSegVecsFew = 32;                  // the same where tokens are few: 512 bytes, one load per lane

// A (token, segment) range of the grid's CTA `cta`: contiguous, so a CTA meets few tokens and every row is spread over
// as many CTAs as there are when tokens are few.
__device__ __forceinline__ void MoeItems(const MoeArgs &A, uint32_t segVecs, uint32_t cta, uint32_t G, uint32_t *segs, uint64_t *lo, uint64_t *hi)
{
    *segs = (A.H / 8 + segVecs - 1) / segVecs;
    const uint64_t items = (uint64_t)A.T * *segs;
    *lo = items * cta / G;
    *hi = items * (cta + 1) / G;
}

// Dispatch. What bounds it is writing topK copies of every token row (NVLink between ranks, HBM on one); the rest is kept
// short of that:
//   1. every CTA counts ALL routed entries itself, split into those before its first token and the others (shared-memory
//      atomics; 32768 entries are 16 loads of four per thread). That replaces a per-CTA histogram in global memory, a grid-wide
//      barrier and the walk over all CTAs' counts.
//   2. with several ranks CTA 0 publishes the rank's totals and the grid waits for everyone's; with one rank (SOLO) the
//      totals are already here and the kernel is launched without any grid barrier.
//   3. base rows by one prefix sum over the experts; the ordinal of an entry among those of its expert (token order) from
//      __match_any_sync within a warp and a running count over the warps: the layout is a function of the routing alone.
//   4. a warp reads a 2 KB piece of a token row ONCE, quantises it once (block-scaled form: four lanes share a 1 x 32 block,
//      so loads and stores stay coalesced) and writes it to all topK destinations.
// One rank has a kernel of its own (moe_bulk.cuh: 256 experts, top-8, hidden 7168, 4096 tokens, bf16, one B200 109 us with this one, 100.5 with that); the form here
// serves contexts that do not grant that kernel's shared memory.
template <bool EMU, bool SOLO>
__global__ void __launch_bounds__(kMoeThreads) MoeDispatchKernel(const DevComm *comms, const __grid_constant__ MoeArgs av, const MoeArgs *emuArgs)
{
    const DevComm *c = EMU ? &comms[blockIdx.y] : comms;
    const MoeArgs &A = EMU ? emuArgs[blockIdx.y] : av;
    const int n = SOLO ? 1 : c->nranks, me = SOLO ? 0 : c->rank;
    char *ws = c->heap[me] + A.wsOff;
    const uint32_t E = A.E, EL = E / n, K = A.K, entries = A.T * K;
    const uint32_t G = gridDim.x, cta = blockIdx.x;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint64_t *slotMap = (uint64_t *)(ws + A.L.slotMap);
    const uint64_t noSlot = NoSlot((uint32_t)me, A.cap);
    int32_t *recvCounts = (int32_t *)(ws + A.L.recvCounts);
    __shared__ uint32_t sBefore[kMaxExperts];          // own entries of expert e before this CTA's first token, then the next row of e
    __shared__ uint32_t sTotal[kMaxExperts];           // own entries of expert e
    __shared__ uint32_t sScan[2][kMaxExperts];         // prefix sum over the experts of all ranks' entries
    __shared__ uint32_t sWarp[kMoeWarps][kMaxExperts]; // per warp: entries of e in the current batch, then the first row of the warp's entries
    __shared__ uint32_t sRow[kMoeThreads];             // destination row of the batch's entries

    if (SOLO) { sm100::LetDependentsStart(); sm100::DependencyWait(); }
    uint32_t segs;
    uint64_t itemLo, itemHi;
    MoeItems(A, kSegVecs, cta, G, &segs, &itemLo, &itemHi);
    const uint32_t tLo = (uint32_t)(itemLo / segs), tHi = (uint32_t)((itemHi + segs - 1) / segs);    // tokens this CTA touches

    // 1. histogram of this rank's entries
    for (uint32_t e = tid; e < E; e += kMoeThreads) { sBefore[e] = 0; sTotal[e] = 0; }
    __syncthreads();
    {
        const uint32_t split = tLo * K;
        auto add = [&](uint32_t i, uint32_t e) { if (e < E) atomicAdd(i < split ? &sBefore[e] : &sTotal[e], 1u); };
        uint32_t done = 0;
        if (((uintptr_t)A.topkIdx & 15u) == 0) {             // four entries per load, eight loads in flight
            const uint4 *v = (const uint4 *)A.topkIdx;
            const uint32_t vecs = entries / 4;
            for (uint32_t i = tid; i < vecs; i += 8 * kMoeThreads) {
                uint4 e[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) if (i + j * kMoeThreads < vecs) e[j] = v[i + j * kMoeThreads];
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (i + j * kMoeThreads < vecs) {
                        const uint32_t at = (i + j * kMoeThreads) * 4;
                        add(at, e[j].x); add(at + 1, e[j].y); add(at + 2, e[j].z); add(at + 3, e[j].w);
                    }
            }
            done = vecs * 4;
        }
        for (uint32_t i = done + tid; i < entries; i += kMoeThreads) add(i, (uint32_t)A.topkIdx[i]);
    }
    __syncthreads();
    for (uint32_t e = tid; e < E; e += kMoeThreads) sTotal[e] += sBefore[e];
    __syncthreads();

    // 2. everyone's totals
    KCtx k;
    if (!SOLO) {
        k = MoeEnter(c, 0);
        if (cta == 0) {
            for (uint32_t e = tid; e < E; e += kMoeThreads)
                for (int r = 0; r < n; ++r) FlagsOf(c->heap[r])->moeCount[me][e] = sTotal[e];
            ChannelBarrier(k, 61);
            __threadfence();
        }
        cg::this_grid().sync();
    }

    // 3. first row of every expert at its destination: rows of the rank's earlier experts + rows of earlier sources
    const uint32_t e0 = tid;
    uint32_t all = 0, earlier = 0;
    static_assert(kMaxExperts <= kMoeThreads, "one thread per expert");
    if (e0 < E) {
        if (SOLO) all = sTotal[e0];
        else
            for (int s = 0; s < n; ++s) {
                const uint32_t v = k.flags->moeCount[s][e0];
                all += v;
                if (s < me) earlier += v;
            }
        sScan[0][e0] = all;
    }
    __syncthreads();
    uint32_t cur = 0;
    for (uint32_t d = 1; d < E; d <<= 1) {
        if (e0 < E) sScan[cur ^ 1][e0] = sScan[cur][e0] + (e0 >= d ? sScan[cur][e0 - d] : 0u);
        cur ^= 1;
        __syncthreads();
    }
    const uint32_t *incl = sScan[cur];
    if (e0 < E) {
        const uint32_t first = e0 / EL * EL;
        sBefore[e0] += incl[e0] - all - (first ? incl[first - 1] : 0u) + earlier;
        if (cta == 0 && e0 >= (uint32_t)me * EL && e0 < (uint32_t)(me + 1) * EL) recvCounts[e0 - me * EL] = (int32_t)all;
    }
    __syncthreads();
    // every CTA of every rank checks every destination's load against the capacity (same numbers everywhere -> same decision)
    bool overflow = false;
    for (int d = 0; d < n; ++d) {
        const uint32_t rows = incl[(d + 1) * EL - 1] - (d ? incl[d * EL - 1] : 0u);
        if (rows <= A.cap) continue;
        overflow = true;
        if (d == me && cta == 0 && tid == 0) {     // receive buffer too small: report, move nothing
            DevStatus *st = c->status;
            st->rank = (uint32_t)me; st->observed = rows; st->expected = A.cap; st->phase = 62;
            __threadfence_system();
            *((volatile uint32_t *)&st->code) = 2u;
        }
    }

    if (cta == 0)
        for (uint32_t v = tid; v < A.H / 8; v += kMoeThreads) ((uint4 *)(ws + A.L.yBuf + (uint64_t)A.cap * A.H * 2))[v] = make_uint4(0, 0, 0, 0);
    if (overflow)
        for (uint32_t i = tLo * K + tid; i < tHi * K; i += kMoeThreads) slotMap[i] = noSlot;

    // 4. scatter, in batches of whole tokens of at most kMoeThreads entries
    const uint32_t batch = kMoeThreads / K;
    const uint32_t rowVecs = A.H / 8, rowBytes = A.H * 2;
    for (uint32_t tb = tLo; tb < tHi && !overflow; tb += batch) {
        const uint32_t te = tb + batch < tHi ? tb + batch : tHi, cnt = (te - tb) * K;
        for (uint32_t j = tid; j < kMoeWarps * (uint32_t)kMaxExperts; j += kMoeThreads) ((uint32_t *)sWarp)[j] = 0;
        __syncthreads();
        const uint32_t e = tid < cnt ? (uint32_t)A.topkIdx[tb * K + tid] : 0xffffffffu;
        const uint32_t same = __match_any_sync(0xffffffffu, e);
        const uint32_t ord = __popc(same & ((1u << lane) - 1));
        if (ord == 0 && e < E) sWarp[warp][e] = __popc(same);
        __syncthreads();
        if (e0 < E) {
            uint32_t run = sBefore[e0];
#pragma unroll
            for (int w = 0; w < kMoeWarps; ++w) { const uint32_t v = sWarp[w][e0]; sWarp[w][e0] = run; run += v; }
            sBefore[e0] = run;
        }
        __syncthreads();
        if (e < E) sRow[tid] = sWarp[warp][e] + ord;
        __syncthreads();
        const uint64_t from = (uint64_t)tb * segs > itemLo ? (uint64_t)tb * segs : itemLo, to = (uint64_t)te * segs < itemHi ? (uint64_t)te * segs : itemHi;
        for (uint64_t it = from + warp; it < to; it += kMoeWarps) {
            const uint32_t t = (uint32_t)(it / segs), seg = (uint32_t)(it % segs);
            const uint4 *src = (const uint4 *)((const char *)A.x + (uint64_t)t * rowBytes);
            const uint32_t v0 = seg * kSegVecs + lane;
            uint4 r[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) if (v0 + j * 32 < rowVecs) r[j] = src[v0 + j * 32];
            uint2 q[4];
            uint8_t se[4];
            if (A.mxfp8) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (v0 + j * 32 >= rowVecs) break;                     // rows are multiples of 32 vectors: whole warps take this
                    q[j] = QuantizeVec(r[j], &se[j]);
                }
            }
            for (uint32_t kk = 0; kk < K; ++kk) {
                const uint32_t i = t * K + kk, ex = (uint32_t)A.topkIdx[i];
                if (ex >= E) {
                    if (seg == 0 && lane == 0) slotMap[i] = noSlot;
                    continue;
                }
                const uint32_t d = ex / EL, row = sRow[(t - tb) * K + kk];
                char *dws = c->heap[d] + A.wsOff;
                // one rank: the debug flavor's heap check reads the communicator that MoeEnter registers, which this form does not call
                if (SOLO ? row >= A.cap : !HCCL_RANGE_OK(dws + A.L.recvX + (uint64_t)row * (A.mxfp8 ? A.H : rowBytes), A.mxfp8 ? A.H : rowBytes)) {
                    if (seg == 0 && lane == 0) slotMap[i] = noSlot;
                    continue;
                }
                if (!A.mxfp8) {
                    uint4 *dst = (uint4 *)(dws + A.L.recvX + (uint64_t)row * rowBytes);
#pragma unroll
                    for (int j = 0; j < 4; ++j) if (v0 + j * 32 < rowVecs) dst[v0 + j * 32] = r[j];
                } else {
                    uint2 *dst = (uint2 *)(dws + A.L.recvX + (uint64_t)row * A.H);
                    uint8_t *ds = (uint8_t *)(dws + A.L.recvScales + (uint64_t)row * (A.H / 32));
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (v0 + j * 32 < rowVecs) {
                            dst[v0 + j * 32] = q[j];
                            if ((lane & 3) == 0) ds[(v0 + j * 32) / 4] = se[j];
                        }
                }
                if (seg == 0 && lane == 0) {
                    ((int32_t *)(dws + A.L.recvSrc))[row] = (int32_t)(((uint32_t)me << 24) | t);
                    slotMap[i] = ((uint64_t)d << 32) | row;
                }
            }
        }
        __syncthreads();
    }
    if (SOLO) return;
    __threadfence_system();
    cg::this_grid().sync();
    // 5. everyone has finished writing: after this barrier the received rows are visible
    if (cta == 0) {
        ChannelBarrier(k, 63);
        MoeLeave(k);
        __threadfence();
    }
    if (A.identity && !overflow) {     // emulation helper: "experts" that return their input
        cg::this_grid().sync();
        uint32_t rows = 0;
        for (uint32_t le = 0; le < EL; ++le) rows += (uint32_t)recvCounts[le];
        if (!A.mxfp8) {
            Part p = PartOf((uint64_t)rows * A.H * 2, G, cta);
            BlockCopy(ws + A.L.yBuf + p.off, ws + A.L.recvX + p.off, p.len);
        } else {
            // block-scaled payload: the stand-in expert dequantises (e4m3 value x 2^(scale - 127)) into the bf16 output buffer
            const uint32_t blocksPerRow = A.H / 32;
            const uint64_t blocks = (uint64_t)rows * blocksPerRow;
            for (uint64_t b = (uint64_t)cta * blockDim.x + threadIdx.x; b < blocks; b += (uint64_t)G * blockDim.x) {
                const uint8_t *q = (const uint8_t *)(ws + A.L.recvX) + b * 32;
                const float scale = exp2f((float)((int)((const uint8_t *)(ws + A.L.recvScales))[b] - 127));
                __nv_bfloat16 *y = (__nv_bfloat16 *)(ws + A.L.yBuf) + b * 32;
                for (int j = 0; j < 32; ++j) {
                    __half_raw hr = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)q[j], __NV_E4M3);
                    y[j] = __float2bfloat16(__half2float(__half(hr)) * scale);
                }
            }
        }
    }
}

// Combine: out[t] = sum over k, in order, of weight * expert row (zeros for an entry without one). Bound by reading topK rows per token. KMAX (8 or 16) keeps
// the row addresses and weights of a token in registers; a warp takes 2 KB of the output row at a time, all KMAX source rows
// of a vector in flight. One rank (SOLO): few tokens, in pieces of 512 bytes;
// moe_bulk.cuh has the kernel for more.
template <bool EMU, bool SOLO, int KMAX>
__global__ void __launch_bounds__(kMoeThreads) MoeCombineKernel(const DevComm *comms, const __grid_constant__ MoeArgs av, const MoeArgs *emuArgs)
{
    const DevComm *c = EMU ? &comms[blockIdx.y] : comms;
    const MoeArgs &A = EMU ? emuArgs[blockIdx.y] : av;
    const int me = SOLO ? 0 : c->rank;
    char *ws = c->heap[me] + A.wsOff;
    const uint64_t *slotMap = (const uint64_t *)(ws + A.L.slotMap);
    if (SOLO) { sm100::LetDependentsStart(); sm100::DependencyWait(); }
    if (!SOLO) {
        // every rank's expert outputs are complete once it has entered this kernel
        if (blockIdx.x == 0) {
            KCtx k = MoeEnter(c, 0);
            ChannelBarrier(k, 71);
            MoeLeave(k);
            __threadfence();
        }
        cg::this_grid().sync();
    }
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, K = A.K, rowVecs = A.H / 8;
    uint32_t segs;
    uint64_t itemLo, itemHi;
    MoeItems(A, A.segVecs, blockIdx.x, gridDim.x, &segs, &itemLo, &itemHi);
    for (uint64_t it = itemLo + warp; it < itemHi; it += kMoeWarps) {
        const uint32_t t = (uint32_t)(it / segs), seg = (uint32_t)(it % segs);
        const uint4 *rows[KMAX];
        float w[KMAX];
#pragma unroll
        for (int j = 0; j < KMAX; ++j)
            if ((uint32_t)j < K) {
                const uint64_t s = slotMap[t * K + j];
                rows[j] = (const uint4 *)(c->heap[SOLO ? 0 : (uint32_t)(s >> 32)] + A.wsOff + A.L.yBuf + (uint64_t)(uint32_t)s * A.H * 2);
                w[j] = A.weights[t * K + j];
            }
        uint4 *dst = (uint4 *)((char *)A.out + (uint64_t)t * A.H * 2);
        const uint32_t vEnd = (seg + 1) * A.segVecs < rowVecs ? (seg + 1) * A.segVecs : rowVecs;
        for (uint32_t v = seg * A.segVecs + lane; v < vEnd; v += 32) {
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            uint4 raw[KMAX];
#pragma unroll
            for (int j = 0; j < KMAX; ++j) if ((uint32_t)j < K) raw[j] = rows[j][v];
#pragma unroll
            for (int j = 0; j < KMAX; ++j) {
                if ((uint32_t)j >= K) break;
                const __nv_bfloat162 *h = (const __nv_bfloat162 *)&raw[j];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 f = __bfloat1622float2(h[q]);
                    acc[2 * q] += w[j] * f.x;
                    acc[2 * q + 1] += w[j] * f.y;
                }
            }
            uint4 o;
            __nv_bfloat162 t0 = __floats2bfloat162_rn(acc[0], acc[1]), t1 = __floats2bfloat162_rn(acc[2], acc[3]);
            __nv_bfloat162 t2 = __floats2bfloat162_rn(acc[4], acc[5]), t3 = __floats2bfloat162_rn(acc[6], acc[7]);
            o.x = *(uint32_t *)&t0; o.y = *(uint32_t *)&t1; o.z = *(uint32_t *)&t2; o.w = *(uint32_t *)&t3;
            dst[v] = o;
        }
    }
}

}  // namespace moe
}  // namespace hccl
