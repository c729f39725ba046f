// MoE dispatch and combine on one rank (sm_100a): rows move through shared memory by asynchronous copies. What bounds both is HBM: topK copies of every
// token row are written, or read. A load per thread leaves an SM with the bytes its registers can hold, and waits for all of them before the
// next; a ring keeps up to 192 KB per SM on the way whatever the threads do. Ranges of CTAs, piece sizes and the layout are those of moe_kernels.cuh,
// which has the kernels of several ranks.
// One B200, top-8 of 256 experts, hidden 7168, us in a graph, with registers / with the rings: dispatch of 4096 tokens bf16 108.7 / 100.5, block-scaled 71.4 / 62.8,
// 512 tokens 23.3 / 14.7, 64 tokens 7.7 / 5.0; combine of 4096 tokens 88.4 / 85.9, 512 14.6 / 12.9; 2048 tokens of hidden 4096, top-16: 62.4 / 54.7 and
// 52.0 / 48.5. Writing 470 MB in rows takes 80 us by itself, reading it 67.
#pragma once
#include "moe_kernels.cuh"

namespace hccl {
namespace moe {

using namespace sm100;

// Shared memory -> global; addresses and size are multiples of 16 bytes.
__device__ __forceinline__ void BulkStoreS2G(void *gdst, const void *smemSrc, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(SmemAddr(smemSrc)), "r"(bytes) : "memory");
}
template <int N> __device__ __forceinline__ void BulkStoresRead() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }

// A wait of these kernels ran out (2 s): reported as a timeout.
__device__ __forceinline__ void ReportStuck(const DevComm *c, uint32_t phase)
{
    DevStatus *st = c->status;
    st->rank = 0; st->phase = phase;
    __threadfence_system();
    *((volatile uint32_t *)&st->code) = 1u;
}

// Dispatch of any number of tokens. Every warp owns kSlots pieces of the ring and loads its first pieces before anything else; meanwhile the CTA counts all routed entries
// (one CTA per SM counts half of what two would, and eight tables keep lanes that meet a popular expert apart). Then lane j of the warp
// stores the piece to the row of choice j, straight from shared memory. The block-scaled form quantises a piece once and stores it from registers (4096
// tokens: 62.8 us; back into the ring and from there by bulk copies 67.7).
constexpr uint32_t kPieceBytes = kSegVecs * 16, kSlots = 6, kTables = 8;
constexpr uint32_t kDispatchRing = kMoeWarps * kSlots * kPieceBytes;
constexpr uint32_t kTableWords = kMaxExperts + 1;                   // the tables start in different banks
template <bool MX> __global__ void __launch_bounds__(kMoeThreads, 1) MoeDispatchBulkKernel(const DevComm *c, const __grid_constant__ MoeArgs A)
{
    extern __shared__ __align__(128) uint8_t ring[];
    __shared__ uint32_t sBefore[kMaxExperts];                       // entries of expert e before this CTA's first token, then the next row of e
    __shared__ uint32_t sWork[2 * kTables * kTableWords];           // counting: [table][before | after][expert]; batches: [warp][expert]
    __shared__ uint32_t sRow[kMoeThreads];                          // row of the batch's entries, all ones where there is none
    __shared__ uint32_t sWarpSum[kMoeWarps];
    __shared__ uint64_t full[kMoeWarps][kSlots];
    __shared__ uint32_t sAbort;
    static_assert(2 * kTables * kTableWords >= kMoeWarps * kMaxExperts, "the batches fit");
    static_assert(kMaxExperts <= kMoeThreads, "one thread per expert");
    const uint32_t E = A.E, K = A.K, entries = A.T * K, rowBytes = A.H * 2, G = gridDim.x, cta = blockIdx.x;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (lane < kSlots) MbarInit(&full[warp][lane], 1);
    if (tid == 0) sAbort = 0;
    MbarInitFence();
    for (uint32_t i = tid; i < 2 * kTables * kTableWords; i += kMoeThreads) sWork[i] = 0;
    __syncthreads();
    LetDependentsStart();
    DependencyWait();

    uint32_t segs;
    uint64_t itemLo, itemHi;
    MoeItems(A, kSegVecs, cta, G, &segs, &itemLo, &itemHi);
    const uint32_t tLo = (uint32_t)(itemLo / segs), tHi = (uint32_t)((itemHi + segs - 1) / segs);
    uint8_t *mine = ring + warp * kSlots * kPieceBytes;
    auto pieceLen = [&](uint32_t seg) { return min(kPieceBytes, rowBytes - seg * kPieceBytes); };
    auto load = [&](uint64_t it, uint32_t slot) {                    // one thread
        const uint32_t seg = (uint32_t)(it % segs), len = pieceLen(seg);
        MbarExpectTx(&full[warp][slot], len);
        BulkLoadG2S(mine + slot * kPieceBytes, (const char *)A.x + it / segs * rowBytes + (uint64_t)seg * kPieceBytes, len, &full[warp][slot]);
    };
    if (lane == 0)
        for (uint32_t s = 0; s < kSlots; ++s) if (itemLo + warp + s * kMoeWarps < itemHi) load(itemLo + warp + s * kMoeWarps, s);
    __syncwarp();

    // 1. histogram of the entries before this CTA's first token and of the others
    {
        uint32_t *table = sWork + (lane % kTables) * 2 * kTableWords;
        const uint32_t split = tLo * K;
        auto add = [&](uint32_t i, uint32_t e) { if (e < E) atomicAdd(&table[(i < split ? 0 : kTableWords) + e], 1u); };
        uint32_t done = 0;
        if (((uintptr_t)A.topkIdx & 15u) == 0) {                     // four entries per load, eight loads in flight
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
    // 2. first row of every expert: a prefix sum over the totals
    uint32_t before = 0, all = 0;
    if (tid < E) {
#pragma unroll
        for (uint32_t r = 0; r < kTables; ++r) { before += sWork[r * 2 * kTableWords + tid]; all += sWork[(r * 2 + 1) * kTableWords + tid]; }
        all += before;
    }
    uint32_t incl = all;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) { const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d); if (lane >= d) incl += v; }
    if (lane == 31) sWarpSum[warp] = incl;
    __syncthreads();
    uint32_t rows = 0;
#pragma unroll
    for (uint32_t w = 0; w < kMoeWarps; ++w) { if (w < warp) incl += sWarpSum[w]; rows += sWarpSum[w]; }
    char *ws = c->heap[0] + A.wsOff;
    uint64_t *slotMap = (uint64_t *)(ws + A.L.slotMap);
    const uint64_t noSlot = NoSlot(0, A.cap);
    if (tid < E) {
        sBefore[tid] = incl - all + before;
        if (cta == 0) ((int32_t *)(ws + A.L.recvCounts))[tid] = (int32_t)all;
    }
    const bool overflow = rows > A.cap;                              // receive buffer too small: report, move nothing
    if (cta == 0) {
        for (uint32_t v = tid; v < A.H / 8; v += kMoeThreads) ((uint4 *)(ws + A.L.yBuf + (uint64_t)A.cap * rowBytes))[v] = make_uint4(0, 0, 0, 0);
        if (overflow && tid == 0) {
            DevStatus *st = c->status;
            st->rank = 0; st->observed = rows; st->expected = A.cap; st->phase = 62;
            __threadfence_system();
            *((volatile uint32_t *)&st->code) = 2u;
        }
    }
    if (overflow)
        for (uint32_t i = tLo * K + tid; i < tHi * K; i += kMoeThreads) slotMap[i] = noSlot;

    // 3. rows of the entries in batches of whole tokens, and the pieces of those tokens
    const uint32_t batch = kMoeThreads / K;
    uint64_t it = itemLo + warp;
    uint32_t slot = 0, phase = 0;
    bool ok = true;
    for (uint32_t tb = tLo; tb < tHi && !overflow; tb += batch) {
        const uint32_t te = tb + batch < tHi ? tb + batch : tHi, cnt = (te - tb) * K;
        __syncthreads();
        for (uint32_t j = tid; j < kMoeWarps * (uint32_t)kMaxExperts; j += kMoeThreads) sWork[j] = 0;
        __syncthreads();
        const uint32_t e = tid < cnt ? (uint32_t)A.topkIdx[tb * K + tid] : 0xffffffffu;
        const uint32_t same = __match_any_sync(0xffffffffu, e);
        const uint32_t ord = __popc(same & ((1u << lane) - 1));
        if (ord == 0 && e < E) sWork[warp * kMaxExperts + e] = __popc(same);
        __syncthreads();
        if (tid < E) {
            uint32_t run = sBefore[tid];
#pragma unroll
            for (int w = 0; w < kMoeWarps; ++w) { const uint32_t v = sWork[w * kMaxExperts + tid]; sWork[w * kMaxExperts + tid] = run; run += v; }
            sBefore[tid] = run;
        }
        __syncthreads();
        sRow[tid] = e < E ? sWork[warp * kMaxExperts + e] + ord : 0xffffffffu;
        __syncthreads();
        const uint64_t to = (uint64_t)te * segs < itemHi ? (uint64_t)te * segs : itemHi;
        for (; it < to && ok; it += kMoeWarps) {
            const uint32_t t = (uint32_t)(it / segs), seg = (uint32_t)(it % segs), len = pieceLen(seg);
            uint32_t row = lane < K ? sRow[(t - tb) * K + lane] : 0xffffffffu;
            if (row >= A.cap) row = 0xffffffffu;
            if (seg == 0 && lane < K) {
                slotMap[t * K + lane] = row == 0xffffffffu ? noSlot : (uint64_t)row;
                if (row != 0xffffffffu) ((int32_t *)(ws + A.L.recvSrc))[row] = (int32_t)t;
            }
            ok = MbarWait(&full[warp][slot], phase, &sAbort);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            const uint8_t *src = mine + slot * kPieceBytes;
            if (!MX) {
                if (row != 0xffffffffu) BulkStoreS2G(ws + A.L.recvX + (uint64_t)row * rowBytes + (uint64_t)seg * kPieceBytes, src, len);
                TmaStoreCommit();
            } else {
                uint2 q[4];
                uint8_t se[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j * 512u < len) q[j] = QuantizeVec(((const uint4 *)src)[j * 32 + lane], &se[j]);       // pieces are whole rows of lanes
                const uint32_t v0 = seg * kSegVecs + lane;
                for (uint32_t kk = 0; kk < K; ++kk) {
                    const uint32_t r = __shfl_sync(0xffffffffu, row, kk);
                    if (r == 0xffffffffu) continue;
                    uint2 *dst = (uint2 *)(ws + A.L.recvX + (uint64_t)r * A.H);
                    uint8_t *ds = (uint8_t *)(ws + A.L.recvScales + (uint64_t)r * (A.H / 32));
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j * 512u < len) {
                            dst[v0 + j * 32] = q[j];
                            if ((lane & 3) == 0) ds[(v0 + j * 32) / 4] = se[j];
                        }
                }
            }
            // The slot to fill again: this one where its piece is in registers, the one before last where stores still read the last two.
            constexpr uint32_t kBehind = MX ? 0 : 2;
            if (!MX) BulkStoresRead<kBehind>();
            __syncwarp();
            const uint64_t next = it + (uint64_t)(kSlots - kBehind) * kMoeWarps;
            if (lane == 0 && it >= itemLo + warp + kBehind * kMoeWarps && next < itemHi) load(next, (slot + kSlots - kBehind) % kSlots);
            if (++slot == kSlots) { slot = 0; phase ^= 1; }
        }
    }
    if (overflow)                                                    // loads that are on the way must not outlive the CTA
        for (; it < itemHi && it < itemLo + warp + kSlots * kMoeWarps && ok; it += kMoeWarps) { ok = MbarWait(&full[warp][slot], phase, &sAbort); ++slot; }
    if (!MX) TmaStoreWaitAll();
    if (!ok && lane == 0) ReportStuck(c, 64);
}

// Combine: out[t] = sum over j, in order, of weight * expert row (a row of zeros for an entry without one). A warp takes 512 bytes of an output row at a
// time. Its lanes copy the 16 bytes of every choice that they will add up themselves, DEPTH items ahead, so no barrier is needed; rows and weights
// come from tables in shared memory (looked up in global memory per item: 4096 x 4096, top-6 48.8 us, 41.0 so). One warp that loads for six by bulk copies
// of 2 KB takes 104.6 us at 4096 tokens: what it issues, one piece after the other, is the bound.
constexpr uint32_t kCombineSmem = 208 << 10, kCombineEntries = 2048;
constexpr uint32_t CombineDepth(uint32_t K) { return K <= 3 ? 8 : K <= 6 ? 4 : K <= 8 ? 3 : 2; }
constexpr uint32_t CombineWarps(uint32_t K) { return K <= 13 ? 16 : 12; }
constexpr uint32_t CombineBytes(uint32_t K) { return CombineWarps(K) * CombineDepth(K) * K * 512; }
template <int KMAX, int DEPTH> __global__ void __launch_bounds__(kMoeThreads, 1) MoeCombineBulkKernel(const DevComm *c, const __grid_constant__ MoeArgs A)
{
    extern __shared__ __align__(128) uint8_t ring[];
    __shared__ uint32_t sRow[kCombineEntries];                       // of a batch of whole tokens
    __shared__ float sWeight[kCombineEntries];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5, K = A.K, rowBytes = A.H * 2;
    LetDependentsStart();
    DependencyWait();
    const char *ws = c->heap[0] + A.wsOff;
    const uint64_t *slotMap = (const uint64_t *)(ws + A.L.slotMap);
    const char *y = ws + A.L.yBuf + lane * 16;
    uint32_t segs;
    uint64_t itemLo, itemHi;
    MoeItems(A, 32, blockIdx.x, gridDim.x, &segs, &itemLo, &itemHi);
    const uint32_t tHi = (uint32_t)((itemHi + segs - 1) / segs), batch = kCombineEntries / K;
    const uint32_t base = SmemAddr(ring) + warp * DEPTH * K * 512 + lane * 16;
    for (uint32_t tb = (uint32_t)(itemLo / segs); tb < tHi; tb += batch) {
        const uint32_t te = min(tb + batch, tHi), cnt = (te - tb) * K;
        __syncthreads();
        for (uint32_t i = tid; i < cnt; i += blockDim.x) {
            sRow[i] = (uint32_t)slotMap[(uint64_t)tb * K + i];
            sWeight[i] = A.weights[(uint64_t)tb * K + i];
        }
        __syncthreads();
        const uint64_t lo = max(itemLo, (uint64_t)tb * segs) - (uint64_t)tb * segs + warp, hi = min(itemHi, (uint64_t)te * segs) - (uint64_t)tb * segs;
        // an item of the batch: (token, piece of its row); two walks over the warp's items, one DEPTH - 1 ahead
        uint32_t t = (uint32_t)(lo / segs), seg = (uint32_t)(lo % segs), ta = t, sa = seg, slot = 0;
        const uint32_t stepT = warps / segs, stepS = warps % segs;
        auto advance = [&](uint32_t &tok, uint32_t &sg) {
            tok += stepT;
            sg += stepS;
            if (sg >= segs) { sg -= segs; ++tok; }
        };
        const uint32_t tokens = te - tb;
        const bool last = hi < (uint64_t)tokens * segs;              // the CTA's last token is not whole
        const uint32_t hiT = (uint32_t)(hi / segs), hiS = (uint32_t)(hi % segs);
        auto within = [&](uint32_t tok, uint32_t sg) { return last ? tok < hiT || (tok == hiT && sg < hiS) : tok < tokens; };
        auto copy = [&](uint32_t into) {                             // the pieces of the item ahead, if there is one
            if (within(ta, sa)) {
                const char *at = y + sa * 512;
#pragma unroll
                for (int j = 0; j < KMAX; ++j)
                    if ((uint32_t)j < K)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(base + (into * K + j) * 512), "l"(at + (uint64_t)sRow[ta * K + j] * rowBytes) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            advance(ta, sa);
        };
#pragma unroll
        for (uint32_t i = 0; i < DEPTH - 1; ++i) copy(i);
        for (; within(t, seg); advance(t, seg)) {
            copy(slot == 0 ? DEPTH - 1 : slot - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j0 = 0; j0 < KMAX; j0 += 8) {
                uint4 raw[8];
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if ((uint32_t)(j0 + j) < K)
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(raw[j].x), "=r"(raw[j].y), "=r"(raw[j].z), "=r"(raw[j].w) : "r"(base + (slot * K + j0 + j) * 512) : "memory");
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if ((uint32_t)(j0 + j) >= K) break;
                    const float w = sWeight[t * K + j0 + j];
                    const __nv_bfloat162 *h = (const __nv_bfloat162 *)&raw[j];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float2 f = __bfloat1622float2(h[q]);
                        acc[2 * q] += w * f.x;
                        acc[2 * q + 1] += w * f.y;
                    }
                }
            }
            uint4 o;
            __nv_bfloat162 t0 = __floats2bfloat162_rn(acc[0], acc[1]), t1 = __floats2bfloat162_rn(acc[2], acc[3]);
            __nv_bfloat162 t2 = __floats2bfloat162_rn(acc[4], acc[5]), t3 = __floats2bfloat162_rn(acc[6], acc[7]);
            o.x = *(uint32_t *)&t0; o.y = *(uint32_t *)&t1; o.z = *(uint32_t *)&t2; o.w = *(uint32_t *)&t3;
            *(uint4 *)((char *)A.out + (uint64_t)(tb + t) * rowBytes + seg * 512 + lane * 16) = o;
            if (++slot == DEPTH) slot = 0;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
}
inline const void *CombineBulk(uint32_t K)
{
    return K <= 3 ? (const void *)MoeCombineBulkKernel<8, 8> : K <= 6 ? (const void *)MoeCombineBulkKernel<8, 4>
         : K <= 8 ? (const void *)MoeCombineBulkKernel<8, 3> : (const void *)MoeCombineBulkKernel<16, 2>;
}

}  // namespace moe
}  // namespace hccl
