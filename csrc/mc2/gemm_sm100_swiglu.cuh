// The two products of a SwiGLU layer with its element-wise part in their epilogues, on CTA pairs (see gemm_sm100_2cta.cuh for the skeleton):
//   forward    gate = X Wg^T, up = X Wu^T, h = silu(gate) * up        W = [Wg; Wu] stored as [2F, K]
//   backward   dh = dY Wd, dgate and dup from dh, gate and up         Wd stored as [K, F], read MN-major
// By itself the element-wise part reads what the product has just written, or writes what the next one reads: 176 MB forward and 294 MB backward at 2048 x
// 14336. Here the forward tile holds the same columns of gate and up side by side, one CTA of the pair loading rows of Wg and the other rows of
// Wu as its half of B, and the backward tile fetches gate and up by TMA while the tensor cores work, so dh is never written. gate, up and dh are rounded
// to bf16 before they are used, as separate kernels round them: the bits are those of the product and the element-wise kernel one after the other.
// Eight epilogue warps, because the element-wise part of a tile takes some 8 us by four and a tile's product 15 at K = 4096 and 4 at 1024. One B200, us in a graph,
// separate / fused: forward 2048 x 2 x 14336 x 4096 369 / 356, 2000 x 2 x 7168 x 2048 103 / 98, 1000 x 2 x 3584 x 1024 20.0 / 19.3; backward 253 / 214, 88 / 79, 19.4 / 18.1;
// 8192 x 28672 x 8192 6560 / 5897 and 3619 / 2837.
// No TMA multicast.
#pragma once
#include "../nn/swiglu.cuh"
#include "gemm_sm100_2cta.cuh"

namespace hccl {
namespace mc2 {

struct SwiGluParams {
    CUtensorMap tmapA;                      // [M, K], box 128 rows
    CUtensorMap tmapB;                      // forward [2F, K], box BN / 2 rows; backward [K, F], box 64 rows of K x 64 columns
    CUtensorMap tmapGate, tmapUp;           // [M, F] each, rows 2F apart, box 128 rows x 64 columns: stored (forward) or loaded (backward)
    CUtensorMap tmapOut[2];                 // forward: h; backward: dgate and dup, as gate and up
    uint32_t M, F, K, groupM;
    uint32_t keep;                          // forward: gate and up are wanted too
    uint32_t *errorWord;
};

constexpr int kSwiGluThreads = 384;          // producer, MMA issuer, tensor-memory owner, one spare warp, eight epilogue warps

template <int BN_, bool BWD> struct SwiGluSmem {
    static constexpr int BN = BN_;
    static constexpr int kCols = BWD ? BN : BN / 2;          // columns of F per tile
    static constexpr int kABytes = kBM * kBK * 2;
    static constexpr int kBBytes = (BN / 2) * kBK * 2;
    static constexpr int kTiles = BWD ? 4 : 3;               // store tiles: two of gate and two of up; gate, up and h
    static constexpr int kStages = BN > 128 ? 5 : 6;
    static constexpr int kStagingOff = kStages * (kABytes + kBBytes);
    static constexpr int kBarOff = kStagingOff + kTiles * kStageTileBytes;
    static constexpr int kTotal = kBarOff + 256;
    static_assert(kStagingOff % 1024 == 0 && kTotal + 1024 <= 232448, "shared memory per CTA");
    static_assert(BN % 16 == 0 && BN <= 256 && kCols >= 64 && (!BWD || BN % 128 == 0), "tile widths");
};

template <int BN_, bool BWD> __global__ void __launch_bounds__(kSwiGluThreads, 1) GemmKernelSwiGlu(const __grid_constant__ SwiGluParams p)
{
    using S = SwiGluSmem<BN_, BWD>;
    constexpr int BN = S::BN, STAGES = S::kStages;
    constexpr uint32_t kIdesc = MakeInstrDesc(FMT_BF16, FMT_BF16, 2 * kBM, BN) | (BWD ? kInstrBMajorMN : 0u);
    constexpr uint32_t kSlices = (S::kCols + 63) / 64;
    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem, *sB = smem + STAGES * S::kABytes, *staging = smem + S::kStagingOff;
    uint64_t *full = (uint64_t *)(smem + S::kBarOff);
    uint64_t *empty = full + STAGES, *tmemFull = empty + STAGES, *tmemEmpty = tmemFull + 2, *fetched = tmemEmpty + 2;
    uint32_t *tmemPtr = (uint32_t *)(fetched + 2);
    volatile uint32_t *abortWord = (volatile uint32_t *)(tmemPtr + 1);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cg2::CtaRankInCluster();
    const uint32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const uint32_t mBlocks = (p.M + kBM - 1) / kBM, mPairs = (mBlocks + 1) / 2, nBlocks = (p.F + S::kCols - 1) / S::kCols;
    const uint32_t numTiles = mPairs * nBlocks, kIters = (p.K + kBK - 1) / kBK;
    auto tileAt = [&](uint32_t t, uint32_t *mb, uint32_t *col) {             // groups of groupM row-block pairs, column blocks within
        const uint32_t perGroup = p.groupM * nBlocks, first = t / perGroup * p.groupM, in = t % perGroup;
        const uint32_t size = mPairs - first < p.groupM ? mPairs - first : p.groupM;
        *mb = (first + in % size) * 2 + rank;
        *col = in / size * S::kCols;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { MbarInit(&full[s], 1); MbarInit(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) { MbarInit(&tmemFull[s], 1); MbarInit(&tmemEmpty[s], 512); MbarInit(&fetched[s], 1); }
        *abortWord = 0;
        MbarInitFence();
    }
    if (warp == 2) { cg2::TmemAlloc2(tmemPtr, 512); cg2::TmemRelinquish2(); }
    TcFenceBefore();
    cg2::ClusterSync();                     // both CTAs' barriers are initialised before anything remote touches them
    TcFenceAfter();
    const uint32_t tmemBase = *tmemPtr;
    LetDependentsStart();
    DependencyWait();

    if (warp == 0) {
        if (ElectOne()) {
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            for (uint32_t t = pair; t < numTiles && ok; t += pairs) {
                uint32_t mb, col;
                tileAt(t, &mb, &col);
                const int32_t rowA = (int32_t)((mb < mBlocks ? mb : mBlocks) * kBM);       // past the end: the TMA load fills zeros
                for (uint32_t kb = 0; kb < kIters; ++kb) {
                    ok = MbarWait(&empty[stage], phase ^ 1, abortWord);
                    if (!ok) break;
                    const uint32_t bar = cg2::MapToCta(SmemAddr(&full[stage]), 0);
                    if (rank == 0) MbarExpectTx(&full[stage], 2 * (S::kABytes + S::kBBytes));
                    cg2::TmaLoad2DPair(sA + stage * S::kABytes, &p.tmapA, bar, (int32_t)(kb * kBK), rowA);
                    if (BWD) {
#pragma unroll
                        for (int j = 0; j < BN / 128; ++j)
                            cg2::TmaLoad2DPair(sB + stage * S::kBBytes + j * kMnBoxBytes, &p.tmapB, bar, (int32_t)(col + rank * (BN / 2) + j * 64), (int32_t)(kb * kBK));
                    } else {
                        cg2::TmaLoad2DPair(sB + stage * S::kBBytes, &p.tmapB, bar, (int32_t)(kb * kBK), (int32_t)(rank * p.F + col));
                    }
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && ElectOne()) {
            uint32_t stage = 0, phase = 0, acc = 0, accPhase = 0;
            bool ok = true;
            for (uint32_t t = pair; t < numTiles && ok; t += pairs) {
                ok = MbarWait(&tmemEmpty[acc], accPhase ^ 1, abortWord);
                if (!ok) break;
                TcFenceAfter();
                const uint32_t dTmem = tmemBase + acc * 256;
                for (uint32_t kb = 0; kb < kIters; ++kb) {
                    ok = MbarWait(&full[stage], phase, abortWord);
                    if (!ok) break;
                    TcFenceAfter();
                    const uint64_t aDesc = MakeSmemDescSw128(SmemAddr(sA + stage * S::kABytes));
                    const uint64_t bDesc = BWD ? MakeSmemDescMnSw128(SmemAddr(sB + stage * S::kBBytes)) : MakeSmemDescSw128(SmemAddr(sB + stage * S::kBBytes));
#pragma unroll
                    for (uint32_t k = 0; k < kBK / 16; ++k)
                        cg2::UmmaF16Pair(dTmem, AdvanceDescK(aDesc, k * 32), AdvanceDescK(bDesc, k * (BWD ? 2048 : 32)), kIdesc, (kb | k) != 0 ? 1u : 0u);
                    cg2::UmmaCommitPair(&empty[stage]);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (!ok) break;
                cg2::UmmaCommitPair(&tmemFull[acc]);
                acc ^= 1;
                if (acc == 0) accPhase ^= 1;
            }
        }
    } else if (warp >= 4) {
        // two threads per row, each with 32 of a slice's 64 columns
        const uint32_t et = threadIdx.x - 128, row = et & 127, half = et >> 7, swz = row & 7, laneBase = ((warp & 3) * 32) << 16;
        const uint32_t free0 = cg2::MapToCta(SmemAddr(&tmemEmpty[0]), 0), free1 = cg2::MapToCta(SmemAddr(&tmemEmpty[1]), 0);
        // Backward: gate and up of the slices of this CTA's tiles in turn, two slices ahead. A slice: 64 columns; the last one of a tile may overlap the one before.
        uint32_t ft = pair, fs = 0, fn = 0;                                  // the next slice to fetch
        auto sliceCol = [&](uint32_t s) { return s * 64 < S::kCols - 64 ? s * 64 : (uint32_t)S::kCols - 64; };
        auto fetch = [&] {                                                   // one thread
            for (; ft < numTiles; ft += pairs, fs = 0) {
                uint32_t mb, col;
                tileAt(ft, &mb, &col);
                if (mb >= mBlocks) continue;
                uint8_t *to = staging + (fn & 1) * 2 * kStageTileBytes;
                MbarExpectTx(&fetched[fn & 1], 2 * kStageTileBytes);
                TmaLoad2D(to, &p.tmapGate, &fetched[fn & 1], (int32_t)(col + sliceCol(fs)), (int32_t)(mb * kBM));
                TmaLoad2D(to + kStageTileBytes, &p.tmapUp, &fetched[fn & 1], (int32_t)(col + sliceCol(fs)), (int32_t)(mb * kBM));
                ++fn;
                if (++fs == kSlices) { fs = 0; ft += pairs; }
                return;
            }
        };
        if (BWD && et == 0) { fetch(); fetch(); }
        uint32_t acc = 0, accPhase = 0, n = 0;
        bool ok = true;
        for (uint32_t t = pair; t < numTiles && ok; t += pairs) {
            uint32_t mb, col;
            tileAt(t, &mb, &col);
            ok = MbarWait(&tmemFull[acc], accPhase, abortWord);
            if (!ok) break;
            TcFenceAfter();
            auto released = [&] {                                            // accumulator fully read: hand it back to the leader's MMA thread
                TcFenceBefore();
                cg2::MbarArriveRemote(acc ? free1 : free0);
            };
            if (mb >= mBlocks) released();
            for (uint32_t s = 0; s < kSlices && mb < mBlocks && ok; ++s, ++n) {
                const uint32_t off = sliceCol(s), at = tmemBase + laneBase + acc * 256 + off + half * 32;
                const int32_t x = (int32_t)(col + off), y = (int32_t)(mb * kBM);
                uint8_t *tile = staging + (BWD ? (n & 1) * 2 * kStageTileBytes : 0);
                uint4 *gate = (uint4 *)(tile + row * 128), *up = (uint4 *)(tile + kStageTileBytes + row * 128);
                if (BWD) {
                    uint32_t v[32];
                    TmemLd32x32(at, v);
                    TmemLdWait();
                    if (s + 1 == kSlices) released();
                    ok = MbarWait(&fetched[n & 1], n >> 1 & 1, abortWord);
                    if (!ok) break;
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q) {
                        const uint32_t to = (half * 4 + q) ^ swz;
                        uint4 g = gate[to], u = up[to];
                        nn::SwiGluGrad8<true>(PackBf16x8(&v[8 * q]), g, u, &g, &u);
                        gate[to] = g;
                        up[to] = u;
                    }
                } else {
                    uint32_t g[32], u[32];
                    TmemLd32x32(at, g);
                    TmemLd32x32(at + BN / 2, u);
                    TmemLdWait();
                    if (s + 1 == kSlices) released();
                    if (et == 0) TmaStoreWaitRead<0>();
                    asm volatile("bar.sync 1, 256;" ::: "memory");           // the staging tiles are free
                    uint4 *h = (uint4 *)(tile + 2 * kStageTileBytes + row * 128);
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q) {
                        const uint4 gv = PackBf16x8(&g[8 * q]), uv = PackBf16x8(&u[8 * q]);
                        const uint32_t to = (half * 4 + q) ^ swz;
                        gate[to] = gv;
                        up[to] = uv;
                        h[to] = nn::SwiGlu8(gv, uv);
                    }
                }
                FenceProxyAsyncShared();
                asm volatile("bar.sync 1, 256;" ::: "memory");               // the staging tiles are complete
                if (et == 0 && (uint32_t)x < p.F) {
                    if (BWD) {
                        TmaStore2D(&p.tmapOut[0], tile, x, y);
                        TmaStore2D(&p.tmapOut[1], tile + kStageTileBytes, x, y);
                    } else {
                        if (p.keep) {
                            TmaStore2D(&p.tmapGate, tile, x, y);
                            TmaStore2D(&p.tmapUp, tile + kStageTileBytes, x, y);
                        }
                        TmaStore2D(&p.tmapOut[0], tile + 2 * kStageTileBytes, x, y);
                    }
                    TmaStoreCommit();
                }
                if (BWD && et == 0) {
                    TmaStoreWaitRead<0>();                                   // then the tiles take the slice after the next one
                    fetch();
                }
            }
            acc ^= 1;
            if (acc == 0) accPhase ^= 1;
        }
        if (et == 0) TmaStoreWaitAll();
        __syncwarp();
    }
    // A CTA must not leave while its peer can still reach its shared memory, barriers or tensor memory.
    TcFenceBefore();
    cg2::ClusterSync();
    if (warp == 2) { TcFenceAfter(); cg2::TmemDealloc2(tmemBase, 512); }
    if (threadIdx.x == 0 && *abortWord != 0 && p.errorWord) *p.errorWord = 1;
}

}  // namespace mc2
}  // namespace hccl
