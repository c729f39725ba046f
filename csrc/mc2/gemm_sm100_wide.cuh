// Wide tiles on CTA pairs: one pair computes 256 x BN of the result with BN = 288 ... 512, as two halves of up to 256 columns that share every
// tile of A. Plain products, B K-major or stored [K, N].
//
// Why wide: large products run under the board's power limit, where a result costs what its operands cost on their way from L2 into
// shared memory, and products whose rows straddle 128-byte lines are held up by those loads. A 256 x 256 tile moves 1 / 128 operand elements per
// multiply-add, a 256 x 512 one 3 / 512, a quarter less. And a width that can be chosen in steps of 32 columns fits a product into whole waves of
// tiles (1000 x 6144: 72 tiles of 352 columns on 74 pairs, where 192-wide ones take two waves).
//
// Each half of the accumulator takes up to 256 of the 512 columns of tensor memory, so there is no second accumulator to fill
// while one is stored. What overlaps instead is one half with the other: half 0 runs up to `lead` k-blocks ahead of half 1 at both
// ends of a tile. It is complete while half 1 still computes, and its columns are stored and free again when half 1 is
// complete; the next tile starts on half 0 while half 1 is stored. Two groups of 128 epilogue threads share each half, so that
// storing one takes about as long as the lead lasts.
//
// Signalling as in gemm_sm100_2cta.cuh: full[] in the leader, empty[] and tmemFull[] per CTA, tmemEmpty[] in the leader with one arrival
// per epilogue warp of both CTAs. A stage is handed back when half 1 has read it. No TMA multicast.
#pragma once
#include "gemm_sm100_2cta.cuh"

namespace hccl {
namespace mc2 {

constexpr int kWideThreads = 384;                       // producer, MMA issuer, tensor-memory owner, one spare warp, eight epilogue warps
constexpr uint32_t kWideMaxStages = 8;
constexpr uint32_t kWideStaging = 2 * kStageTileBytes;  // one store tile per epilogue group
constexpr uint32_t kWideSmemMax = 232448 - 1024;        // 227 KB less the alignment of the swizzle atoms
constexpr uint32_t kWideBarBytes = 256;

struct WideParams {
    CUtensorMap tmapA;           // box 64 elements of K x 128 rows
    CUtensorMap tmapB[2];        // K-major: box 64 elements of K x half of that half's columns; MN-major (the first only): 64 columns x 64 rows of K
    CUtensorMap tmapC;           // box 128 rows x 128 bytes
    uint32_t M, N, K;
    uint32_t cols[2];            // columns of the two halves, multiples of 32 up to 256 (MN-major: of 128)
    uint32_t stages, lead, groupM, outFp32;
    uint32_t *errorWord;
};

// One group of 128 epilogue threads stores its share (every other 128-byte slice) of a finished half at tensor-memory address `tmem` to
// columns col0 ... of C. released() is called once by every thread when the group has read its share.
template <class Released>
__device__ __forceinline__ void StoreHalfTma(const CUtensorMap *tmapC, bool fp32, uint32_t N, uint32_t tmem, uint8_t *tile, uint32_t et, uint32_t group, uint32_t row0,
                                             uint32_t col0, uint32_t cols, Released released)
{
    const uint32_t swz = et & 7, width = fp32 ? 32 : 64;
    const uint32_t wanted = col0 >= N ? 0 : N - col0 < cols ? N - col0 : cols, slices = (wanted + width - 1) / width;
    uint4 *mine = (uint4 *)(tile + et * 128);
    if (group >= slices) { released(); return; }
#pragma unroll 1
    for (uint32_t c = group; c < slices; c += 2) {
        const uint32_t off = c * width < cols - width ? c * width : cols - width;        // cols = 32 mod 64: the last slice stores 32 columns a second time
        uint32_t v[64];
        TmemLd32x32(tmem + off, *(uint32_t(*)[32])&v[0]);
        if (!fp32) TmemLd32x32(tmem + off + 32, *(uint32_t(*)[32])&v[32]);
        TmemLdWait();
        if (c + 2 >= slices) released();
        if (et == 0) TmaStoreWaitRead<0>();
        asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");       // the staging tile is free
        if (fp32) {
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) mine[q ^ swz] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        } else {
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) mine[q ^ swz] = PackBf16x8(&v[8 * q]);
        }
        FenceProxyAsyncShared();
        asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");       // the staging tile is complete
        if (et == 0) {
            TmaStore2D(tmapC, tile, (int32_t)(col0 + off), (int32_t)row0);
            TmaStoreCommit();
        }
    }
}

// BMN: B is [K, N] row-major, read MN-major (see GemmKernel).
template <bool BMN>
__global__ void __launch_bounds__(kWideThreads, 1) GemmKernelWide(const __grid_constant__ WideParams p)
{
    constexpr uint32_t kABytes = kBM * kBK * 2;
    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
    const uint32_t stages = p.stages, cols0 = p.cols[0], cols1 = p.cols[1], BN = cols0 + cols1;
    const uint32_t b0Bytes = cols0 / 2 * 128, b1Bytes = cols1 / 2 * 128, stageBytes = kABytes + b0Bytes + b1Bytes;   // B: this CTA's half of either half
    uint8_t *staging = smem + stages * stageBytes;
    uint64_t *full = (uint64_t *)(staging + kWideStaging);
    uint64_t *empty = full + kWideMaxStages, *tmemFull = empty + kWideMaxStages, *tmemEmpty = tmemFull + 2;
    uint32_t *tmemPtr = (uint32_t *)(tmemEmpty + 2);
    volatile uint32_t *abortWord = (volatile uint32_t *)(tmemPtr + 1);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cg2::CtaRankInCluster();
    const uint32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const uint32_t mBlocks = (p.M + kBM - 1) / kBM, mPairs = (mBlocks + 1) / 2, nBlocks = (p.N + BN - 1) / BN;
    const uint32_t numTiles = mPairs * nBlocks, kIters = (p.K + kBK - 1) / kBK;
    auto tileAt = [&](uint32_t t, uint32_t *mb, uint32_t *col) {             // groups of groupM row-block pairs, column blocks within
        const uint32_t perGroup = p.groupM * nBlocks, first = t / perGroup * p.groupM, in = t % perGroup;
        const uint32_t size = mPairs - first < p.groupM ? mPairs - first : p.groupM;
        *mb = (first + in % size) * 2 + rank;
        *col = in / size * BN;
    };

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < stages; ++s) { MbarInit(&full[s], 1); MbarInit(&empty[s], 1); }
        for (int h = 0; h < 2; ++h) { MbarInit(&tmemFull[h], 1); MbarInit(&tmemEmpty[h], 16); }
        *abortWord = 0;
        MbarInitFence();
    }
    if (warp == 2) { cg2::TmemAlloc2(tmemPtr, 512); cg2::TmemRelinquish2(); }
    TcFenceBefore();
    cg2::ClusterSync();                     // both CTAs' barriers are initialised before anything remote touches them
    TcFenceAfter();
    const uint32_t tmemBase = *tmemPtr, tmemHalf1 = tmemBase + 256;
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
                const int32_t colB0 = (int32_t)(col + rank * (cols0 / 2)), colB1 = (int32_t)(col + cols0 + rank * (cols1 / 2));
                for (uint32_t kb = 0; kb < kIters; ++kb) {
                    ok = MbarWait(&empty[stage], phase ^ 1, abortWord);
                    if (!ok) break;
                    const uint32_t bar = cg2::MapToCta(SmemAddr(&full[stage]), 0);
                    if (rank == 0) MbarExpectTx(&full[stage], 2 * stageBytes);
                    uint8_t *sA = smem + stage * stageBytes, *sB0 = sA + kABytes, *sB1 = sB0 + b0Bytes;
                    const int32_t k0 = (int32_t)(kb * kBK);
                    cg2::TmaLoad2DPair(sA, &p.tmapA, bar, k0, rowA);
                    if (BMN) {
                        for (uint32_t j = 0; j * kMnBoxBytes < b0Bytes; ++j) cg2::TmaLoad2DPair(sB0 + j * kMnBoxBytes, &p.tmapB[0], bar, colB0 + (int32_t)j * 64, k0);
                        for (uint32_t j = 0; j * kMnBoxBytes < b1Bytes; ++j) cg2::TmaLoad2DPair(sB1 + j * kMnBoxBytes, &p.tmapB[0], bar, colB1 + (int32_t)j * 64, k0);
                    } else {
                        cg2::TmaLoad2DPair(sB0, &p.tmapB[0], bar, k0, colB0);
                        cg2::TmaLoad2DPair(sB1, &p.tmapB[1], bar, k0, colB1);
                    }
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && ElectOne()) {
            const uint32_t idesc[2] = {MakeInstrDesc(FMT_BF16, FMT_BF16, 2 * kBM, cols0) | (BMN ? kInstrBMajorMN : 0u),
                                       MakeInstrDesc(FMT_BF16, FMT_BF16, 2 * kBM, cols1) | (BMN ? kInstrBMajorMN : 0u)};
            uint32_t stage[2] = {0, 0}, phase = 0, accPhase = 0;
            bool ok = true;
            // the k-block kb of half h; half 0 meets a stage first, half 1 hands it back
            auto block = [&](int h, uint32_t kb) {
                const uint32_t st = stage[h];
                if (h == 0) {
                    ok = MbarWait(&full[st], phase, abortWord);
                    if (!ok) return;
                    TcFenceAfter();
                }
                const uint32_t sA = SmemAddr(smem + st * stageBytes), sB = sA + kABytes + (h ? b0Bytes : 0);
                const uint64_t aDesc = MakeSmemDescSw128(sA);
                const uint64_t bDesc = BMN ? MakeSmemDescMnSw128(sB) : MakeSmemDescSw128(sB);
                const uint32_t d = h ? tmemHalf1 : tmemBase;
#pragma unroll
                for (uint32_t k = 0; k < kBK / 16; ++k)
                    cg2::UmmaF16Pair(d, AdvanceDescK(aDesc, k * 32), AdvanceDescK(bDesc, k * (BMN ? 2048 : 32)), idesc[h], (kb | k) != 0 ? 1u : 0u);
                if (h) cg2::UmmaCommitPair(&empty[st]);
                if (kb + 1 == kIters) cg2::UmmaCommitPair(&tmemFull[h]);
                if (++stage[h] == stages) { stage[h] = 0; if (h == 0) phase ^= 1; }
            };
            const uint32_t head = p.lead < kIters ? p.lead : kIters, tail = p.lead < kIters - head ? p.lead : kIters - head;
            for (uint32_t t = pair; t < numTiles && ok; t += pairs) {
                ok = MbarWait(&tmemEmpty[0], accPhase ^ 1, abortWord);
                TcFenceAfter();
                for (uint32_t kb = 0; kb < head && ok; ++kb) block(0, kb);
                if (ok) ok = MbarWait(&tmemEmpty[1], accPhase ^ 1, abortWord);
                TcFenceAfter();
                for (uint32_t kb = 0; kb < head && ok; ++kb) block(1, kb);
                for (uint32_t kb = head; kb < kIters - tail && ok; ++kb) {
                    block(0, kb);
                    if (ok) block(1, kb);
                }
                for (uint32_t kb = kIters - tail; kb < kIters && ok; ++kb) block(0, kb);
                for (uint32_t kb = kIters - tail; kb < kIters && ok; ++kb) block(1, kb);
                accPhase ^= 1;
            }
        }
    } else if (warp >= 4) {
        const uint32_t group = (warp - 4) >> 2, et = (threadIdx.x - 128) & 127, laneBase = ((warp & 3) * 32) << 16;
        const uint32_t freeHalf[2] = {cg2::MapToCta(SmemAddr(&tmemEmpty[0]), 0), cg2::MapToCta(SmemAddr(&tmemEmpty[1]), 0)};
        uint8_t *tile = staging + group * kStageTileBytes;
        uint32_t accPhase = 0;
        bool ok = true;
        for (uint32_t t = pair; t < numTiles && ok; t += pairs) {
            uint32_t mb, col;
            tileAt(t, &mb, &col);
#pragma unroll 1
            for (uint32_t h = 0; h < 2; ++h) {
                ok = MbarWait(&tmemFull[h], accPhase, abortWord);
                if (!ok) break;
                TcFenceAfter();
                auto released = [&] {                                        // this warp has read its part: tell the leader's MMA thread
                    TcFenceBefore();
                    __syncwarp();
                    if (lane == 0) cg2::MbarArriveRemote(h ? freeHalf[1] : freeHalf[0]);
                };
                if (mb < mBlocks)
                    StoreHalfTma(&p.tmapC, p.outFp32 != 0, p.N, (h ? tmemHalf1 : tmemBase) + laneBase, tile, et, group, mb * kBM, col + (h ? cols0 : 0), h ? cols1 : cols0,
                                 released);
                else released();
            }
            accPhase ^= 1;
        }
        if (et == 0) TmaStoreWaitAll();
    }
    __syncwarp();
    // A CTA must not leave while its peer can still reach its shared memory, barriers or tensor memory.
    TcFenceBefore();
    cg2::ClusterSync();
    if (warp == 2) { TcFenceAfter(); cg2::TmemDealloc2(tmemBase, 512); }
    if (threadIdx.x == 0 && *abortWord != 0 && p.errorWord) *p.errorWord = 1;
}

}  // namespace mc2
}  // namespace hccl
