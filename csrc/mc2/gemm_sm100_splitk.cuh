// Split-K tcgen05 GEMM for few rows (decode batches, short prompts):  C[M,N] = A[M,K] * B[N,K]^T, bf16 or block-scaled fp8.
//
// What bounds such a product is reading B once. The persistent kernels give every 128-row block of A a tile, so a decode
// batch leaves them with N / 64 tiles at most (32 to 128 CTAs), each walking all of K alone, and they stage 128 rows of A
// per k-block whatever M is. Here instead
//   * the ROWS OF B take the M = 128 side of the instruction and the BT rows of A (16 ... 256) its N side: a stage holds
//     16 KB of B and only BT rows of A, and small rings let two CTAs share an SM (one loads while the other drains);
//   * a cluster of S CTAs (S <= 8) shares one 128 x BT tile, each taking a contiguous part of K. Every CTA parks its fp32
//     partial in its own shared memory (the ring, free by then), and after one cluster barrier each CTA adds up 1/S of the
//     tile from all of them through distributed shared memory, in rank order: no workspace, no atomics, the same bits on
//     every run.
// One B200, us per product before / with this kernel (weights rotating through more than L2): 4 x 4096 x 4096 25.2 / 9.3 (floor 5.1), 16 x 4096 x 14336
// 42.3 / 21.8 (18.1), 64 x 128256 x 4096 196 / 171 (164); block-scaled 32 x 8192 x 14336 31.6 / 24.1 (18.8). What is left over the floor is start,
// drain and the reduction, about 4 us.
// The automatic choice takes BT = 128 and 192 for bf16 products only. 192 rows, one CTA per SM with five stages: 384 x 4096 x 14336 41.5 us, 128 x 128 tiles of one CTA 76.9, 256 rows 50.0.
// No TMA multicast. Rows of A past M and of B past N are zero-filled by the TMA loads and never stored.
#pragma once
#include "gemm_sm100_2cta.cuh"
#include "gemm_sm100_mx.cuh"
#include "mx_quantize.cuh"

namespace hccl {
namespace mc2 {

template <int BT_, bool MX_> struct GemmSplitKSmem {
    static_assert(BT_ == 16 || BT_ == 32 || BT_ == 64 || BT_ == 128 || (BT_ == 192 && !MX_) || BT_ == 256, "rows of A per tile; block-scaled ones start on half a scale atom");
    static constexpr int BT = BT_;
    static constexpr int kStageK = MX_ ? kMxBK : kBK;                        // elements of K per stage: 128 bytes per row either way
    static constexpr int kBBytes = 128 * 128;                                // 128 rows of B
    static constexpr int kABytes = BT * 128;
    static constexpr int kAtomsA = (BT + 127) / 128;                         // scale atoms of A (block-scaled form)
    static constexpr int kSfBytes = MX_ ? (1 + kAtomsA) * kSfAtomBytes : 0;
    static constexpr int kStages = BT <= 16 ? (MX_ ? 5 : 6) : BT <= 32 ? 5 : BT <= 64 ? 4 : BT <= 128 ? 3 : BT <= 192 ? 5 : 4;   // BT <= 128: two CTAs per SM
    static constexpr int kRing = kStages * (kBBytes + kABytes);
    static constexpr int kSfOff = kRing;
    static constexpr int kBarOff = kSfOff + kStages * kSfBytes;
    static constexpr int kTotal = kBarOff + 256;
    static constexpr int kPartialBytes = BT * 128 * 4;                       // [BT][128] fp32, reuses the ring
    static constexpr int kSfCols = 4 + 4 * kAtomsA;
    static constexpr int kSfColBase = BT < 32 ? 32 : BT;
    static constexpr int kNeedCols = MX_ ? kSfColBase + kStages * kSfCols : kSfColBase;
    static constexpr int kTmemCols = kNeedCols <= 32 ? 32 : kNeedCols <= 64 ? 64 : kNeedCols <= 128 ? 128 : kNeedCols <= 256 ? 256 : 512;
    static constexpr int kCtasPerSm = BT <= 128 ? 2 : 1;
    static_assert(kPartialBytes <= kRing, "the partial tile reuses the ring");
    static_assert(kCtasPerSm * kTmemCols <= 512 && kCtasPerSm * (kTotal + 2048) <= 233472, "residency");
};

struct SplitKParams {
    CUtensorMap tmapB;            // [N, K], box 128 rows; BMN: [K, N], box 64 columns x 64 rows of K
    CUtensorMap tmapA;            // [M, K], box BT rows
    void *C;
    uint32_t M, N, K;
    uint32_t split;               // CTAs per tile = cluster size
    uint32_t outFp32;
    uint32_t *errorWord;
    const uint8_t *sfB, *sfA;     // block-scaled form: scale atoms [rows / 128][K / 128][512]
    uint32_t sfAtomsA;            // 128-row atoms A's scale array holds
    const __nv_bfloat16 *a;       // QUANT: A in bf16
    uint32_t earlyB;              // the kernel before this one wrote A only: B may be read while it runs
};

namespace splitk {
__device__ __forceinline__ float4 LdDsmemF4(uint32_t clusterAddr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(clusterAddr));
    return v;
}
__device__ __forceinline__ void ClusterArrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void ClusterWait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
}  // namespace splitk

// BMN: B is [K, N] row-major, read MN-major (see GemmKernel).
// QUANT (block-scaled, up to 32 rows per tile): A is given in bf16. The four epilogue warps, which have nothing to do before the accumulator is complete, turn this CTA's part of it into
// e4m3 values and scales, straight into the ring, in place of the TMA loads.
template <int BT_, bool MX, bool QUANT = false, bool BMN = false>
__global__ void __launch_bounds__(kGemmThreads, (GemmSplitKSmem<BT_, MX>::kCtasPerSm)) GemmKernelSplitK(const __grid_constant__ SplitKParams p)
{
    using S = GemmSplitKSmem<BT_, MX>;
    constexpr int BT = S::BT, STAGES = S::kStages;
    static_assert(!QUANT || (MX && BT <= 32 && STAGES >= 4), "rows that an epilogue warp quantises, stages for four of them");
    static_assert(!BMN || !MX, "MN-major operands are bf16");
    constexpr uint32_t kIdesc = MakeInstrDesc(FMT_BF16, FMT_BF16, 128, BT) | (BMN ? kInstrAMajorMN : 0u);
    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
    uint8_t *sB = smem;
    uint8_t *sA = smem + STAGES * S::kBBytes;
    uint8_t *sSF = smem + S::kSfOff;
    uint64_t *full = (uint64_t *)(smem + S::kBarOff);
    uint64_t *empty = full + STAGES;
    uint64_t *done = empty + STAGES;
    uint32_t *tmemPtr = (uint32_t *)(done + 1);
    volatile uint32_t *abortWord = (volatile uint32_t *)(tmemPtr + 1);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t split = p.split, rank = split > 1 ? cg2::CtaRankInCluster() : 0;
    const uint32_t tile = blockIdx.x / split;
    const uint32_t nTiles = (p.N + 127) / 128;
    const uint32_t n0 = (tile % nTiles) * 128, m0 = (tile / nTiles) * BT;
    const uint32_t kTotal = (p.K + S::kStageK - 1) / S::kStageK;
    const uint32_t kLo = (uint32_t)((uint64_t)kTotal * rank / split), kHi = (uint32_t)((uint64_t)kTotal * (rank + 1) / split);

    if (threadIdx.x == 0) {
        PrefetchTmap(&p.tmapB);
        if (!QUANT) PrefetchTmap(&p.tmapA);
        for (int s = 0; s < STAGES; ++s) { MbarInit(&full[s], QUANT ? 2 : 1); MbarInit(&empty[s], 1); }
        MbarInit(done, 1);
        *abortWord = 0;
        MbarInitFence();
    }
    if (warp == 2) { TmemAlloc(tmemPtr, S::kTmemCols); TmemRelinquish(); }
    TcFenceBefore();
    __syncthreads();
    TcFenceAfter();
    const uint32_t tmemBase = *tmemPtr;
    LetDependentsStart();
    const uint8_t *sfB = MX ? p.sfB + (uint64_t)(n0 / 128) * kTotal * kSfAtomBytes : nullptr;
    auto loadB = [&](uint32_t kb, uint32_t stage) {
        MbarExpectTx(&full[stage], QUANT ? S::kBBytes + kSfAtomBytes : S::kBBytes + S::kABytes + S::kSfBytes);
        if (BMN) {
#pragma unroll
            for (int j = 0; j < 2; ++j) TmaLoad2D(sB + stage * S::kBBytes + j * kMnBoxBytes, &p.tmapB, &full[stage], (int32_t)(n0 + j * 64), (int32_t)(kb * S::kStageK));
        } else {
            TmaLoad2D(sB + stage * S::kBBytes, &p.tmapB, &full[stage], (int32_t)(kb * S::kStageK), (int32_t)n0);
        }
        if (MX) BulkLoadG2S(sSF + stage * S::kSfBytes, sfB + (uint64_t)kb * kSfAtomBytes, kSfAtomBytes, &full[stage]);
    };
    const uint32_t early = !p.earlyB ? 0 : kHi - kLo < (uint32_t)STAGES ? kHi - kLo : (uint32_t)STAGES;
    if (warp == 0 && ElectOne())
        for (uint32_t i = 0; i < early; ++i) loadB(kLo + i, i);
    __syncwarp();
    DependencyWait();                        // up to here nothing touched global memory but the kernel's own parameters and, where allowed, B

    if (warp == 0) {
        if (ElectOne()) {
            uint32_t stage = 0, phase = 0;
            const uint8_t *sfA[2] = {nullptr, nullptr};
            if (MX && !QUANT) {
#pragma unroll
                for (int j = 0; j < S::kAtomsA; ++j) {
                    uint32_t atom = m0 / 128 + j;                            // rows past M: any finite scales do (their operands are zero)
                    if (atom >= p.sfAtomsA) atom = p.sfAtomsA - 1;
                    sfA[j] = p.sfA + (uint64_t)atom * kTotal * kSfAtomBytes;
                }
            }
            for (uint32_t kb = kLo; kb < kHi; ++kb) {
                if (!MbarWaitRelaxed(&empty[stage], phase ^ 1, abortWord, 0)) break;
                if (kb - kLo >= early) loadB(kb, stage);
                if (!QUANT) TmaLoad2D(sA + stage * S::kABytes, &p.tmapA, &full[stage], (int32_t)(kb * S::kStageK), (int32_t)m0);
                if (MX && !QUANT) {
                    uint8_t *sf = sSF + stage * S::kSfBytes;
#pragma unroll
                    for (int j = 0; j < S::kAtomsA; ++j) BulkLoadG2S(sf + (1 + j) * kSfAtomBytes, sfA[j] + (uint64_t)kb * kSfAtomBytes, kSfAtomBytes, &full[stage]);
                }
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        if (ElectOne()) {
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            for (uint32_t kb = kLo; kb < kHi; ++kb) {
                ok = MbarWait(&full[stage], phase, abortWord);
                if (!ok) break;
                TcFenceAfter();
                const uint64_t bDesc = BMN ? MakeSmemDescMnSw128(SmemAddr(sB + stage * S::kBBytes)) : MakeSmemDescSw128(SmemAddr(sB + stage * S::kBBytes));
                const uint64_t aDesc = MakeSmemDescSw128(SmemAddr(sA + stage * S::kABytes));
                if (MX) {
                    const uint32_t sfCol = tmemBase + S::kSfColBase + stage * S::kSfCols, sfSmem = SmemAddr(sSF + stage * S::kSfBytes);
#pragma unroll
                    for (int j = 0; j < 1 + S::kAtomsA; ++j) TmemCpSfAtom(sfCol + 4 * j, MakeSfSmemDesc(sfSmem + j * kSfAtomBytes));
                    // BT = 64: the tile's rows sit 0 or 64 rows, that is 0 or 2 columns, into their scale atom (BT < 64: m0 = 0)
                    const uint32_t sfaCol = sfCol + 4 + (m0 % 128) / 32;
#pragma unroll
                    for (uint32_t k = 0; k < kMxBK / 32; ++k)
                        UmmaMxf8(tmemBase, AdvanceDescK(bDesc, k * 32), AdvanceDescK(aDesc, k * 32), MakeInstrDescMx(128, BT, k), sfCol, sfaCol,
                                 kb != kLo || k != 0 ? 1u : 0u);
                } else {
#pragma unroll
                    for (uint32_t k = 0; k < kBK / 16; ++k)
                        UmmaF16(tmemBase, AdvanceDescK(bDesc, k * (BMN ? 2048 : 32)), AdvanceDescK(aDesc, k * 32), kIdesc, kb != kLo || k != 0 ? 1u : 0u);
                }
                UmmaCommit(&empty[stage]);
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
            if (ok) UmmaCommit(done);
        }
    }
    if (QUANT && warp >= 4) {
        // a warp takes every fourth k-block, so that four are on their way from memory; four lanes per row of 128 values, eight rows at a time
        constexpr int ITEMS = BT / 8;
        const uint32_t block = lane & 3, row = lane >> 2;
        uint4 next[ITEMS][4];
        auto fetch = [&](uint32_t kb) {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const uint32_t r = m0 + row + i * 8;
                const uint4 *src = (const uint4 *)(p.a + (size_t)r * p.K + (size_t)kb * kMxBK + block * 32);
#pragma unroll
                for (int j = 0; j < 4; ++j) next[i][j] = r < p.M ? src[j] : make_uint4(0, 0, 0, 0);
            }
        };
        uint32_t kb = kLo + warp - 4, stage = (warp - 4) % STAGES, phase = (warp - 4) / STAGES & 1;
        if (kb < kHi) fetch(kb);
        for (; kb < kHi; kb += 4) {
            uint4 q[ITEMS][2];
            uint8_t se[ITEMS];
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                se[i] = QuantizeBlock(next[i], q[i]);
                if (m0 + row + i * 8 >= p.M) se[i] = 127;
            }
            if (kb + 4 < kHi) fetch(kb + 4);
            if (!MbarWaitRelaxed(&empty[stage], phase ^ 1, abortWord, 0)) break;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const uint32_t r = row + i * 8, inAtom = m0 % 128 + r;
                uint4 *dst = (uint4 *)(sA + stage * S::kABytes + r * 128);        // 128-byte swizzle
                dst[(block * 2) ^ (r & 7)] = q[i][0];
                dst[(block * 2 + 1) ^ (r & 7)] = q[i][1];
                sSF[stage * S::kSfBytes + kSfAtomBytes + (inAtom % 32) * 16 + inAtom / 32 * 4 + block] = se[i];
            }
            FenceProxyAsyncShared();
            __syncwarp();
            if (lane == 0) MbarArrive(&full[stage]);
            stage += 4;
            if (stage >= STAGES) { stage -= STAGES; phase ^= 1; }
        }
    }
    __syncwarp();
    // accumulator -> [BT][128] fp32 in the ring: thread = row of B, so a warp's stores are 32 consecutive words
    float *part = (float *)smem;
    const uint32_t mHere = p.M - m0 < (uint32_t)BT ? p.M - m0 : (uint32_t)BT;
    if (warp >= 4) {
        const uint32_t q = warp - 4;
        if (MbarWaitRelaxed(done, 0, abortWord, 0)) {
            TcFenceAfter();
            constexpr int CH = BT < 32 ? BT : 32;
#pragma unroll 1
            for (uint32_t c = 0; c < mHere; c += CH) {
                uint32_t v[32];
                TmemLd32x32(tmemBase + ((q * 32) << 16) + c, v);             // BT = 16: the upper half of the 32 columns is not part of the tile
                TmemLdWait();
#pragma unroll
                for (int j = 0; j < CH; ++j) part[(c + j) * 128 + q * 32 + lane] = __uint_as_float(v[j]);
            }
            TcFenceBefore();
        }
    }
    __syncwarp();
    if (split > 1) { splitk::ClusterArrive(); splitk::ClusterWait(); }
    else __syncthreads();
    if (warp == 2) { TcFenceAfter(); TmemDealloc(tmemBase, S::kTmemCols); }

    // this CTA's share of the tile: groups of four columns of C, summed over the ranks in order
    const uint32_t groups = mHere * 32;
    const uint32_t gLo = groups * rank / split, gHi = groups * (rank + 1) / split;
    const uint32_t partAddr = SmemAddr(part);
    uint32_t peer[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) peer[r] = split > 1 && (uint32_t)r < split ? cg2::MapToCta(partAddr, r) : partAddr;
    for (uint32_t g = gLo + threadIdx.x; g < gHi; g += kGemmThreads) {
        const uint32_t t = g >> 5, col = (g & 31) * 4, n = n0 + col;
        if (n >= p.N) continue;
        const uint32_t off = (t * 128 + col) * 4;
        float4 acc;
        if (split > 1) {
            float4 v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) if ((uint32_t)r < split) v[r] = splitk::LdDsmemF4(peer[r] + off);
            acc = v[0];
#pragma unroll
            for (int r = 1; r < 8; ++r)
                if ((uint32_t)r < split) { acc.x += v[r].x; acc.y += v[r].y; acc.z += v[r].z; acc.w += v[r].w; }
        } else {
            acc = *(const float4 *)((const char *)part + off);
        }
        const size_t at = (size_t)(m0 + t) * p.N + n;
        if (p.outFp32) {
            *(float4 *)((float *)p.C + at) = acc;
        } else {
            __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x, acc.y), hi = __floats2bfloat162_rn(acc.z, acc.w);
            uint2 o;
            o.x = *(uint32_t *)&lo; o.y = *(uint32_t *)&hi;
            *(uint2 *)((__nv_bfloat16 *)p.C + at) = o;
        }
    }
    if (threadIdx.x == 0 && *abortWord != 0 && p.errorWord) *p.errorWord = 1;
    __syncwarp();
    if (split > 1) { splitk::ClusterArrive(); splitk::ClusterWait(); }       // nobody leaves while a peer still reads its partial
}

}  // namespace mc2
}  // namespace hccl
