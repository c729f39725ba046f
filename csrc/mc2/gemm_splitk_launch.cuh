// Host side of the split-K GEMM: parameters and launch, shared by the bf16 and the block-scaled entry.
#pragma once
#include <algorithm>
#include <atomic>
#include "../common/launch_count.h"
#include "../common/log.h"
#include "gemm_host.h"
#include "gemm_sm100_splitk.cuh"
#include "tile_choice.h"

namespace hccl {
namespace mc2 {

template <int BT, bool MX, bool QUANT = false, bool BMN = false>
HcclResult LaunchSplitKT(const void *a, const void *sfa, const void *b, const void *sfb, void *c, uint32_t M, uint32_t N, uint32_t K, uint32_t split, bool outFp32,
                         bool earlyB, cudaStream_t s)
{
    using S = GemmSplitKSmem<BT, MX>;
    SplitKParams p{};
    const uint32_t elem = MX ? 1 : 2, boxK = 128 / elem;
    if (BMN) CHK_RET(EncodeTmap2D(&p.tmapB, b, K, N, (uint64_t)N * 2, kBK, 64, 2));
    else CHK_RET(EncodeTmap2D(&p.tmapB, b, N, K, (uint64_t)K * elem, 128, boxK, elem));
    if (QUANT) p.a = (const __nv_bfloat16 *)a;
    else CHK_RET(EncodeTmap2D(&p.tmapA, a, M, K, (uint64_t)K * elem, BT, boxK, elem));
    p.C = c; p.M = M; p.N = N; p.K = K; p.split = split; p.outFp32 = outFp32; p.errorWord = GemmErrorWord();
    p.sfA = (const uint8_t *)sfa; p.sfB = (const uint8_t *)sfb; p.sfAtomsA = (M + 127) / 128; p.earlyB = earlyB;
    static std::atomic<bool> attrSet{false};
    auto kern = GemmKernelSplitK<BT, MX, QUANT, BMN>;
    const size_t smem = S::kTotal + 1024;
    if (!attrSet) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return HCCL_E_RUNTIME;
        attrSet = true;
    }
    const uint64_t tiles = (uint64_t)((N + 127) / 128) * ((M + BT - 1) / BT);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((uint32_t)(tiles * split));
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = split; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = split > 1 ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
    CountLaunch();
    if (e != cudaSuccess) { HCCL_ERROR("split-K GEMM launch failed: %s", cudaGetErrorString(e)); (void)cudaGetLastError(); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

// earlyB: the kernel before this one in the stream wrote nothing but A, and itself waited for all before it
template <bool MX, bool BMN = false>
HcclResult LaunchSplitK(SplitKChoice ch, const void *a, const void *sfa, const void *b, const void *sfb, void *c, uint32_t M, uint32_t N, uint32_t K, bool outFp32,
                        cudaStream_t s, bool earlyB = false)
{
    if (((uintptr_t)c | (uintptr_t)sfa | (uintptr_t)sfb) & 15u) {           // four results per store, 16-byte bulk copies of the scales
        HCCL_ERROR("split-K GEMM: result %p and block scales %p, %p must be 16-byte aligned", c, sfa, sfb);
        return HCCL_E_PARA;
    }
    const uint32_t kBlocks = (K + (MX ? kMxBK : kBK) - 1) / (MX ? kMxBK : kBK);
    // every CTA needs a k-block; the tensor-memory address of block scales is a multiple of two columns (64 rows), so smaller
    // block-scaled tiles have to start on a scale atom
    if (ch.split == 0 || ch.split > 8 || ch.split > kBlocks || (MX && ch.bt < 64 && M > ch.bt)) return HCCL_E_PARA;
    switch (ch.bt) {
        case 16: return LaunchSplitKT<16, MX, false, BMN>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        case 32: return LaunchSplitKT<32, MX, false, BMN>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        case 64: return LaunchSplitKT<64, MX, false, BMN>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        case 128: return LaunchSplitKT<128, MX, false, BMN>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        case 192: if constexpr (!MX) return LaunchSplitKT<192, MX, false, BMN>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s); else return HCCL_E_PARA;
        case 256: return LaunchSplitKT<256, MX, false, BMN>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        default: return HCCL_E_PARA;
    }
}

// Block-scaled, A in bf16 and quantised by the kernel itself: up to 32 rows, one tile.
inline HcclResult LaunchSplitKQuantized(SplitKChoice ch, const void *a, const void *b, const void *sfb, void *c, uint32_t M, uint32_t N, uint32_t K, bool outFp32, cudaStream_t s)
{
    if (((uintptr_t)c | (uintptr_t)a | (uintptr_t)sfb) & 15u) {
        HCCL_ERROR("split-K GEMM: activations %p, result %p and block scales %p must be 16-byte aligned", a, c, sfb);
        return HCCL_E_PARA;
    }
    if (ch.split == 0 || ch.split > 8 || ch.split > K / kMxBK || M > ch.bt) return HCCL_E_PARA;
    switch (ch.bt) {
        case 16: return LaunchSplitKT<16, true, true>(a, nullptr, b, sfb, c, M, N, K, ch.split, outFp32, false, s);
        case 32: return LaunchSplitKT<32, true, true>(a, nullptr, b, sfb, c, M, N, K, ch.split, outFp32, false, s);
        default: return HCCL_E_PARA;
    }
}

}  // namespace mc2
}  // namespace hccl
