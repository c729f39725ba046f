// Host side of the wide pair tiles: parameters and launch.
#pragma once
#include <algorithm>
#include <atomic>
#include "../common/launch_count.h"
#include "../common/log.h"
#include "gemm_host.h"
#include "gemm_sm100_wide.cuh"

namespace hccl {
namespace mc2 {

// C[M,N] = A * B with tiles of 256 x BN, BN a multiple of 32 from 288 to 512 (B stored [K, N]: of 128, since a CTA's part of a half is
// whole 64-column boxes).
template <bool BMN> HcclResult LaunchWide(uint32_t BN, const void *a, const void *b, void *c, uint32_t M, uint32_t N, uint32_t K, bool outFp32, uint32_t groupM, cudaStream_t s)
{
    constexpr uint32_t unit = BMN ? 128 : 32;
    if (BN % unit || BN < 288 || BN > 512) return HCCL_E_PARA;
    WideParams p{};
    p.M = M; p.N = N; p.K = K;
    p.cols[0] = (BN / 2 + unit - 1) / unit * unit;
    p.cols[1] = BN - p.cols[0];
    p.groupM = groupM; p.outFp32 = outFp32; p.errorWord = GemmErrorWord();
    CHK_RET(EncodeTmap2D(&p.tmapA, a, M, K, (uint64_t)K * 2, kBM, kBK, 2));
    if (BMN) CHK_RET(EncodeTmap2D(&p.tmapB[0], b, K, N, (uint64_t)N * 2, kBK, 64, 2));
    else for (int h = 0; h < 2; ++h) CHK_RET(EncodeTmap2D(&p.tmapB[h], b, N, K, (uint64_t)K * 2, p.cols[h] / 2, kBK, 2));
    CHK_RET(EncodeTmapC(&p.tmapC, c, M, N, outFp32));
    const uint32_t stageBytes = kBM * kBK * 2 + BN / 2 * kBK * 2;
    p.stages = std::min<uint32_t>(kWideMaxStages, (kWideSmemMax - kWideStaging - kWideBarBytes) / stageBytes);
    p.lead = 3;                  // of 4 to 5 stages; 1 / 2 / 3: 8192 x 28672 x 8192 2837 / 2814 / 2795 us, 2048 x 4096 x 14336 182.3 / 181.9 / 180.7
    const size_t smem = (size_t)p.stages * stageBytes + kWideStaging + kWideBarBytes + 1024;
    static std::atomic<bool> attrSet{false};
    auto kern = GemmKernelWide<BMN>;
    if (!attrSet) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWideSmemMax + 1024) != cudaSuccess) return HCCL_E_RUNTIME;
        attrSet = true;
    }
    const uint32_t tiles = ((M + 2 * kBM - 1) / (2 * kBM)) * ((N + BN - 1) / BN);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(std::min<uint32_t>(tiles, (uint32_t)SmCount() / 2) * 2);
    cfg.blockDim = dim3(kWideThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
    CountLaunch();
    if (e != cudaSuccess) { HCCL_ERROR("wide GEMM launch failed: %s", cudaGetErrorString(e)); (void)cudaGetLastError(); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

}  // namespace mc2
}  // namespace hccl
