// Host side of the split-K GEMM: parameters and launch, shared by the bf16 and the block-scaled entry.
#pragma once
#include <algorithm>
#include <atomic>
#include "../common/launch_count.h"
#include "../common/log.h"
#include "gemm_host.h"
#include "gemm_sm100_splitk.cuh"

namespace hccl {
namespace mc2 {

// bt rows of A per tile (16, 32, 64, 128, 256), split CTAs along K per tile (1 ... 8)
struct SplitKChoice { uint32_t bt = 0, split = 0; };

// Whether the split-K form is the better one for this product, and its shape.
// Measured on one B200 with weights that rotate through more than L2, us per product in a graph of many (tile kernels / split-K):
//   rows <= 64, K >= 2048: split-K wins or ties. m x n x k = 4 x 4096 x 4096: 25.2 / 10.3; 16 x 4096 x 14336: 42.3 / 22.9; 1 x 512 x 16384:
//     47.8 / 11.1; 8 x 28672 x 4096: 50.5 / 40.6; 64 x 128256 x 4096: 195.8 / 171; 64 x 28672 x 8192: 81.3 / 79.8. With K = 1024 it
//     wins with up to 16 rows (16 x 8192 x 1024: 9.8 / 7.1) and not with 64 (64 x 4096 x 1024: 7.2 / 7.4).
//   more rows: where the tile kernels leave the GPU partly empty (200 x 1024 x 8192: 26.1 / 13.4; 512 x 1024 x 4096: 15.4 / 12.2), not
//     where they have about as many CTAs as SMs (128 x 8192 x 1024: 8.1 / 10.3).
//   CTAs in all: about one per SM while K is short (32 tiles, K 4096: split 4 10.3, 8 11.0; 64 tiles, K 1024: 2 7.1, 4 7.9), two per SM for a
//     long K (64 tiles, K 8192: 2 27.6, 4 25.9) or several row tiles (100 x 4096 x 4096: 3 14.2, 4 13.5).
//   65 to 512 rows, bf16, us with 64-row tiles / chosen (split x rows): one tile of 128 rows in two CTAs per SM 88 x 10120 x 7160 74 / 39 (3 x 128),
//     122 x 10368 x 13952 91 / 56 (3 x 128), 69 x 4088 x 13504 30.7 / 24.3 (8 x 128); 256-row tiles, one CTA per SM, 241 x 5400 x 3240 32.6 / 18.0 (3 x 256),
//     336 x 3704 x 15208 143 / 76 (3 x 256, a wave and a bit, 2 x 256 91), 196 x 1744 x 5240 17.4 / 13.4 (8 x 256), 398 x 1280 x 7800 28.6 / 20.6 (6 x 256). Clusters of
//     more than four pack badly beyond 120 CTAs (408 x 1448 x 10496: 4 x 256 21.2, 6 x 256 29.1). 64-row tiles stay where six CTAs share one
//     (109 x 2088 x 15896 26.5 / 31.7 with 6 x 128) or three to five share a short K (229 x 1552 x 2464 9.1 / 10.0 with 8 x 256).
inline SplitKChoice ChooseSplitK(uint64_t m, uint64_t n, uint64_t k, bool mx)
{
    const uint64_t nt = (n + 127) / 128, tileCtas = (m + 127) / 128 * nt;       // tileCtas: CTAs that 128-wide tiles would use
    if (m <= 64 ? (k < 2048 && (m > 16 || k < 512)) : (k < 2048 || m > 512 || tileCtas >= 90)) return {};
    auto parts = [&](uint64_t s) { return (uint32_t)std::min<uint64_t>(8, std::min<uint64_t>(std::max<uint64_t>(1, s), k / 256)); };
    const uint32_t bt = m <= 16 ? 16 : m <= 32 ? 32 : 64;
    const uint64_t tiles = nt * ((m + bt - 1) / bt), ctas = k > 6144 || m > 64 ? 256 : 148;
    const SplitKChoice narrow{bt, parts(ctas / tiles)};
    if (m <= 64 || mx || narrow.split >= 6 || (k < 5000 && narrow.split >= 3)) return narrow;
    if (m <= 128) return k >= 4096 ? SplitKChoice{128, parts(256 / nt)} : SplitKChoice{};     // 72 x 7192 x 2576: 11.6, tiles 10.6
    const uint64_t t256 = nt * ((m + 255) / 256), s = 148 / t256;
    return {256, parts(s > 4 ? std::max<uint64_t>(4, 120 / t256) : std::max<uint64_t>(3, s))};
}

template <int BT, bool MX>
HcclResult LaunchSplitKT(const void *a, const void *sfa, const void *b, const void *sfb, void *c, uint32_t M, uint32_t N, uint32_t K, uint32_t split, bool outFp32,
                         bool earlyB, cudaStream_t s)
{
    using S = GemmSplitKSmem<BT, MX>;
    SplitKParams p{};
    const uint32_t elem = MX ? 1 : 2, boxK = 128 / elem;
    CHK_RET(EncodeTmap2D(&p.tmapB, b, N, K, (uint64_t)K * elem, 128, boxK, elem));
    CHK_RET(EncodeTmap2D(&p.tmapA, a, M, K, (uint64_t)K * elem, BT, boxK, elem));
    p.C = c; p.M = M; p.N = N; p.K = K; p.split = split; p.outFp32 = outFp32; p.errorWord = GemmErrorWord();
    p.sfA = (const uint8_t *)sfa; p.sfB = (const uint8_t *)sfb; p.sfAtomsA = (M + 127) / 128; p.earlyB = earlyB;
    static std::atomic<bool> attrSet{false};
    auto kern = GemmKernelSplitK<BT, MX>;
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
template <bool MX>
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
        case 16: return LaunchSplitKT<16, MX>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        case 32: return LaunchSplitKT<32, MX>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        case 64: return LaunchSplitKT<64, MX>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        case 128: return LaunchSplitKT<128, MX>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        case 256: return LaunchSplitKT<256, MX>(a, sfa, b, sfb, c, M, N, K, ch.split, outFp32, earlyB, s);
        default: return HCCL_E_PARA;
    }
}

}  // namespace mc2
}  // namespace hccl
