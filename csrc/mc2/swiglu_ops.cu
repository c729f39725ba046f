// Host side of the SwiGLU products: argument checks, choice between the fused kernel and the product with the element-wise kernel behind it, launch.
#include <algorithm>
#include <atomic>
#include "../common/launch_count.h"
#include "../common/log.h"
#include "gemm_host.h"
#include "gemm_sm100_swiglu.cuh"
#include "hccl/hccl_mc2.h"
#include "hccl/hccl_nn.h"
#include "tile_choice.h"

namespace hccl {
namespace mc2 {

namespace {

template <int BN, bool BWD>
HcclResult LaunchSwiGlu(const void *a, const void *b, const void *gateUp, void *out, uint32_t M, uint32_t F, uint32_t K, bool keep, cudaStream_t s)
{
    using S = SwiGluSmem<BN, BWD>;
    SwiGluParams p{};
    const uint64_t rowBytes = (uint64_t)F * 2, pairBytes = rowBytes * 2;
    CHK_RET(EncodeTmap2D(&p.tmapA, a, M, K, (uint64_t)K * 2, kBM, kBK, 2));
    if (BWD) CHK_RET(EncodeTmap2D(&p.tmapB, b, K, F, rowBytes, kBK, 64, 2));
    else CHK_RET(EncodeTmap2D(&p.tmapB, b, 2 * (uint64_t)F, K, (uint64_t)K * 2, BN / 2, kBK, 2));
    CHK_RET(EncodeTmap2D(&p.tmapGate, gateUp, M, F, pairBytes, 128, 64, 2));
    CHK_RET(EncodeTmap2D(&p.tmapUp, (const char *)gateUp + rowBytes, M, F, pairBytes, 128, 64, 2));
    if (BWD) {
        CHK_RET(EncodeTmap2D(&p.tmapOut[0], out, M, F, pairBytes, 128, 64, 2));
        CHK_RET(EncodeTmap2D(&p.tmapOut[1], (char *)out + rowBytes, M, F, pairBytes, 128, 64, 2));
    } else {
        CHK_RET(EncodeTmap2D(&p.tmapOut[0], out, M, F, rowBytes, 128, 64, 2));
    }
    p.M = M; p.F = F; p.K = K; p.groupM = 8; p.keep = keep; p.errorWord = GemmErrorWord();
    static std::atomic<bool> attrSet{false};
    auto kern = GemmKernelSwiGlu<BN, BWD>;
    const size_t smem = S::kTotal + 1024;
    if (!attrSet) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return HCCL_E_RUNTIME;
        attrSet = true;
    }
    const uint32_t tiles = ((M + 2 * kBM - 1) / (2 * kBM)) * ((F + S::kCols - 1) / S::kCols);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(std::min<uint32_t>(tiles, (uint32_t)SmCount() / 2) * 2);
    cfg.blockDim = dim3(kSwiGluThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
    CountLaunch();
    if (e != cudaSuccess) { HCCL_ERROR("SwiGLU GEMM launch failed: %s", cudaGetErrorString(e)); (void)cudaGetLastError(); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

bool ShapeOk(uint64_t m, uint64_t ffn, uint64_t k) { return m > 0 && ffn > 0 && k > 0 && ffn % 8 == 0 && k % 8 == 0 && m <= 0x7fffffff && ffn <= 0x3fffffff && k <= 0x7fffffff; }

}  // namespace
}  // namespace mc2
}  // namespace hccl

using namespace hccl;
using namespace hccl::mc2;

extern "C" {

HcclResult HcclMatmulSwiGlu(const void *x, const void *w, void *gateUp, void *h, uint64_t m, uint64_t ffn, uint64_t k, int keepGateUp, cudaStream_t stream)
{
    if (!x || !w || !gateUp || !h) return HCCL_E_PTR;
    if (!ShapeOk(m, ffn, k)) { HCCL_ERROR("HcclMatmulSwiGlu: unsupported shape %llu x 2 * %llu x %llu", (unsigned long long)m, (unsigned long long)ffn, (unsigned long long)k); return HCCL_E_PARA; }
    const uint32_t M = (uint32_t)m, F = (uint32_t)ffn, K = (uint32_t)k;
    switch (ChooseSwiGlu(m, ffn, k, false, SmCount(), Gemm2CtaEnabled())) {
        case 128: return LaunchSwiGlu<128, false>(x, w, gateUp, h, M, F, K, keepGateUp != 0, stream);
        case 192: return LaunchSwiGlu<192, false>(x, w, gateUp, h, M, F, K, keepGateUp != 0, stream);
        case 224: return LaunchSwiGlu<224, false>(x, w, gateUp, h, M, F, K, keepGateUp != 0, stream);
        case 256: return LaunchSwiGlu<256, false>(x, w, gateUp, h, M, F, K, keepGateUp != 0, stream);
    }
    CHK_RET(HcclGemmBf16(x, w, gateUp, m, 2 * ffn, k, 0, stream));
    return HcclSwiGlu(gateUp, h, m, ffn, stream);
}

HcclResult HcclMatmulSwiGluBwd(const void *dy, const void *w, const void *gateUp, void *dGateUp, void *dh, uint64_t m, uint64_t ffn, uint64_t k, cudaStream_t stream)
{
    if (!dy || !w || !gateUp || !dGateUp) return HCCL_E_PTR;
    if (!ShapeOk(m, ffn, k)) { HCCL_ERROR("HcclMatmulSwiGluBwd: unsupported shape %llu x %llu x %llu", (unsigned long long)m, (unsigned long long)ffn, (unsigned long long)k); return HCCL_E_PARA; }
    const uint32_t M = (uint32_t)m, F = (uint32_t)ffn, K = (uint32_t)k;
    switch (ChooseSwiGlu(m, ffn, k, true, SmCount(), Gemm2CtaEnabled())) {
        case 128: return LaunchSwiGlu<128, true>(dy, w, gateUp, dGateUp, M, F, K, true, stream);
        case 256: return LaunchSwiGlu<256, true>(dy, w, gateUp, dGateUp, M, F, K, true, stream);
    }
    if (!dh) return HCCL_E_PTR;
    CHK_RET(HcclGemmBf16Nn(dy, w, dh, m, ffn, k, 0, stream));
    return HcclSwiGluBwd(dh, gateUp, dGateUp, m, ffn, stream);
}

int HcclMatmulSwiGluBwdNeedsDh(uint64_t m, uint64_t ffn, uint64_t k)
{
    return ChooseSwiGlu(m, ffn, k, true, SmCount(), Gemm2CtaEnabled()) == 0;
}

}  // extern "C"
