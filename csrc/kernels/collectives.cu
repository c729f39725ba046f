// Launch tables and host entry points of the collective kernels.
#include "collectives.cuh"

namespace hccl {

namespace {

// ---------------------------------------------------------------------------------------------- launch tables
template <bool EMU> CollKernelFn TypedKernelFor(SmKernelId id, HcclDataType dt)
{
    switch (dt) {
        case HCCL_DATA_TYPE_INT8: return TypedKernel<int8_t>(id, EMU);
        case HCCL_DATA_TYPE_INT16: return TypedKernel<int16_t>(id, EMU);
        case HCCL_DATA_TYPE_INT32: return TypedKernel<int32_t>(id, EMU);
        case HCCL_DATA_TYPE_INT64: return TypedKernel<long long>(id, EMU);
        case HCCL_DATA_TYPE_UINT64: return TypedKernel<unsigned long long>(id, EMU);
        case HCCL_DATA_TYPE_UINT8: return TypedKernel<uint8_t>(id, EMU);
        case HCCL_DATA_TYPE_UINT16: return TypedKernel<uint16_t>(id, EMU);
        case HCCL_DATA_TYPE_UINT32: return TypedKernel<uint32_t>(id, EMU);
        case HCCL_DATA_TYPE_FP16: return TypedKernel<__half>(id, EMU);
        case HCCL_DATA_TYPE_FP32: return TypedKernel<float>(id, EMU);
        case HCCL_DATA_TYPE_FP64: return TypedKernel<double>(id, EMU);
        case HCCL_DATA_TYPE_BFP16: return TypedKernel<__nv_bfloat16>(id, EMU);
        default: return nullptr;
    }
}

template <bool EMU> CollKernelFn NvlsKernel(SmKernelId id, HcclDataType dt, HcclReduceOp op)
{
#define PICKN(KERN)                                                                                         \
    if (dt == HCCL_DATA_TYPE_FP32 && op == HCCL_REDUCE_SUM) return KERN<float, HCCL_REDUCE_SUM, EMU>;       \
    if (dt == HCCL_DATA_TYPE_BFP16 && op == HCCL_REDUCE_SUM) return KERN<__nv_bfloat16, HCCL_REDUCE_SUM, EMU>; \
    if (dt == HCCL_DATA_TYPE_BFP16 && op == HCCL_REDUCE_MAX) return KERN<__nv_bfloat16, HCCL_REDUCE_MAX, EMU>; \
    if (dt == HCCL_DATA_TYPE_BFP16 && op == HCCL_REDUCE_MIN) return KERN<__nv_bfloat16, HCCL_REDUCE_MIN, EMU>; \
    if (dt == HCCL_DATA_TYPE_FP16 && op == HCCL_REDUCE_SUM) return KERN<__half, HCCL_REDUCE_SUM, EMU>;      \
    if (dt == HCCL_DATA_TYPE_FP16 && op == HCCL_REDUCE_MAX) return KERN<__half, HCCL_REDUCE_MAX, EMU>;      \
    if (dt == HCCL_DATA_TYPE_FP16 && op == HCCL_REDUCE_MIN) return KERN<__half, HCCL_REDUCE_MIN, EMU>;      \
    return nullptr;
    switch (id) {
        case K_ALLREDUCE_NVLS_ONESHOT: PICKN(KAllReduceNvlsOneShot)
        case K_ALLREDUCE_NVLS_TWOSHOT: PICKN(KAllReduceNvlsTwoShot)
        case K_REDUCESCATTER_NVLS: PICKN(KReduceScatterNvls)
        case K_ALLREDUCE_PIPE_NVLS: PICKN(KAllReducePipeNvls)
        case K_ALLREDUCE_CONCURRENT_NVLS: PICKN(KAllReduceConcurrentNvls)
        case K_ALLREDUCE_ZC_NVLS: PICKN(KAllReduceZcNvls)
        case K_REDUCESCATTER_ZC_NVLS: PICKN(KReduceScatterZcNvls)
        case K_REDUCESCATTER_PIPE_NVLS: PICKN(KReduceScatterPipeNvls)
        default: return nullptr;
    }
#undef PICKN
}

template <bool EMU> CollKernelFn KernelFor(const SmLaunch &l)
{
    switch (l.kernel) {
        case K_ALLREDUCE_ONESHOT: case K_ALLREDUCE_TWOSHOT: case K_REDUCESCATTER_V: case K_REDUCE: case K_ALLREDUCE_PIPE: case K_REDUCESCATTER_PIPE: case K_ALLREDUCE_RING: case K_ALLREDUCE_CONCURRENT: case K_ALLREDUCE_ZC: case K_REDUCESCATTER_ZC:
            return TypedKernelFor<EMU>(l.kernel, l.dtype);
        case K_ALLREDUCE_NVLS_ONESHOT: case K_ALLREDUCE_NVLS_TWOSHOT: case K_REDUCESCATTER_NVLS: case K_ALLREDUCE_PIPE_NVLS: case K_REDUCESCATTER_PIPE_NVLS: case K_ALLREDUCE_CONCURRENT_NVLS: case K_ALLREDUCE_ZC_NVLS: case K_REDUCESCATTER_ZC_NVLS:
            return NvlsKernel<EMU>(l.kernel, l.dtype, (HcclReduceOp)l.args.op);
        case K_ALLGATHER_PIPE: return KAllGatherPipe<EMU>;
        case K_ALLGATHER_PIPE_NVLS: return KAllGatherPipeNvls<EMU>;
        case K_ALLTOALL_PIPE: return KAlltoAllPipe<EMU>;
        case K_ALLGATHER_ZC: return KAllGatherZc<EMU>;
        case K_ALLGATHER_ZC_NVLS: return KAllGatherZcNvls<EMU>;
        case K_BROADCAST_ZC: return KBroadcastZc<EMU>;
        case K_BROADCAST_ZC_NVLS: return KBroadcastZcNvls<EMU>;
        case K_ALLGATHER_V: return KAllGatherV<EMU>;
        case K_BROADCAST: return KBroadcast<EMU>;
        case K_BROADCAST_NVLS: return KBroadcastNvls<EMU>;
        case K_SCATTER: return KScatter<EMU>;
        case K_ALLTOALL_V: return KAlltoAllV<EMU>;
        case K_BARRIER: return KBarrier<EMU>;
        case K_SEND: return KSend<EMU>;
        case K_RECV: return KRecv<EMU>;
        default: return nullptr;
    }
}

}  // namespace

// ---------------------------------------------------------------------------------------------- host entry points
HcclResult SmIssueLaunch(const DevComm *devComm, const SmLaunch &l, cudaStream_t stream)
{
    if (l.kernel == K_BATCH_SEND_RECV) {
        KBatchSendRecv<false><<<l.ctas, kThreads, 0, stream>>>(devComm, l.batch, nullptr);
    } else {
        CollKernelFn fn = KernelFor<false>(l);
        if (!fn) return HCCL_E_NOT_SUPPORT;
        fn<<<l.ctas, kThreads, 0, stream>>>(devComm, l.args, nullptr);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

// Emulation: one cooperative launch covers all ranks (grid = ctas x nranks); argument blocks come from device memory.
HcclResult SmIssueEmuLaunch(const DevComm *devComms, int nranks, const SmLaunch &l0, const CollArgs *devArgs, const BatchArgs *devBatch,
                            cudaStream_t stream, bool pairKernel)
{
    dim3 grid(l0.ctas, nranks), block(kThreads);
    cudaError_t e;
    if (l0.kernel == K_BATCH_SEND_RECV) {
        BatchArgs dummyB = l0.batch;
        void *params[] = {(void *)&devComms, (void *)&dummyB, (void *)&devBatch};
        e = cudaLaunchCooperativeKernel((void *)KBatchSendRecv<true>, grid, block, params, 0, stream);
    } else {
        CollKernelFn fn = pairKernel ? (CollKernelFn)KSendRecvPair<true> : KernelFor<true>(l0);
        if (!fn) return HCCL_E_NOT_SUPPORT;
        CollArgs dummy = l0.args;
        void *params[] = {(void *)&devComms, (void *)&dummy, (void *)&devArgs};
        e = cudaLaunchCooperativeKernel((void *)fn, grid, block, params, 0, stream);
    }
    if (e != cudaSuccess) return e == cudaErrorCooperativeLaunchTooLarge ? HCCL_E_PARA : HCCL_E_RUNTIME;
    return HCCL_SUCCESS;
}

}  // namespace hccl
