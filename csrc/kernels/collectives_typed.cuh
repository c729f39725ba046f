// The collective kernels of one element type; a source names its types with HCCL_COLLECTIVES_OF.
#pragma once
#include "collectives.cuh"

namespace hccl {

template <typename T, bool EMU> static CollKernelFn TypedKernelOf(SmKernelId id)
{
    switch (id) {
        case K_ALLREDUCE_ONESHOT: return KAllReduceOneShot<T, EMU>;
        case K_ALLREDUCE_TWOSHOT: return KAllReduceTwoShot<T, EMU>;
        case K_REDUCESCATTER_V: return KReduceScatterV<T, EMU>;
        case K_REDUCE: return KReduce<T, EMU>;
        case K_ALLREDUCE_RING: return KAllReduceRing<T, EMU>;
        case K_ALLREDUCE_CONCURRENT: return KAllReduceConcurrentPlain<T, EMU>;
        case K_ALLREDUCE_ZC: return KAllReduceZc<T, EMU>;
        case K_REDUCESCATTER_ZC: return KReduceScatterZc<T, EMU>;
        case K_ALLREDUCE_PIPE: return KAllReducePipe<T, EMU>;
        case K_REDUCESCATTER_PIPE: return KReduceScatterPipe<T, EMU>;
        default: return nullptr;
    }
}
template <typename T> CollKernelFn TypedKernel(SmKernelId id, bool emu) { return emu ? TypedKernelOf<T, true>(id) : TypedKernelOf<T, false>(id); }

}  // namespace hccl

#define HCCL_COLLECTIVES_OF(T) template hccl::CollKernelFn hccl::TypedKernel<T>(hccl::SmKernelId, bool)
