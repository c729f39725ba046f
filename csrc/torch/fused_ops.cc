// Native face of the matmul operators for PyTorch: argument checks, result allocation, the current stream and the C call in one
// step. A decode-sized product takes under ten microseconds on the device; the same steps in Python and ctypes took
// longer than that, so the GPU waited for the host between such calls.
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/extension.h>

#include "hccl/hccl_mc2.h"

namespace {

bool IsOperand(const at::Tensor &t) { return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous(); }

cudaStream_t StreamOf(const std::optional<uint64_t> &stream)
{
    return stream ? (cudaStream_t)(uintptr_t)*stream : c10::cuda::getCurrentCUDAStream().stream();
}

// `elems` results are written at the tensor's address: it has to be that large, dense and of a type the kernels write.
void CheckResult(const std::optional<at::Tensor> &t, int64_t elems, bool fp32Too, const char *what)
{
    if (!t) return;
    if (!t->is_contiguous() || t->numel() < elems || !(t->scalar_type() == at::kBFloat16 || (fp32Too && t->scalar_type() == at::kFloat)))
        throw py::value_error(std::string(what) + " must be a contiguous tensor of at least " + std::to_string(elems) + (fp32Too ? " bf16 or fp32 elements" : " bf16 elements"));
    if (!t->is_cuda()) throw py::value_error(std::string(what) + " must be a CUDA tensor");
}

// Both return (HcclResult, out).
std::pair<int, at::Tensor> Gemm(const at::Tensor &a, const at::Tensor &w, const std::optional<at::Tensor> &out, bool fp32, bool transposedB, int variant,
                                std::optional<uint64_t> stream)
{
    const int64_t m = a.size(0), k = a.size(1), n = w.size(transposedB ? 1 : 0);
    CheckResult(out, m * n, true, "out");
    py::gil_scoped_release nogil;
    at::Tensor o = out ? *out : at::empty({m, n}, a.options().dtype(fp32 ? at::kFloat : at::kBFloat16));
    const int o32 = o.scalar_type() == at::kFloat;
    cudaStream_t s = StreamOf(stream);
    const HcclResult r = transposedB ? HcclGemmBf16Nn(a.data_ptr(), w.data_ptr(), o.data_ptr(), m, n, k, o32, s)
                                     : HcclGemmBf16Variant(a.data_ptr(), w.data_ptr(), o.data_ptr(), m, n, k, o32, variant, s);
    return {(int)r, std::move(o)};
}

// kind 0 AllGather + matmul, 1 matmul + ReduceScatter, 2 matmul + AllReduce
std::pair<int, at::Tensor> Fused(uint64_t comm, int kind, int64_t ranks, const at::Tensor &a, const at::Tensor &w, const std::optional<at::Tensor> &out,
                                 const std::optional<at::Tensor> &gathered, std::optional<uint64_t> stream)
{
    if (a.dim() != 2 || w.dim() < 1 || w.numel() != w.size(0) * a.size(1)) throw py::value_error("fused ops take matrices [m, k] and [n, k]");
    const int64_t m = a.size(0), k = a.size(1), n = w.size(0), rows = kind == 0 ? m * ranks : kind == 1 ? m / ranks : m;
    CheckResult(out, rows * n, false, "out");
    CheckResult(gathered, rows * k, false, "gathered");
    if (!IsOperand(a) || !IsOperand(w)) throw py::value_error("fused ops take contiguous bf16 CUDA tensors");
    py::gil_scoped_release nogil;            // ranks may be threads of one process that meet inside the call
    at::Tensor o = out ? *out : at::empty({rows, n}, a.options());
    cudaStream_t s = StreamOf(stream);
    HcclComm c = (HcclComm)(uintptr_t)comm;
    void *g = gathered ? gathered->data_ptr() : nullptr;
    const HcclResult r = kind == 0   ? HcclAllGatherMatmul(a.data_ptr(), w.data_ptr(), o.data_ptr(), g, m, n, k, HCCL_DATA_TYPE_BFP16, c, s)
                         : kind == 1 ? HcclMatmulReduceScatter(a.data_ptr(), w.data_ptr(), o.data_ptr(), m, n, k, HCCL_DATA_TYPE_BFP16, c, s)
                                     : HcclMatmulAllReduce(a.data_ptr(), w.data_ptr(), o.data_ptr(), m, n, k, HCCL_DATA_TYPE_BFP16, c, s);
    return {(int)r, std::move(o)};
}

}  // namespace

void BindFusedOps(py::module &m)
{
    m.def("gemm", &Gemm);
    m.def("fused", &Fused);
}
