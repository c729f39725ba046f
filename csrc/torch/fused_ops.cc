// Native face of the matmul, block-scaled and MoE operators for PyTorch: argument checks, result allocation, the current stream and the C call in one
// step. A decode-sized product takes under ten microseconds on the device; the same steps in Python and ctypes took
// longer than that, so the GPU waited for the host between such calls.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/extension.h>

#include "hccl/hccl_mc2.h"
#include "hccl/hccl_moe.h"

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

// A kernel reads or writes `bytes` at the tensor's address.
void CheckMemory(const at::Tensor &t, uint64_t bytes, const char *what)
{
    if (!t.is_contiguous() || t.nbytes() < bytes) throw py::value_error(std::string(what) + " must be a contiguous tensor of at least " + std::to_string(bytes) + " bytes");
}
void CheckOnGpu(std::initializer_list<const at::Tensor *> ts)
{
    for (const at::Tensor *t : ts)
        if (!t->is_cuda()) throw py::value_error("a CUDA tensor is needed, not one on " + t->device().str());
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

c10::cuda::CUDAStream OfTorch(cudaStream_t s, c10::DeviceIndex device)
{
    return s == cudaStreamLegacy ? c10::cuda::getDefaultCUDAStream(device) : c10::cuda::getStreamFromExternal(s, device);
}

// The quantised activations live for the call alone and are allocated for the stream that uses them: a block that has just become free on another stream may still be read there.
// Nothing is shared between threads or kept between calls, and a captured graph has them in its own pool.
std::pair<int, at::Tensor> MxMatmul(uint64_t comm, const at::Tensor &a, const at::Tensor &payload, const at::Tensor &scales, int64_t n, const std::optional<at::Tensor> &out,
                                    std::optional<uint64_t> stream)
{
    if (a.dim() != 2 || n < 0 || a.scalar_type() != at::kBFloat16 || !a.is_contiguous()) throw py::value_error("the product takes contiguous bf16 activations [m, k]");
    const int64_t m = a.size(0), k = a.size(1);
    CheckResult(out, m * n, false, "out");
    CheckMemory(payload, (uint64_t)n * k, "the weight's payload");
    CheckMemory(scales, HcclMxfp8ScaleBytes(n, k), "the weight's scales");
    CheckOnGpu({&a, &payload, &scales});
    py::gil_scoped_release nogil;
    at::Tensor o = out ? *out : at::empty({m, n}, a.options());
    cudaStream_t s = StreamOf(stream);
    at::Tensor act;
    uint8_t *q = nullptr;
    if (!HcclQuantizeGemmMxfp8InOne(m, n, k)) {
        c10::cuda::OptionalCUDAStreamGuard on;
        if (stream) on.reset_stream(OfTorch(s, a.device().index()));
        act = at::empty({m * k + (int64_t)HcclMxfp8ScaleBytes(m, k)}, a.options().dtype(at::kByte));
        q = act.data_ptr<uint8_t>();
    }
    const HcclResult r = HcclQuantizeMatmulMxfp8(a.data_ptr(), q, q ? q + m * k : nullptr, payload.data_ptr(), scales.data_ptr(), o.data_ptr(), m, n, k, (HcclComm)(uintptr_t)comm, s);
    return {(int)r, std::move(o)};
}

std::tuple<int, at::Tensor, at::Tensor> MxQuantize(const at::Tensor &x, const std::optional<at::Tensor> &payload, const std::optional<at::Tensor> &scales,
                                                   std::optional<uint64_t> stream)
{
    if (x.dim() != 2 || x.scalar_type() != at::kBFloat16 || !x.is_contiguous()) throw py::value_error("quantize takes a contiguous bf16 tensor [rows, k]");
    const int64_t rows = x.size(0), k = x.size(1);
    if (payload) CheckMemory(*payload, (uint64_t)rows * k, "the payload");
    if (scales) CheckMemory(*scales, HcclMxfp8ScaleBytes(rows, k), "the scales");
    CheckOnGpu({&x, payload ? &*payload : &x, scales ? &*scales : &x});
    py::gil_scoped_release nogil;
    at::Tensor p = payload ? *payload : at::empty({rows, k}, x.options().dtype(at::kByte));
    at::Tensor f = scales ? *scales : at::empty({(int64_t)HcclMxfp8ScaleBytes(rows, k)}, x.options().dtype(at::kByte));
    const HcclResult r = HcclQuantizeMxfp8(x.data_ptr(), p.data_ptr(), f.data_ptr(), rows, k, StreamOf(stream));
    return {(int)r, std::move(p), std::move(f)};
}

// `kept` holds the tensors over the receive buffers that the caller made for the addresses `at`. -> (HcclResult, addresses, new tensors over the same memory with a
// version count of their own, or None where the addresses are others)
py::tuple MoeDispatch(uint64_t handle, int64_t topK, int64_t hidden, const at::Tensor &x, const at::Tensor &idx, std::optional<uint64_t> stream, const py::object &at, const py::tuple &kept)
{
    if (x.dim() == 0) throw py::value_error("x must be [tokens, hidden]");
    CheckMemory(x, (uint64_t)x.size(0) * hidden * 2, "x");
    CheckMemory(idx, (uint64_t)x.size(0) * topK * 4, "topk_idx");
    CheckOnGpu({&x, &idx});
    void *rx = nullptr, *rs = nullptr;
    int32_t *rc = nullptr, *src = nullptr;
    HcclResult r;
    {
        py::gil_scoped_release nogil;
        r = HcclMoeDispatch((HcclMoeHandle)(uintptr_t)handle, x.data_ptr(), idx.data_ptr<int32_t>(), (uint32_t)x.size(0), &rx, &rs, &rc, &src, StreamOf(stream));
    }
    const py::tuple now = py::make_tuple((uint64_t)(uintptr_t)rx, (uint64_t)(uintptr_t)rs, (uint64_t)(uintptr_t)rc, (uint64_t)(uintptr_t)src);
    if (r != HCCL_SUCCESS || !now.equal(at)) return py::make_tuple((int)r, now, py::none());
    py::tuple out(kept.size());
    for (size_t i = 0; i < kept.size(); ++i) out[i] = kept[i].is_none() ? py::object(py::none()) : py::cast(kept[i].cast<at::Tensor>().variable_data());
    return py::make_tuple((int)r, now, out);
}

std::pair<int, at::Tensor> MoeCombine(uint64_t handle, int64_t topK, const at::Tensor &weights, int64_t tokens, int64_t hidden, const std::optional<at::Tensor> &out,
                                      std::optional<uint64_t> stream)
{
    CheckMemory(weights, (uint64_t)tokens * topK * 4, "topk_weights");
    CheckResult(out, tokens * hidden, false, "out");
    CheckOnGpu({&weights});
    py::gil_scoped_release nogil;
    at::Tensor o = out ? *out : at::empty({tokens, hidden}, weights.options().dtype(at::kBFloat16));
    const HcclResult r = HcclMoeCombine((HcclMoeHandle)(uintptr_t)handle, weights.data_ptr<float>(), o.data_ptr(), (uint32_t)tokens, StreamOf(stream));
    return {(int)r, std::move(o)};
}

}  // namespace

void BindFusedOps(py::module &m)
{
    m.def("gemm", &Gemm);
    m.def("fused", &Fused);
    m.def("mx_matmul", &MxMatmul);
    m.def("mx_quantize", &MxQuantize);
    m.def("moe_dispatch", &MoeDispatch);
    m.def("moe_combine", &MoeCombine);
}
