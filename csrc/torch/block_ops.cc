// Autograd nodes of a decoder block's parts in native code: RMSNorm, rotary embedding, SwiGLU, the linear layers of one rank and their cross
// entropy. A small model's step is bound by the host: a Python autograd function costs 20 to 45 us a pass beside a kernel of 2 to 5,
// and its backward pass takes the interpreter from the engine's thread. These nodes check, allocate and launch in C++ and enter
// the interpreter in the backward pass only to ask whether something watches it. tiny decoder (2 layers, hidden 256, 256 tokens), forward and
// backward on one B200: 1812 us with the Python functions, 906 with these (in turn in one process).
//
// Each function returns None where it does not apply and the caller takes the Python form, which has the same kernels behind Python
// functions. A backward pass that something has to see, or whose tensors are not the plain ones that the kernels read, is handed to
// the Python form's own backward. What a node holds of Python must not lead back to a module: a graph node is invisible to the
// garbage collector, and a module may hold its own output.
#include <ATen/Context.h>
#include <ATen/SDPBackend.h>
#include <ATen/autocast_mode.h>
#include <ATen/ops/_fused_sdp_choice.h>
#include <ATen/ops/_scaled_dot_product_cudnn_attention.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>
#include <torch/extension.h>

#include <atomic>
#include <memory>
#include <mutex>

#include "hccl/hccl_mc2.h"
#include "hccl/hccl_nn.h"

namespace {

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// Python objects that the nodes use; set once by block_init and never freed.
struct Env {
    PyTypeObject *tensor = nullptr, *parameter = nullptr;
    py::object *watched = nullptr, *check = nullptr, *backward = nullptr;   // ops/block.py: _watched, _lib.check, the Python forms' backward passes
};
Env g_env;
std::atomic<bool> g_nativeGemm{true}, g_nativeWgrad{false};        // mirrors of the switches in parallel/tensor_parallel.py

// A Python object held by a graph node, which may be freed by any thread and after the interpreter is gone.
struct PyRef {
    py::object o;
    explicit PyRef(py::object v) : o(std::move(v)) {}
    PyRef(const PyRef &) = delete;
    ~PyRef()
    {
        if (!o) return;
        if (!Py_IsInitialized()) { (void)o.release(); return; }
        py::gil_scoped_acquire gil;
        o = py::object();
    }
};

bool Watched() { return (*g_env.watched)().cast<bool>(); }

void Check(HcclResult r, const char *what)
{
    if (r == HCCL_SUCCESS) return;
    py::gil_scoped_acquire gil;
    (*g_env.check)((int)r, what);
}

cudaStream_t Stream(const at::Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// The checks of ops/block.py. The interpreter is held: a plain tensor is exactly a Tensor or a Parameter, with memory of its own.
bool PlainObject(PyObject *o) { return Py_TYPE(o) == g_env.tensor || Py_TYPE(o) == g_env.parameter; }
bool Plain(const at::Tensor &t)
{
    if (!t.defined()) return false;
    py::object o = py::reinterpret_steal<py::object>(THPVariable_Wrap(t));
    return PlainObject(o.ptr()) && t.has_storage();
}
bool Dense(const at::Tensor &t, at::ScalarType type, c10::DeviceIndex device)
{
    return t.scalar_type() == type && t.is_cuda() && t.device().index() == device && t.is_contiguous() && ((uintptr_t)t.data_ptr() & 15u) == 0;
}
bool Operand(const at::Tensor &t, c10::DeviceIndex device) { return Plain(t) && Dense(t, at::kBFloat16, device) && t.numel() > 0; }
bool Floats(const at::Tensor &t, c10::DeviceIndex device) { return Plain(t) && Dense(t, at::kFloat, device) && !t.requires_grad(); }
// A tensor argument on the current GPU that a kernel may read; undefined where it may not.
at::Tensor OperandArg(py::handle h)
{
    if (!PlainObject(h.ptr())) return {};
    const at::Tensor &t = THPVariable_Unpack(h.ptr());
    return t.has_storage() && t.is_cuda() && Dense(t, at::kBFloat16, c10::cuda::current_device()) && t.numel() > 0 ? t : at::Tensor();
}
// An incoming gradient as the kernels read it.
bool PlainGrad(const at::Tensor &t) { return Plain(t) && t.scalar_type() == at::kBFloat16 && t.is_cuda(); }
at::Tensor Aligned(const at::Tensor &t)
{
    at::Tensor c = t.contiguous();
    return ((uintptr_t)c.data_ptr() & 15u) ? c.clone() : c;
}

variable_list FromPython(const py::object &r, size_t n)
{
    variable_list out(n);
    py::tuple t(r);
    for (size_t i = 0; i < n && i < t.size(); ++i)
        if (!t[i].is_none()) out[i] = t[i].cast<at::Tensor>();
    return out;
}

struct OpNode : Node {
    std::unique_ptr<PyRef> held;               // what the Python form's backward pass needs beside tensors
    struct Saved { SavedVariable *v; bool output; };
    bool traced = false;                       // compiled autograd runs this backward pass, on stand-ins
    virtual variable_list Backward(variable_list &&g) = 0;
    virtual std::vector<Saved> Keeps() = 0;
    // What the traced single operations depend on beside the node's tensors and its type.
    virtual void Constants(torch::dynamo::autograd::CompiledNodeArgs &) const {}
    // Compiled autograd takes one traced graph for all nodes that collect the same, so nothing traced may come from `held`. It cannot run a
    // backward pass inside another: the traced forms are written out.
    void compiled_args(torch::dynamo::autograd::CompiledNodeArgs &args) const override
    {
        for (const Saved &k : const_cast<OpNode *>(this)->Keeps()) args.collect(*k.v, k.output);
        Constants(args);
    }
    variable_list apply_with_saved(const variable_list &inputs, torch::dynamo::autograd::SwapSavedVariables &saved) override
    {
        for (const Saved &k : Keeps()) saved.before(*k.v);
        struct Tracing {
            bool &on;
            explicit Tracing(bool &t) : on(t) { on = true; }
            ~Tracing() { on = false; }
        } tracing(traced);
        variable_list r = apply(variable_list(inputs));
        for (const Saved &k : Keeps()) saved.after(*k.v);
        return r;
    }
    variable_list apply(variable_list &&g) final
    {
        try {
            return Backward(std::move(g));
        } catch (py::error_already_set &e) {                 // an exception of the Python form keeps its type on its way through the engine
            py::gil_scoped_acquire gil;
            e.restore();
            python_error err;
            err.persist();
            throw err;
        }
    }
    void release_variables() override
    {
        std::lock_guard<std::mutex> lock(mutex_);
        for (const Saved &k : Keeps()) k.v->reset_data();
    }
    // the saved tensors; not locked longer, since the Python form may run other graphs
    template <class... S> std::tuple<std::conditional_t<true, at::Tensor, S>...> Unpack(const S &...saved)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        auto self = shared_from_this();
        return {saved.unpack(self)...};
    }
    // whether a gradient may be asked for
    static bool Wanted(std::initializer_list<at::Tensor> in)
    {
        if (!at::GradMode::is_enabled()) return false;
        for (const at::Tensor &t : in) if (t.requires_grad()) return true;
        return false;
    }
};

template <class N, class... In> std::shared_ptr<N> MakeNode(py::object held, const In &...in)
{
    std::shared_ptr<N> n(new N(), torch::autograd::deleteNode);
    n->set_next_edges(torch::autograd::collect_next_edges(in...));
    n->held = std::make_unique<PyRef>(std::move(held));
    return n;
}

at::Tensor ZerosWhereUndefined(const at::Tensor &g, at::IntArrayRef shape, const at::TensorOptions &o) { return g.defined() ? g : at::zeros(shape, o); }
c10::DeviceIndex DeviceOf(const at::Tensor &t) { return t.is_cuda() ? t.device().index() : (c10::DeviceIndex)-1; }

// ---- RMSNorm ---------------------------------------------------------------------------------------------------------
// Outputs y and the copies of x and w that the kernel makes on its way: the backward pass reads the values that the forward pass saw, and the
// gradient of a gradient finds its way to x and w through them. With `added` the input is x + d and the copy is that sum. The copy may be used further, as the
// residual stream of a decoder: the gradient that comes back by it is added in the same kernel.
struct RmsNormNode : OpNode {
    SavedVariable x, w, rstd;
    bool added = false;
    std::string name() const override { return "_RmsNormBackward"; }
    void Constants(torch::dynamo::autograd::CompiledNodeArgs &args) const override { args.collect(added); }
    variable_list Inputs(at::Tensor dx, at::Tensor dw) const { return added ? variable_list{dx, dx, dw} : variable_list{dx, dw}; }
    std::vector<Saved> Keeps() override { return {{&x, true}, {&w, true}, {&rstd, false}}; }
    variable_list Backward(variable_list &&g) override
    {
        if (!g[0].defined()) return Inputs(g[1], g[2]);
        const auto [xv, wv, r] = Unpack(x, w, rstd);
        variable_list out(2);
        bool together = false, direct = !traced && !at::GradMode::is_enabled();
        {
            py::gil_scoped_acquire gil;
            if (direct) {
                const auto dev = DeviceOf(g[0]);
                direct = !Watched() && PlainGrad(g[0]) && Operand(xv, dev) && Operand(wv, dev) && Floats(r, dev) && xv.sizes() == g[0].sizes() && wv.dim() == 1 &&
                         wv.size(0) == xv.size(-1) && r.numel() * wv.size(0) == xv.numel();
                together = direct && g[1].defined() && PlainGrad(g[1]) && g[1].device() == g[0].device() && g[1].sizes() == g[0].sizes();
            }
            if (traced) out = FromPython((*g_env.backward)("rms_norm traced", xv, wv, r, g[0]), 2);
            else if (!direct) out = FromPython((*g_env.backward)("rms_norm", held->o, xv, wv, g[0]), 2);
        }
        if (direct) {
            const at::Tensor dy = Aligned(g[0]), past = together ? Aligned(g[1]) : at::Tensor();
            const int64_t h = xv.size(-1), rows = r.numel();
            out[0] = at::empty_like(xv);
            out[1] = at::empty_like(wv);
            const at::Tensor partial = at::empty({(int64_t)HcclRmsNormBwdParts((uint64_t)rows, (uint64_t)h), h}, r.options());
            Check(HcclRmsNormBwdAdd(dy.data_ptr(), xv.data_ptr(), wv.data_ptr(), r.data_ptr<float>(), together ? past.data_ptr() : nullptr, out[0].data_ptr(), out[1].data_ptr(),
                                    partial.data_ptr<float>(), rows, h, Stream(xv)), "HcclRmsNormBwdAdd");
        }
        for (int i = together ? 1 : 0; i < 2; ++i)
            if (g[i + 1].defined()) out[i] = out[i].defined() ? out[i] + g[i + 1] : g[i + 1];
        return Inputs(out[0], out[1]);
    }
};

bool NormOperands(const at::Tensor &x, const at::Tensor &w)
{
    if (!x.defined() || !w.defined() || x.dim() == 0) return false;
    const int64_t h = x.size(-1);
    return h % 8 == 0 && h <= 12288 && w.dim() == 1 && w.size(0) == h;
}

// y; with `kept` (y, the copy of x) where a gradient may be asked for, (y, x) where not
py::object RmsNorm(py::handle xh, py::handle wh, double eps, py::object plain, bool kept)
{
    const at::Tensor x = OperandArg(xh), w = OperandArg(wh);
    if (!NormOperands(x, w)) return py::none();
    const int64_t h = x.size(-1);
    at::Tensor y, rstd, xk, wk;
    const bool wanted = OpNode::Wanted({x, w});
    {
        auto node = wanted ? MakeNode<RmsNormNode>(std::move(plain), x, w) : nullptr;
        py::gil_scoped_release nogil;
        const uint64_t rows = (uint64_t)(x.numel() / h);
        {
            at::NoGradGuard noGrad;
            y = at::empty_like(x);
            rstd = at::empty({(int64_t)rows}, x.options().dtype(at::kFloat));
            if (wanted) {
                xk = at::empty_like(x);
                wk = at::empty_like(w);
                Check(HcclRmsNormKeep(x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr<float>(), xk.data_ptr(), wk.data_ptr(), rows, h, (float)eps, Stream(x)),
                      "HcclRmsNormKeep");
            } else {
                Check(HcclRmsNorm(x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr<float>(), rows, h, (float)eps, Stream(x)), "HcclRmsNorm");
            }
        }
        if (wanted) {
            torch::autograd::set_history({y, xk, wk}, node);
            node->x = SavedVariable(xk, true);
            node->w = SavedVariable(wk, true);
            node->rstd = SavedVariable(rstd, false);
        }
    }
    if (!kept) return py::cast(y);
    return py::make_tuple(y, wanted ? py::cast(xk) : py::reinterpret_borrow<py::object>(xh));
}

// (the norm of x + d, x + d)
py::object RmsNormAdd(py::handle xh, py::handle dh, py::handle wh, double eps, py::object plain)
{
    const at::Tensor x = OperandArg(xh), d = OperandArg(dh), w = OperandArg(wh);
    if (!NormOperands(x, w) || !d.defined() || x.sizes() != d.sizes()) return py::none();
    const int64_t h = x.size(-1);
    at::Tensor y, sum;
    {
        const bool wanted = OpNode::Wanted({x, d, w});
        auto node = wanted ? MakeNode<RmsNormNode>(std::move(plain), x, d, w) : nullptr;
        py::gil_scoped_release nogil;
        const uint64_t rows = (uint64_t)(x.numel() / h);
        at::Tensor rstd, wk;
        {
            at::NoGradGuard noGrad;
            y = at::empty_like(x);
            sum = at::empty_like(x);
            rstd = at::empty({(int64_t)rows}, x.options().dtype(at::kFloat));
            if (wanted) wk = at::empty_like(w);
            Check(HcclRmsNormAdd(x.data_ptr(), d.data_ptr(), w.data_ptr(), sum.data_ptr(), y.data_ptr(), rstd.data_ptr<float>(), wanted ? wk.data_ptr() : nullptr, rows, h,
                                 (float)eps, Stream(x)), "HcclRmsNormAdd");
        }
        if (wanted) {
            torch::autograd::set_history({y, sum, wk}, node);
            node->added = true;
            node->x = SavedVariable(sum, true);
            node->w = SavedVariable(wk, true);
            node->rstd = SavedVariable(rstd, false);
        }
    }
    return py::make_tuple(y, sum);
}

// ---- rotary embedding --------------------------------------------------------------------------------------------------
struct RopeNode : OpNode {
    SavedVariable cos, sin;
    std::vector<int64_t> in, q, kv;
    uint32_t heads = 0, kvHeads = 0, headDim = 0;
    at::TensorOptions options;
    std::string name() const override { return "_RopeQkvBackward"; }
    void Constants(torch::dynamo::autograd::CompiledNodeArgs &args) const override
    {
        for (const std::vector<int64_t> *v : {&in, &q, &kv}) args.collect(*v);
    }
    std::vector<Saved> Keeps() override { return {{&cos, false}, {&sin, false}}; }
    variable_list Backward(variable_list &&g) override
    {
        const auto [c, s] = Unpack(cos, sin);
        const at::Tensor dq = ZerosWhereUndefined(g[0], q, options), dk = ZerosWhereUndefined(g[1], kv, options), dv = ZerosWhereUndefined(g[2], kv, options);
        bool direct = !traced && !at::GradMode::is_enabled();
        {
            py::gil_scoped_acquire gil;
            if (direct) {
                const auto dev = DeviceOf(dq);
                direct = !Watched() && PlainGrad(dq) && PlainGrad(dk) && PlainGrad(dv) && Floats(c, dev) && Floats(s, dev) && c.sizes() == at::IntArrayRef({q[1], headDim / 2}) &&
                         s.sizes() == c.sizes();
            }
            if (traced) return FromPython((*g_env.backward)("rope_qkv traced", c, s, py::cast(in), dq, dk, dv), 1);
            if (!direct) return FromPython((*g_env.backward)("rope_qkv", held->o, py::cast(in), dq, dk, dv), 1);
        }
        const at::Tensor a = Aligned(dq), b = Aligned(dk), v = Aligned(dv), out = at::empty(in, a.options());
        Check(HcclRopeQkv(out.data_ptr(), a.data_ptr(), b.data_ptr(), v.data_ptr(), c.data_ptr<float>(), s.data_ptr<float>(), in[0], c.size(0), heads, kvHeads, headDim, 1,
                          Stream(out)), "HcclRopeQkv");
        return {out};
    }
};

py::object RopeQkv(py::handle qkvh, py::handle cosh, py::handle sinh, int64_t batch, int64_t heads, int64_t kvHeads, int64_t headDim, py::object plain)
{
    const at::Tensor qkv = OperandArg(qkvh);
    if (!qkv.defined() || Py_TYPE(cosh.ptr()) != g_env.tensor || Py_TYPE(sinh.ptr()) != g_env.tensor) return py::none();
    const at::Tensor cos = THPVariable_Unpack(cosh.ptr()), sin = THPVariable_Unpack(sinh.ptr());
    const auto dev = qkv.device().index();
    if (!Floats(cos, dev) || !Floats(sin, dev) || cos.dim() != 2 || qkv.dim() != 2 || headDim % 16) return py::none();
    const int64_t seq = cos.size(0), tokens = batch * seq;
    if (qkv.size(0) != tokens || qkv.size(1) != (heads + 2 * kvHeads) * headDim || cos.size(1) != headDim / 2 || cos.sizes() != sin.sizes()) return py::none();
    at::Tensor q, k, v;
    {
        const bool wanted = OpNode::Wanted({qkv});
        auto node = wanted ? MakeNode<RopeNode>(std::move(plain), qkv) : nullptr;
        py::gil_scoped_release nogil;
        {
            at::NoGradGuard noGrad;
            q = at::empty({batch, seq, heads, headDim}, qkv.options());
            k = at::empty({batch, seq, kvHeads, headDim}, qkv.options());
            v = at::empty_like(k);
            Check(HcclRopeQkv(qkv.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), cos.data_ptr<float>(), sin.data_ptr<float>(), tokens, seq, heads, kvHeads, headDim, 0,
                              Stream(qkv)), "HcclRopeQkv");
        }
        if (wanted) {
            node->cos = SavedVariable(cos, false);           // the rotation is linear: its gradient does not depend on qkv
            node->sin = SavedVariable(sin, false);
            node->in = qkv.sizes().vec();
            node->q = q.sizes().vec();
            node->kv = k.sizes().vec();
            node->options = q.options();
            node->heads = (uint32_t)heads; node->kvHeads = (uint32_t)kvHeads; node->headDim = (uint32_t)headDim;
            torch::autograd::set_history({q, k, v}, node);
        }
    }
    return py::make_tuple(q, k, v);
}

// ---- attention of short sequences ---------------------------------------------------------------------------------------
// From the packed projection to the attention's output. Forward: the rotary kernel and the library's attention, which the dispatcher would choose as well; backward: one kernel.
// Keeps the projection, which nobody but the caller's own layer may have.
struct AttentionNode : OpNode {
    SavedVariable qkv, o, lse, cos, sin;
    int64_t batch = 0, heads = 0, kvHeads = 0, headDim = 0;
    std::string name() const override { return "_AttentionBackward"; }
    void Constants(torch::dynamo::autograd::CompiledNodeArgs &args) const override
    {
        for (int64_t v : {batch, heads, kvHeads, headDim}) args.collect(v);
    }
    std::vector<Saved> Keeps() override { return {{&qkv, false}, {&o, true}, {&lse, false}, {&cos, false}, {&sin, false}}; }
    variable_list Backward(variable_list &&g) override
    {
        const auto [x, out, l, c, s] = Unpack(qkv, o, lse, cos, sin);
        const at::Tensor dO = g[0].defined() ? g[0] : at::zeros_like(out);
        bool direct = !traced && !at::GradMode::is_enabled();
        {
            py::gil_scoped_acquire gil;
            if (direct) {
                const auto dev = DeviceOf(dO);
                direct = !Watched() && PlainGrad(dO) && Operand(x, dev) && Operand(out, dev) && Floats(l, dev) && Floats(c, dev) && Floats(s, dev) && c.dim() == 2 && c.sizes() == s.sizes() &&
                         c.size(1) == headDim / 2 && x.dim() == 2 && x.size(0) == batch * c.size(0) && x.size(1) == (heads + 2 * kvHeads) * headDim && out.dim() == 2 &&
                         out.size(0) == x.size(0) && out.size(1) == heads * headDim && dO.sizes() == out.sizes() && l.numel() == x.size(0) * heads;
            }
            if (traced) return FromPython((*g_env.backward)("attention traced", x, c, s, batch, heads, kvHeads, headDim, dO), 1);
            if (!direct) return FromPython((*g_env.backward)("attention", held->o, x, dO), 1);
        }
        const at::Tensor d = Aligned(dO), dx = at::empty_like(x);
        Check(HcclAttentionBwd(d.data_ptr(), x.data_ptr(), out.data_ptr(), l.data_ptr<float>(), dx.data_ptr(), c.data_ptr<float>(), s.data_ptr<float>(), batch, c.size(0), heads,
                               kvHeads, headDim, Stream(x)), "HcclAttentionBwd");
        return {dx};
    }
};

// Whether nothing asks for another attention than the default one.
bool DefaultAttention()
{
    const at::Context &c = at::globalContext();
    return c.userEnabledFlashSDP() && c.userEnabledMemEfficientSDP() && c.userEnabledMathSDP() && c.userEnabledCuDNNSDP() && !at::autocast::is_autocast_enabled(at::kCUDA);
}

py::object Attention(py::handle qkvh, py::handle cosh, py::handle sinh, int64_t batch, int64_t heads, int64_t kvHeads, int64_t headDim, py::object plain)
{
    const at::Tensor qkv = OperandArg(qkvh);
    if (!qkv.defined() || Py_TYPE(cosh.ptr()) != g_env.tensor || Py_TYPE(sinh.ptr()) != g_env.tensor || batch <= 0 || heads <= 0 || kvHeads <= 0) return py::none();
    const at::Tensor cos = THPVariable_Unpack(cosh.ptr()), sin = THPVariable_Unpack(sinh.ptr());
    const auto dev = qkv.device().index();
    if (!Floats(cos, dev) || !Floats(sin, dev) || cos.dim() != 2 || qkv.dim() != 2 || cos.sizes() != sin.sizes() || cos.size(1) != headDim / 2) return py::none();
    const int64_t seq = cos.size(0), tokens = batch * seq;
    if (qkv.size(0) != tokens || qkv.size(1) != (heads + 2 * kvHeads) * headDim || !DefaultAttention() || !HcclAttentionBwdSuits(batch, seq, heads, kvHeads, headDim)) return py::none();
    if (!OpNode::Wanted({qkv})) return py::none();
    at::Tensor o;
    {
        auto node = MakeNode<AttentionNode>(std::move(plain), qkv);
        py::gil_scoped_release nogil;
        at::Tensor lse;
        {
            at::NoGradGuard noGrad;
            const at::Tensor q = at::empty({batch, seq, heads, headDim}, qkv.options()), k = at::empty({batch, seq, kvHeads, headDim}, qkv.options()), v = at::empty_like(k);
            const at::Tensor qt = q.transpose(1, 2), kt = k.transpose(1, 2), vt = v.transpose(1, 2);
            if (at::_fused_sdp_choice(qt, kt, vt, {}, 0.0, true, {}, heads != kvHeads) != (int64_t)at::SDPBackend::cudnn_attention) o = at::Tensor();
            else {
                Check(HcclRopeQkv(qkv.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), cos.data_ptr<float>(), sin.data_ptr<float>(), tokens, seq, heads, kvHeads, headDim, 0,
                                  Stream(qkv)), "HcclRopeQkv");
                const auto r = at::_scaled_dot_product_cudnn_attention(qt, kt, vt, {}, true, 0.0, true, false, {});
                o = std::get<0>(r).transpose(1, 2).reshape({tokens, heads * headDim});
                lse = std::get<1>(r).reshape({batch, heads, seq}).contiguous();
            }
        }
        if (o.defined()) {
            torch::autograd::set_history({o}, node);
            node->qkv = SavedVariable(qkv, false);
            node->o = SavedVariable(o, true);
            node->lse = SavedVariable(lse, false);
            node->cos = SavedVariable(cos, false);
            node->sin = SavedVariable(sin, false);
            node->batch = batch; node->heads = heads; node->kvHeads = kvHeads; node->headDim = headDim;
        }
    }
    return o.defined() ? py::cast(o) : py::none();
}

// ---- SwiGLU ------------------------------------------------------------------------------------------------------------
struct SwiGluNode : OpNode {
    SavedVariable gu;
    std::string name() const override { return "_SwiGluBackward"; }
    std::vector<Saved> Keeps() override { return {{&gu, false}}; }
    variable_list Backward(variable_list &&g) override
    {
        const auto [in] = Unpack(gu);
        const at::Tensor dh = g[0].defined() ? g[0] : at::zeros({in.size(0), in.size(1) / 2}, in.options());
        bool direct = !traced && !at::GradMode::is_enabled();
        {
            py::gil_scoped_acquire gil;
            if (traced) return FromPython((*g_env.backward)("swiglu traced", in, dh), 1);
            if (direct) direct = !Watched() && PlainGrad(dh) && Operand(in, DeviceOf(dh)) && in.dim() == 2 && dh.dim() == 2 && in.size(0) == dh.size(0) && in.size(1) == 2 * dh.size(1);
            if (!direct) return FromPython((*g_env.backward)("swiglu", held->o, in, dh), 1);
        }
        const at::Tensor d = Aligned(dh), out = at::empty_like(in);
        Check(HcclSwiGluBwd(d.data_ptr(), in.data_ptr(), out.data_ptr(), in.size(0), in.size(1) / 2, Stream(in)), "HcclSwiGluBwd");
        return {out};
    }
};

py::object SwiGlu(py::handle guh, py::object plain)
{
    const at::Tensor gu = OperandArg(guh);
    if (!gu.defined() || gu.dim() != 2 || gu.size(1) % 16) return py::none();
    at::Tensor h;
    {
        const bool wanted = OpNode::Wanted({gu});
        auto node = wanted ? MakeNode<SwiGluNode>(std::move(plain), gu) : nullptr;
        py::gil_scoped_release nogil;
        {
            at::NoGradGuard noGrad;
            h = at::empty({gu.size(0), gu.size(1) / 2}, gu.options());
            Check(HcclSwiGlu(gu.data_ptr(), h.data_ptr(), gu.size(0), gu.size(1) / 2, Stream(gu)), "HcclSwiGlu");
        }
        if (wanted) {
            node->gu = SavedVariable(gu, false);
            torch::autograd::set_history({h}, node);
        }
    }
    return py::cast(h);
}

// Gradients of a node that may keep a copy of its first input. The copy is then its second output: a gradient of the gradient finds its way to the caller's
// tensor through it, and comes back here by itself.
template <class F> variable_list WithCopy(bool copied, const variable_list &g, size_t inputs, F gradients)
{
    if (!copied || !g[1].defined()) return gradients();
    variable_list out = g[0].defined() ? gradients() : variable_list(inputs);
    out[0] = out[0].defined() ? out[0] + g[1] : g[1];
    return out;
}

// ---- linear layers of one rank -------------------------------------------------------------------------------------------
// y = x @ w^T. The column-parallel layer keeps the gathered activations, on one rank a copy of x unless the caller gives x away; the row-parallel one keeps x.
struct LinearNode : OpNode {
    SavedVariable x, w;
    std::vector<int64_t> shape;
    at::TensorOptions options;
    bool column = false, copied = false;       // copied: x is the node's own copy, see WithCopy
    std::string name() const override { return column ? "_ColumnSeqParallelBackward" : "_RowSeqParallelBackward"; }
    void Constants(torch::dynamo::autograd::CompiledNodeArgs &args) const override { args.collect(shape); args.collect(copied); }
    std::vector<Saved> Keeps() override { return {{&x, copied}, {&w, false}}; }
    variable_list Backward(variable_list &&g) override
    {
        return WithCopy(copied, g, 2, [&] { return Gradients(g[0]); });
    }
    variable_list Gradients(const at::Tensor &incoming)
    {
        const auto [xv, wv] = Unpack(x, w);
        at::Tensor dy = ZerosWhereUndefined(incoming, shape, options);
        bool direct = !traced && !at::GradMode::is_enabled() && g_nativeGemm && !g_nativeWgrad;
        {
            py::gil_scoped_acquire gil;
            if (direct) {
                const auto dev = DeviceOf(dy);
                direct = !Watched() && PlainGrad(dy) && dy.dim() == 2 && Operand(xv, dev) && Operand(wv, dev) && xv.dim() == 2 && wv.dim() == 2 && dy.numel() > 0 &&
                         dy.size(0) == xv.size(0) && dy.size(1) == wv.size(0) && wv.size(1) == xv.size(1) && xv.size(1) % 8 == 0 && py::getattr(held->o, "fused", py::bool_(true)).cast<bool>();
            }
            if (traced) return FromPython((*g_env.backward)("linear traced", xv, wv, dy), 2);
            if (!direct) return FromPython((*g_env.backward)(column ? "column" : "row", held->o, xv, wv, dy), 2);
        }
        dy = Aligned(dy);
        at::Tensor dx = at::empty(xv.sizes(), xv.options());
        Check(HcclGemmBf16Nn(dy.data_ptr(), wv.data_ptr(), dx.data_ptr(), dy.size(0), wv.size(1), wv.size(0), 0, Stream(dy)), "HcclGemmBf16Nn");
        return {dx, at::matmul(dy.t(), xv)};
    }
};

// column: all_gather_matmul, else matmul_reduce_scatter; `comm` is the communicator (one rank) and `handle` its address. own: nobody else has x, so the
// column-parallel layer needs no copy of it. Any number of rows: one rank has no tiles to agree on with others.
py::object Linear(py::handle xh, py::handle wh, py::object comm, uint64_t handle, bool column, bool own)
{
    const at::Tensor x = OperandArg(xh), w = OperandArg(wh);
    if (!x.defined() || !w.defined() || x.dim() != 2 || w.dim() != 2) return py::none();
    const int64_t m = x.size(0), k = x.size(1), n = w.size(0);
    if (w.size(1) != k || k % 8 || n % 8) return py::none();
    at::Tensor y;
    {
        const bool wanted = OpNode::Wanted({x, w});
        auto node = wanted ? MakeNode<LinearNode>(std::move(comm), x, w) : nullptr;
        py::gil_scoped_release nogil;
        at::Tensor gathered;
        {
            at::NoGradGuard noGrad;
            y = at::empty({m, n}, x.options());
            HcclComm c = (HcclComm)(uintptr_t)handle;
            if (column) {
                if (wanted && !own) gathered = at::empty({m, k}, x.options());
                Check(HcclAllGatherMatmul(x.data_ptr(), w.data_ptr(), y.data_ptr(), gathered.defined() ? gathered.data_ptr() : nullptr, m, n, k, HCCL_DATA_TYPE_BFP16, c, Stream(x)), "HcclAllGatherMatmul");
            } else {
                Check(HcclMatmulReduceScatter(x.data_ptr(), w.data_ptr(), y.data_ptr(), m, n, k, HCCL_DATA_TYPE_BFP16, c, Stream(x)), "HcclMatmulReduceScatter");
            }
        }
        if (wanted) {
            node->column = column;
            node->copied = gathered.defined();
            node->shape = y.sizes().vec();
            node->options = y.options();
            torch::autograd::set_history(node->copied ? variable_list{y, gathered} : variable_list{y}, node);
            node->x = SavedVariable(node->copied ? gathered : x, node->copied);
            node->w = SavedVariable(w, false);
        }
    }
    return py::cast(y);
}

// ---- SwiGLU layer of one rank ------------------------------------------------------------------------------------------
// y = (silu(x Wg^T) * (x Wu^T)) Wd^T with W = [Wg; Wu]: the column-parallel product, SwiGLU and the row-parallel product in one node, whose products have the
// element-wise part in their epilogues where that is faster.
struct MlpNode : OpNode {
    SavedVariable x, w, gu, h, wd;
    std::vector<int64_t> shape;
    at::TensorOptions options;
    bool copied = false;                       // x is the node's own copy, see WithCopy
    std::string name() const override { return "_SwiGluMlpBackward"; }
    void Constants(torch::dynamo::autograd::CompiledNodeArgs &args) const override { args.collect(shape); args.collect(copied); }
    std::vector<Saved> Keeps() override { return {{&x, copied}, {&w, false}, {&gu, false}, {&h, false}, {&wd, false}}; }
    variable_list Backward(variable_list &&g) override
    {
        return WithCopy(copied, g, 3, [&] { return Gradients(g[0]); });
    }
    variable_list Gradients(const at::Tensor &incoming)
    {
        const auto [xv, wv, guv, hv, wdv] = Unpack(x, w, gu, h, wd);
        at::Tensor dy = ZerosWhereUndefined(incoming, shape, options);
        bool direct = !traced && !at::GradMode::is_enabled() && g_nativeGemm && !g_nativeWgrad;
        {
            py::gil_scoped_acquire gil;
            if (direct) {
                const auto dev = DeviceOf(dy);
                direct = !Watched() && PlainGrad(dy) && dy.dim() == 2 && dy.numel() > 0;
                for (const at::Tensor &t : {xv, wv, guv, hv, wdv}) direct = direct && Operand(t, dev) && t.dim() == 2;
                direct = direct && dy.size(0) == xv.size(0) && dy.size(1) == wdv.size(0) && wv.size(1) == xv.size(1) && guv.size(0) == xv.size(0) && guv.size(1) == wv.size(0) &&
                         hv.size(0) == xv.size(0) && 2 * hv.size(1) == wv.size(0) && wdv.size(1) == hv.size(1) && xv.size(1) % 8 == 0 && hv.size(1) % 8 == 0 && dy.size(1) % 8 == 0 &&
                         py::getattr(held->o, "fused", py::bool_(true)).cast<bool>();
            }
            if (traced) return FromPython((*g_env.backward)("mlp traced", xv, wv, guv, hv, wdv, dy), 3);
            if (!direct) return FromPython((*g_env.backward)("mlp", held->o, xv, wv, guv, hv, wdv, dy), 3);
        }
        dy = Aligned(dy);
        const int64_t m = xv.size(0), f = hv.size(1);
        at::Tensor dgu = at::empty_like(guv), dh, dx = at::empty_like(xv);
        if (HcclMatmulSwiGluBwdNeedsDh(m, f, dy.size(1))) dh = at::empty_like(hv);
        Check(HcclMatmulSwiGluBwd(dy.data_ptr(), wdv.data_ptr(), guv.data_ptr(), dgu.data_ptr(), dh.defined() ? dh.data_ptr() : nullptr, m, f, dy.size(1), Stream(dy)),
              "HcclMatmulSwiGluBwd");
        const at::Tensor dwd = at::matmul(dy.t(), hv);
        Check(HcclGemmBf16Nn(dgu.data_ptr(), wv.data_ptr(), dx.data_ptr(), m, wv.size(1), 2 * f, 0, Stream(dy)), "HcclGemmBf16Nn");
        return {dx, at::matmul(dgu.t(), xv), dwd};
    }
};

py::object Mlp(py::handle xh, py::handle wh, py::handle wdh, py::object comm, uint64_t handle, bool own)
{
    const at::Tensor x = OperandArg(xh), w = OperandArg(wh), wd = OperandArg(wdh);
    if (!x.defined() || !w.defined() || !wd.defined() || x.dim() != 2 || w.dim() != 2 || wd.dim() != 2) return py::none();
    const int64_t m = x.size(0), k = x.size(1), f = wd.size(1), n = wd.size(0);
    if (w.size(1) != k || w.size(0) != 2 * f || k % 8 || f % 8 || n % 8) return py::none();
    at::Tensor y;
    {
        const bool wanted = OpNode::Wanted({x, w, wd});
        auto node = wanted ? MakeNode<MlpNode>(std::move(comm), x, w, wd) : nullptr;
        py::gil_scoped_release nogil;
        at::Tensor kept = x, gu, h;
        {
            at::NoGradGuard noGrad;
            if (wanted && !own) kept = x.clone();
            gu = at::empty({m, 2 * f}, x.options());
            h = at::empty({m, f}, x.options());
            y = at::empty({m, n}, x.options());
            Check(HcclMatmulSwiGlu(x.data_ptr(), w.data_ptr(), gu.data_ptr(), h.data_ptr(), m, f, k, wanted, Stream(x)), "HcclMatmulSwiGlu");
            Check(HcclMatmulReduceScatter(h.data_ptr(), wd.data_ptr(), y.data_ptr(), m, n, f, HCCL_DATA_TYPE_BFP16, (HcclComm)(uintptr_t)handle, Stream(x)), "HcclMatmulReduceScatter");
        }
        if (wanted) {
            node->copied = !own;
            node->shape = y.sizes().vec();
            node->options = y.options();
            torch::autograd::set_history(own ? variable_list{y} : variable_list{y, kept}, node);
            node->x = SavedVariable(kept, !own);
            node->w = SavedVariable(w, false);
            node->gu = SavedVariable(gu, false);
            node->h = SavedVariable(h, false);
            node->wd = SavedVariable(wd, false);
        }
    }
    return py::cast(y);
}

// ---- cross entropy of one rank -------------------------------------------------------------------------------------------
struct XentNode : OpNode {
    SavedVariable logits, targets, mx, packed;
    int64_t vocabStart = 0;
    at::TensorOptions options;
    std::string name() const override { return "_VocabParallelCrossEntropyBackward"; }
    void Constants(torch::dynamo::autograd::CompiledNodeArgs &args) const override { args.collect(vocabStart); }
    std::vector<Saved> Keeps() override { return {{&logits, false}, {&targets, false}, {&mx, false}, {&packed, false}}; }
    variable_list Backward(variable_list &&g) override
    {
        const auto [l, t, m, p] = Unpack(logits, targets, mx, packed);
        const at::Tensor up = ZerosWhereUndefined(g[0], {}, options);
        bool direct = !traced && !at::GradMode::is_enabled();
        {
            py::gil_scoped_acquire gil;
            if (direct) {
                const auto dev = c10::cuda::current_device();
                direct = !Watched() && Plain(up) && up.is_cuda() && Operand(l, dev) && l.dim() == 2 && Plain(t) && t.scalar_type() == at::kLong && t.device() == l.device() &&
                         t.is_contiguous() && t.dim() == 1 && t.size(0) == l.size(0) && Floats(m, dev) && m.numel() == l.size(0) && Floats(p, dev) && p.numel() == 2 * l.size(0);
            }
            if (traced) return FromPython((*g_env.backward)("xent traced", held->o, l, t, m, p, up), 1);
            if (!direct) return FromPython((*g_env.backward)("xent", held->o, l, t, m, p, up), 1);
        }
        const at::Tensor out = at::empty_like(l), scale = up.to(at::kFloat);
        Check(HcclXent(2, l.data_ptr(), t.data_ptr<int64_t>(), vocabStart, m.data_ptr<float>(), p.data_ptr<float>(), scale.data_ptr<float>(), out.data_ptr(), l.size(0),
                       l.size(1), Stream(l)), "HcclXent");
        return {out};
    }
};

py::object Xent(py::handle lh, py::handle th, int64_t vocabStart)
{
    const at::Tensor l = OperandArg(lh);
    if (!l.defined() || l.dim() != 2 || !PlainObject(th.ptr())) return py::none();
    const at::Tensor t = THPVariable_Unpack(th.ptr());
    if (!t.has_storage() || t.scalar_type() != at::kLong || t.device() != l.device() || !t.is_contiguous() || t.dim() != 1 || t.size(0) != l.size(0)) return py::none();
    at::Tensor loss;
    {
        const bool wanted = OpNode::Wanted({l});
        auto node = wanted ? MakeNode<XentNode>(py::int_(vocabStart), l) : nullptr;
        py::gil_scoped_release nogil;
        at::Tensor mx, packed, lk, tk;
        {
            at::NoGradGuard noGrad;
            const int64_t rows = l.size(0), vocab = l.size(1);
            mx = at::empty({rows}, l.options().dtype(at::kFloat));
            packed = at::empty({2, rows}, mx.options());
            loss = at::empty({}, mx.options());
            const at::Tensor each = at::empty({rows}, mx.options());
            if (wanted) { lk = at::empty_like(l); tk = at::empty_like(t); }  // the caller may write its tensors before the backward pass
            Check(HcclXentLoss(l.data_ptr(), t.data_ptr<int64_t>(), vocabStart, mx.data_ptr<float>(), packed.data_ptr<float>(), each.data_ptr<float>(), wanted ? lk.data_ptr() : nullptr,
                               wanted ? tk.data_ptr<int64_t>() : nullptr, loss.data_ptr<float>(), rows, vocab, Stream(l)), "HcclXentLoss");
        }
        if (wanted) {
            node->logits = SavedVariable(lk, false);
            node->targets = SavedVariable(tk, false);
            node->mx = SavedVariable(mx, false);
            node->packed = SavedVariable(packed, false);
            node->vocabStart = vocabStart;
            node->options = loss.options();
            torch::autograd::set_history({loss}, node);
        }
    }
    return py::cast(loss);
}

// ---- embedding ---------------------------------------------------------------------------------------------------------
// Rows of w by ids; its gradient by the few tokens' kernel.
struct EmbeddingNode : OpNode {
    SavedVariable ids;
    int64_t vocab = 0, hidden = 0, tokens = 0;
    at::TensorOptions options;
    std::string name() const override { return "_EmbeddingBackward"; }
    void Constants(torch::dynamo::autograd::CompiledNodeArgs &args) const override
    {
        for (int64_t v : {vocab, hidden, tokens}) args.collect(v);
    }
    std::vector<Saved> Keeps() override { return {{&ids, false}}; }
    variable_list Backward(variable_list &&g) override
    {
        const auto [t] = Unpack(ids);
        const at::Tensor dy = ZerosWhereUndefined(g[0], {tokens, hidden}, options);
        bool direct = !traced && !at::GradMode::is_enabled();
        {
            py::gil_scoped_acquire gil;
            if (direct)
                direct = !Watched() && PlainGrad(dy) && Plain(t) && t.scalar_type() == at::kLong && t.device() == dy.device() && t.is_contiguous() && t.dim() == 1 && dy.dim() == 2 &&
                         dy.size(0) == t.size(0) && dy.size(1) == hidden && t.size(0) > 0 && (uint64_t)t.size(0) <= HcclEmbeddingGradTokens();
            if (!direct) return FromPython((*g_env.backward)("embedding", t, vocab, hidden, dy), 1);
        }
        const at::Tensor d = Aligned(dy), dw = at::empty({vocab, hidden}, options);
        Check(HcclEmbeddingGrad(t.data_ptr<int64_t>(), d.data_ptr(), dw.data_ptr(), t.size(0), hidden, vocab, Stream(dw)), "HcclEmbeddingGrad");
        return {dw};
    }
};

py::object Embedding(py::handle wh, py::handle ih)
{
    const at::Tensor w = OperandArg(wh);
    if (!w.defined() || w.dim() != 2 || w.size(1) % 8 || !PlainObject(ih.ptr())) return py::none();
    const at::Tensor t = THPVariable_Unpack(ih.ptr());
    if (!t.has_storage() || t.scalar_type() != at::kLong || t.device() != w.device() || !t.is_contiguous() || t.dim() != 1 || t.numel() == 0 ||
        (uint64_t)t.size(0) > HcclEmbeddingGradTokens() || !OpNode::Wanted({w})) return py::none();
    at::Tensor y;
    {
        auto node = MakeNode<EmbeddingNode>(py::none(), w);
        py::gil_scoped_release nogil;
        {
            at::NoGradGuard noGrad;
            y = at::index(w, {t});
        }
        node->ids = SavedVariable(t, false);
        node->vocab = w.size(0);
        node->hidden = w.size(1);
        node->tokens = t.size(0);
        node->options = w.options().requires_grad(false);
        torch::autograd::set_history({y}, node);
    }
    return py::cast(y);
}

void Init(py::object tensor, py::object parameter, py::object check, py::object watched, py::object backward)
{
    if (g_env.watched) return;
    g_env.tensor = (PyTypeObject *)tensor.release().ptr();
    g_env.parameter = (PyTypeObject *)parameter.release().ptr();
    g_env.check = new py::object(std::move(check));
    g_env.backward = new py::object(std::move(backward));
    g_env.watched = new py::object(std::move(watched));
}

}  // namespace

void BindBlockOps(py::module &m)
{
    m.def("block_init", &Init);
    m.def("set_native_gemm", [](bool v) { g_nativeGemm = v; });
    m.def("set_native_wgrad", [](bool v) { g_nativeWgrad = v; });
    m.def("rms_norm", &RmsNorm);
    m.def("rms_norm_add", &RmsNormAdd);
    m.def("rope_qkv", &RopeQkv);
    m.def("attention", &Attention);
    m.def("swiglu", &SwiGlu);
    m.def("linear", &Linear);
    m.def("mlp", &Mlp);
    m.def("xent", &Xent);
    m.def("embedding", &Embedding);
}
