"""Element-wise parts of a decoder block on one kernel each (include/hccl/hccl_nn.h): RMSNorm, rotary embedding of a packed
QKV projection, SwiGLU, vocabulary-parallel cross entropy.

Each function returns None where its kernel does not apply (another type or device, odd sizes, an active function transform,
tracing or dispatch mode) and the caller keeps its plain PyTorch form. The same plain form computes the gradient of a gradient,
and the gradient where the incoming one is batched or dual or something watches the backward pass. What the backward kernels read
is not changed by a caller that writes its tensors in between.

The autograd functions exist twice: as nodes in native code (csrc/torch/block_ops.cc), which the extension brings, and as the Python
functions below for another flavor of the library. The native nodes hand an unusual backward pass to `PYTHON_BACKWARD`.
"""
from __future__ import annotations

import ctypes
from typing import Callable, Optional

import torch
from torch.utils._device import DeviceContext

from .._ext import ops as _extension
from .._lib import check, lib

PYTHON_BACKWARD: dict = {}      # kind -> backward pass by single operations, for the native nodes


def _decl():
    l = lib()
    if not getattr(l, "_nn_declared", False):
        vp, u32, u64, i32, i64, f32 = ctypes.c_void_p, ctypes.c_uint32, ctypes.c_uint64, ctypes.c_int, ctypes.c_int64, ctypes.c_float
        l.HcclRmsNorm.argtypes = [vp, vp, vp, vp, u64, u64, f32, vp]
        l.HcclRmsNormKeep.argtypes = [vp, vp, vp, vp, vp, vp, u64, u64, f32, vp]
        l.HcclRmsNormBwdParts.argtypes = [u64, u64]
        l.HcclRmsNormBwdParts.restype = u64
        l.HcclRmsNormBwd.argtypes = [vp, vp, vp, vp, vp, vp, vp, u64, u64, vp]
        l.HcclRopeQkv.argtypes = [vp, vp, vp, vp, vp, vp, u64, u64, u32, u32, u32, i32, vp]
        l.HcclAttentionBwdSuits.argtypes = [u64, u64, u32, u32, u32]
        l.HcclAttentionBwd.argtypes = [vp, vp, vp, vp, vp, vp, vp, u64, u64, u32, u32, u32, vp]
        l.HcclSwiGlu.argtypes = [vp, vp, u64, u64, vp]
        l.HcclSwiGluBwd.argtypes = [vp, vp, vp, u64, u64, vp]
        l.HcclXent.argtypes = [i32, vp, vp, i64, vp, vp, vp, vp, u64, u64, vp]
        l.HcclXentLoss.argtypes = [vp, vp, i64, vp, vp, vp, vp, vp, vp, u64, u64, vp]
        l.HcclEmbeddingGradTokens.restype = u64
        l.HcclEmbeddingGrad.argtypes = [vp, vp, vp, u64, u64, u64, vp]
        for f in (l.HcclXentLoss, l.HcclEmbeddingGrad, l.HcclRmsNorm, l.HcclRmsNormKeep, l.HcclRmsNormBwd, l.HcclRopeQkv, l.HcclAttentionBwdSuits, l.HcclAttentionBwd, l.HcclSwiGlu, l.HcclSwiGluBwd, l.HcclXent):
            f.restype = ctypes.c_int
        l._nn_declared = True
    return l


def _stream(t: torch.Tensor) -> int:
    return torch._C._cuda_getCurrentRawStream(t.device.index)


# bound once: every forward and backward pass of a small model goes through the checks below
_transforms, _modes, _forward_ad = torch._C._functorch.peek_interpreter_stack, torch._C._len_torch_dispatch_stack, torch.autograd.forward_ad
_has_storage, _BF16 = torch._C._has_storage, torch.bfloat16
_any_global_hook = torch.nn.modules.module._has_any_global_hook


def _watched() -> bool:
    """Whether something has to see the single operations: a function transform, dispatch mode, forward-mode level, compiler or tracer."""
    return _transforms() is not None or _modes() > 0 or _forward_ad._current_level >= 0 or torch.compiler.is_compiling() or torch.jit.is_tracing()


_function_modes, _function_mode, _sdpa = torch._C._len_torch_function_stack, torch._C._get_function_stack_at, torch._C._nn.scaled_dot_product_attention


def _functions_watched() -> bool:
    """Whether a function mode has to see the operations that a caller writes as such (the attention, a residual addition, an index). The mode behind a default device
    changes where tensors are made and nothing else."""
    return _function_modes() > 0 and any(type(_function_mode(i)) is not DeviceContext for i in range(_function_modes()))


def _plain_tensor(t) -> bool:
    """Not a subclass, and with memory of its own (a batched gradient has none)."""
    return (type(t) is torch.Tensor or type(t) is torch.nn.Parameter) and _has_storage(t)


def _operand(t, device: int) -> bool:
    """A plain bf16 tensor on that GPU, contiguous and 16-byte aligned."""
    return _plain_tensor(t) and t.dtype is _BF16 and t.get_device() == device and t.is_contiguous() and t.data_ptr() % 16 == 0 and t.numel() > 0


def _usable(*ts: torch.Tensor) -> bool:
    """Operands on the current GPU, and nothing that has to see the single operations."""
    if _watched() or not _plain_tensor(ts[0]) or not ts[0].is_cuda:
        return False
    device = torch._C._cuda_getDevice()
    return all([_operand(t, device) for t in ts])


def _floats_ok(device: int, *ts) -> bool:
    """fp32 constants on that GPU, contiguous and 16-byte aligned."""
    return all([type(t) is torch.Tensor and t.dtype is torch.float32 and t.get_device() == device and t.is_contiguous() and not t.requires_grad and t.data_ptr() % 16 == 0
                for t in ts])


def _plain_backward(plain: Callable, inputs, grads):
    """Gradients of `plain(*inputs)` by the single operations, a differentiable function of inputs and grads under create_graph."""
    again = torch.is_grad_enabled()
    if not again:
        inputs = [t.detach().requires_grad_(t.requires_grad) for t in inputs]
    wanted = [t for t in inputs if t.requires_grad]
    with torch.enable_grad():
        got = iter(torch.autograd.grad(plain(*inputs), wanted, grads, create_graph=again))
    return [next(got) if t.requires_grad else None for t in inputs]


def _direct(inputs, grads):
    """The incoming gradients as the backward kernels read them, or None where the single operations have to run: a gradient that is
    itself differentiated, batched or dual, an active mode, a saved tensor that came back as something else."""
    if torch.is_grad_enabled() or _watched():
        return None
    for g in grads:
        if not _plain_tensor(g) or g.dtype is not _BF16 or not g.is_cuda:
            return None
    device = grads[0].get_device()
    for t in inputs:
        if not _operand(t, device):
            return None
    return [_aligned(g) for g in grads]


def _aligned(t: torch.Tensor) -> torch.Tensor:
    t = t.contiguous()
    return t.clone() if t.data_ptr() % 16 else t


_NODES = False


def nodes():
    """The extension with the native autograd nodes, or None where it is not in use."""
    global _NODES
    if _NODES is False:
        n = _extension()
        if n is not None:
            n.block_init(torch.Tensor, torch.nn.Parameter, check, _watched, lambda kind, *args: PYTHON_BACKWARD[kind](*args))
        _NODES = n
    return _NODES


def native_nodes(t: torch.Tensor):
    """The native nodes for an operation on t, or None where the Python form has to answer (symbolic tracing meets the type first)."""
    return nodes() if (type(t) is torch.Tensor or type(t) is torch.nn.Parameter) and not _watched() and t.is_cuda else None


PYTHON_BACKWARD["rms_norm"] = lambda plain, x, w, dy: _plain_backward(plain, (x, w), dy)
PYTHON_BACKWARD["swiglu"] = lambda plain, gu, dh: _plain_backward(plain, (gu,), dh)


def _rope_backward(plain, shape, dq, dk, dv):
    return _plain_backward(plain, (torch.zeros(shape, dtype=torch.bfloat16, device=dq.device, requires_grad=True),), (dq, dk, dv))


PYTHON_BACKWARD["rope_qkv"] = _rope_backward


# The same under compiled autograd, which traces a backward pass on stand-ins: written out, from the saved tensors alone.
def _rms_norm_traced(x, w, rstd, dy):
    r = rstd.reshape(*x.shape[:-1], 1)
    xhat, d = x.float() * r, dy.float()
    g = d * w.float()
    dx = r * (g - xhat * (g * xhat).mean(-1, keepdim=True))
    return dx.to(x.dtype), (d * xhat).flatten(0, -2).sum(0).to(w.dtype) if x.dim() > 1 else (d * xhat).to(w.dtype)


def _rope_traced(cos, sin, shape, dq, dk, dv):
    def turned_back(d):
        a, b = d.float().chunk(2, -1)
        c, s = cos[:, None], sin[:, None]
        return torch.cat([a * c + b * s, b * c - a * s], -1).to(d.dtype)

    return (torch.cat([t.flatten(2) for t in (turned_back(dq), turned_back(dk), dv)], -1).reshape(shape),)


def _swiglu_traced(gu, dh):
    g, u = gu.float().chunk(2, -1)
    d, s = dh.float(), torch.sigmoid(g)
    return (torch.cat([d * u * s * (1 + g * (1 - s)), d * (g * s)], -1).to(gu.dtype),)


PYTHON_BACKWARD["rms_norm traced"] = _rms_norm_traced
PYTHON_BACKWARD["rope_qkv traced"] = _rope_traced
PYTHON_BACKWARD["swiglu traced"] = _swiglu_traced
PYTHON_BACKWARD["linear traced"] = lambda x, w, dy: (dy @ w, dy.t() @ x)


class _RmsNorm(torch.autograd.Function):
    """-> (y, x, w). The backward pass reads copies of x and w that the kernel makes on its way, since the caller may change both before it
    (x += f(norm(x)), an optimizer step). The copies are outputs, so that the gradient of a gradient finds its way to x and w."""

    @staticmethod
    def forward(ctx, x, w, eps, plain):
        h = x.shape[-1]
        y, xk, wk = torch.empty_like(x), torch.empty_like(x), torch.empty_like(w)
        rstd = torch.empty(x.numel() // h, dtype=torch.float32, device=x.device)
        check(_decl().HcclRmsNormKeep(x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr(), xk.data_ptr(), wk.data_ptr(), rstd.numel(), h, eps, _stream(x)),
              "HcclRmsNormKeep")
        ctx.set_materialize_grads(False)
        ctx.save_for_backward(xk, wk, rstd)
        ctx.plain = plain
        return y, xk, wk

    @staticmethod
    def backward(ctx, dy, dxk, dwk):
        x, w, rstd = ctx.saved_tensors
        if dy is None:
            return dxk, dwk, None, None
        grads = _direct((x, w), (dy,))
        if grads is None or x.shape != dy.shape or w.shape != x.shape[-1:] or not _floats_ok(x.get_device(), rstd) or rstd.numel() * w.numel() != x.numel():
            dx, dw = _plain_backward(ctx.plain, (x, w), dy)
        else:
            dy, = grads
            h, rows = x.shape[-1], rstd.numel()
            dx, dw = torch.empty_like(x), torch.empty_like(w)
            l = _decl()
            partial = torch.empty(l.HcclRmsNormBwdParts(rows, h), h, dtype=torch.float32, device=x.device)
            check(l.HcclRmsNormBwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr(), dx.data_ptr(), dw.data_ptr(), partial.data_ptr(), rows, h, _stream(x)),
                  "HcclRmsNormBwd")
        return dx if dxk is None else dx + dxk, dw if dwk is None else dw + dwk, None, None


def rms_norm(x: torch.Tensor, w: torch.Tensor, eps: float, plain: Callable) -> Optional[torch.Tensor]:
    """x * rsqrt(mean(x^2) + eps) * w over the last dimension; `plain(x, w)` is the same in PyTorch. What `plain` refers to lives as long as
    the graph does."""
    n = native_nodes(x)
    if n is not None:
        return n.rms_norm(x, w, eps, plain, False)
    if not _usable(x, w):
        return None
    h = x.shape[-1] if x.dim() else 0
    if h % 8 or h > 12288 or w.shape != (h,):
        return None
    if torch.is_grad_enabled() and (x.requires_grad or w.requires_grad):
        return _RmsNorm.apply(x, w, eps, plain)[0]
    y, rstd = torch.empty_like(x), torch.empty(x.numel() // h, dtype=torch.float32, device=x.device)
    check(_decl().HcclRmsNorm(x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr(), rstd.numel(), h, eps, _stream(x)), "HcclRmsNorm")
    return y


def rms_norm_kept(x: torch.Tensor, w: torch.Tensor, eps: float, plain: Callable):
    """(norm of x, x as the residual stream goes on with it): the second is the copy that the norm makes for its backward pass, which then adds the gradient of both
    uses in one kernel. None without the native nodes."""
    n = native_nodes(x)
    return None if n is None else n.rms_norm(x, w, eps, plain, True)


def rms_norm_add(x: torch.Tensor, d: torch.Tensor, w: torch.Tensor, eps: float, plain: Callable):
    """(norm of x + d, x + d), the bits of the two operations one after the other. None without the native nodes."""
    n = native_nodes(x)
    return None if n is None or _functions_watched() else n.rms_norm_add(x, d, w, eps, plain)


def bare(module: torch.nn.Module, cls: type, forward: Callable) -> bool:
    """Whether calling the module does what `forward` of its class says and nothing else: no subclass, no replaced method, no hook of its own or of all modules."""
    return type(module) is cls and cls.forward is forward and "forward" not in module.__dict__ and module._compiled_call_impl is None and not (
        module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks or _any_global_hook())


class _RopeQkv(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, cos, sin, heads, kv_heads, head_dim, plain):
        t, seq = qkv.shape[0], cos.shape[0]
        q = torch.empty(t // seq, seq, heads, head_dim, dtype=qkv.dtype, device=qkv.device)
        k = torch.empty(t // seq, seq, kv_heads, head_dim, dtype=qkv.dtype, device=qkv.device)
        v = torch.empty_like(k)
        check(_decl().HcclRopeQkv(qkv.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), cos.data_ptr(), sin.data_ptr(), t, seq, heads, kv_heads, head_dim, 0,
                                  _stream(qkv)), "HcclRopeQkv")
        ctx.save_for_backward(cos, sin)                # the rotation is linear: its gradient does not depend on qkv
        ctx.shape, ctx.dims, ctx.table, ctx.plain = qkv.shape, (heads, kv_heads, head_dim), cos.shape, plain
        return q, k, v

    @staticmethod
    def backward(ctx, dq, dk, dv):
        cos, sin = ctx.saved_tensors
        grads = _direct((), (dq, dk, dv))
        if grads is None or not _floats_ok(grads[0].get_device(), cos, sin) or not cos.shape == sin.shape == ctx.table:
            return (*_rope_backward(ctx.plain, ctx.shape, dq, dk, dv), None, None, None, None, None, None)
        dq, dk, dv = grads
        out = torch.empty(ctx.shape, dtype=dq.dtype, device=dq.device)
        check(_decl().HcclRopeQkv(out.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), cos.data_ptr(), sin.data_ptr(), ctx.shape[0], cos.shape[0], *ctx.dims, 1,
                                  _stream(out)), "HcclRopeQkv")
        return out, None, None, None, None, None, None


def rope_qkv(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, batch: int, heads: int, kv_heads: int, head_dim: int, plain: Callable):
    """Packed [batch * seq, (heads + 2 kv_heads) * head_dim] -> rotated q, k and v as [batch, seq, heads, head_dim]; cos / sin are fp32
    [seq, head_dim / 2] constants. `plain(qkv)` is the same in PyTorch."""
    n = native_nodes(qkv)
    if n is not None:
        return n.rope_qkv(qkv, cos, sin, batch, heads, kv_heads, head_dim, plain)
    if not _usable(qkv) or not _floats_ok(qkv.get_device(), cos, sin):
        return None
    seq = cos.shape[0] if cos.dim() else 0
    if head_dim % 16 or qkv.shape != (batch * seq, (heads + 2 * kv_heads) * head_dim) or cos.shape != (seq, head_dim // 2) or sin.shape != cos.shape:
        return None
    return _RopeQkv.apply(qkv, cos, sin, heads, kv_heads, head_dim, plain)


class _Attention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, cos, sin, dims, plain):
        batch, heads, kv_heads, head_dim = dims
        q, k, v = _RopeQkv.apply(qkv, cos, sin, heads, kv_heads, head_dim, plain)
        o, lse = torch.ops.aten._scaled_dot_product_cudnn_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), None, True, 0.0, True, False)[:2]
        o, lse = o.transpose(1, 2).reshape(qkv.shape[0], heads * head_dim), lse.reshape(batch, heads, -1).contiguous()
        ctx.save_for_backward(qkv, o, lse, cos, sin)
        ctx.dims, ctx.seq, ctx.plain = dims, cos.shape[0], plain
        return o

    @staticmethod
    def backward(ctx, do):
        qkv, o, lse, cos, sin = ctx.saved_tensors
        batch, heads, kv_heads, head_dim = ctx.dims
        tokens, grads = batch * ctx.seq, _direct((qkv, o), (do,))
        if grads is None or qkv.shape != (tokens, (heads + 2 * kv_heads) * head_dim) or o.shape != (tokens, heads * head_dim) or do.shape != o.shape \
                or not _floats_ok(qkv.get_device(), lse, cos, sin) or lse.numel() != tokens * heads or not cos.shape == sin.shape == (ctx.seq, head_dim // 2):
            return (*_plain_backward(ctx.plain, (qkv,), do), None, None, None, None)
        do, = grads
        out = torch.empty_like(qkv)
        check(_decl().HcclAttentionBwd(do.data_ptr(), qkv.data_ptr(), o.data_ptr(), lse.data_ptr(), out.data_ptr(), cos.data_ptr(), sin.data_ptr(), batch, ctx.seq, heads, kv_heads,
                                       head_dim, _stream(qkv)), "HcclAttentionBwd")
        return out, None, None, None, None


def _default_attention() -> bool:
    b = torch.backends.cuda
    return b.flash_sdp_enabled() and b.mem_efficient_sdp_enabled() and b.math_sdp_enabled() and b.cudnn_sdp_enabled() and not torch.is_autocast_enabled("cuda")


def attention(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, batch: int, heads: int, kv_heads: int, head_dim: int, plain: Callable) -> Optional[torch.Tensor]:
    """Causal attention from the packed projection, [batch * seq, heads * head_dim], for sequences short enough that the backward kernel is the better choice, where a gradient may be asked for and
    the library's attention would run anyway (no function mode, and nothing in the place of `scaled_dot_product_attention`); the tables as `rope_qkv`. The projection is kept as it is, so nobody else
    may change it. `plain(qkv)` is the same in PyTorch."""
    n = native_nodes(qkv)
    if (n is None and not _usable(qkv)) or _functions_watched() or torch.nn.functional.scaled_dot_product_attention is not _sdpa:
        return None
    if n is not None:
        return n.attention(qkv, cos, sin, batch, heads, kv_heads, head_dim, plain)
    if not _floats_ok(qkv.get_device(), cos, sin) or not _default_attention() or not (torch.is_grad_enabled() and qkv.requires_grad):
        return None
    seq = cos.shape[0] if cos.dim() else 0
    if qkv.shape != (batch * seq, (heads + 2 * kv_heads) * head_dim) or cos.shape != (seq, head_dim // 2) or sin.shape != cos.shape:
        return None
    if not _decl().HcclAttentionBwdSuits(batch, seq, heads, kv_heads, head_dim):
        return None
    q, k = (torch.empty(batch, seq, h, head_dim, dtype=qkv.dtype, device=qkv.device).transpose(1, 2) for h in (heads, kv_heads))
    if torch._fused_sdp_choice(q, k, k, is_causal=True, enable_gqa=heads != kv_heads) != torch.nn.attention.SDPBackend.CUDNN_ATTENTION.value:
        return None
    return _Attention.apply(qkv, cos, sin, (batch, heads, kv_heads, head_dim), plain)


PYTHON_BACKWARD["attention"] = lambda plain, qkv, do: _plain_backward(plain, (qkv,), do)


def _attention_traced(qkv, cos, sin, batch, heads, kv_heads, head_dim, do):
    seq, half = cos.shape[0], head_dim // 2
    c, s, group = cos[:, None], sin[:, None], heads // kv_heads
    q, k, v = qkv.float().reshape(batch, seq, -1, head_dim).split([heads, kv_heads, kv_heads], 2)
    turned = lambda t, sn: torch.cat([t[..., :half] * c - t[..., half:] * sn, t[..., half:] * c + t[..., :half] * sn], -1)
    q, k, v, d = (t.transpose(1, 2) for t in (turned(q, s), turned(k, s).repeat_interleave(group, 2), v.repeat_interleave(group, 2), do.float().reshape(batch, seq, heads, head_dim)))
    hidden = torch.arange(seq, device=qkv.device)[None] > torch.arange(seq, device=qkv.device)[:, None]
    p = ((q @ k.transpose(2, 3)) * head_dim ** -0.5).masked_fill(hidden, float("-inf")).softmax(-1)
    dp = d @ v.transpose(2, 3)
    ds = p * (dp - (p * dp).sum(-1, keepdim=True)) * head_dim ** -0.5
    per_key = lambda t: t.reshape(batch, kv_heads, group, seq, head_dim).sum(2).transpose(1, 2)
    parts = turned((ds @ k).transpose(1, 2), -s), turned(per_key(ds.transpose(2, 3) @ q), -s), per_key(p.transpose(2, 3) @ d)
    return (torch.cat(parts, 2).reshape(qkv.shape).to(qkv.dtype),)


PYTHON_BACKWARD["attention traced"] = _attention_traced


class _SwiGlu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gu, plain):
        t, f = gu.shape[0], gu.shape[1] // 2
        h = torch.empty(t, f, dtype=gu.dtype, device=gu.device)
        check(_decl().HcclSwiGlu(gu.data_ptr(), h.data_ptr(), t, f, _stream(gu)), "HcclSwiGlu")
        ctx.save_for_backward(gu)
        ctx.plain = plain
        return h

    @staticmethod
    def backward(ctx, dh):
        gu, = ctx.saved_tensors
        grads = _direct((gu,), (dh,))
        if grads is None or gu.shape != (dh.shape[0], 2 * dh.shape[1]):
            return (*_plain_backward(ctx.plain, (gu,), dh), None)
        dh, = grads
        out = torch.empty_like(gu)
        check(_decl().HcclSwiGluBwd(dh.data_ptr(), gu.data_ptr(), out.data_ptr(), gu.shape[0], gu.shape[1] // 2, _stream(gu)), "HcclSwiGluBwd")
        return out, None


def swiglu(gu: torch.Tensor, plain: Callable) -> Optional[torch.Tensor]:
    """silu(gate) * up for gu = [rows, gate | up]; `plain(gu)` is the same in PyTorch."""
    n = native_nodes(gu)
    if n is not None:
        return n.swiglu(gu, plain)
    if not _usable(gu) or gu.dim() != 2 or gu.shape[1] % 16:
        return None
    return _SwiGlu.apply(gu, plain)


def xent_usable(logits: torch.Tensor, targets: torch.Tensor) -> bool:
    return _usable(logits) and logits.dim() == 2 and _plain_tensor(targets) and targets.dtype is torch.int64 and targets.get_device() == logits.get_device() \
        and targets.is_contiguous() and targets.shape == logits.shape[:1]


def xent_grad_usable(logits: torch.Tensor, targets: torch.Tensor, mx: torch.Tensor, packed: torch.Tensor, g: torch.Tensor) -> bool:
    """Whether the gradient kernel may answer this backward pass: a gradient that is itself differentiated, batched or dual has to see
    the operations, and so has a saved tensor that came back as something else."""
    return not torch.is_grad_enabled() and _plain_tensor(g) and g.is_cuda and xent_usable(logits, targets) and _floats_ok(logits.get_device(), mx, packed) \
        and mx.shape == logits.shape[:1] and packed.shape == (2, logits.shape[0])


def xent_row_max(logits: torch.Tensor) -> torch.Tensor:
    mx = torch.empty(logits.shape[0], dtype=torch.float32, device=logits.device)
    check(_decl().HcclXent(0, logits.data_ptr(), None, 0, mx.data_ptr(), None, None, None, *logits.shape, _stream(logits)), "HcclXent")
    return mx


def xent_sums(logits: torch.Tensor, targets: torch.Tensor, vocab_start: int, mx: torch.Tensor) -> torch.Tensor:
    """[2, rows]: sum of exp(logit - max) over this shard, the target's logit - max (0 where another shard owns it)."""
    packed = torch.empty(2, logits.shape[0], dtype=torch.float32, device=logits.device)
    check(_decl().HcclXent(1, logits.data_ptr(), targets.data_ptr(), vocab_start, mx.data_ptr(), packed.data_ptr(), None, None, *logits.shape, _stream(logits)), "HcclXent")
    return packed


def xent_grad(logits: torch.Tensor, targets: torch.Tensor, vocab_start: int, mx: torch.Tensor, packed: torch.Tensor, g: torch.Tensor) -> torch.Tensor:
    out, g = torch.empty_like(logits), g.float()
    check(_decl().HcclXent(2, logits.data_ptr(), targets.data_ptr(), vocab_start, mx.data_ptr(), packed.data_ptr(), g.data_ptr(), out.data_ptr(), *logits.shape,
                           _stream(logits)), "HcclXent")
    return out


def xent_loss(logits: torch.Tensor, targets: torch.Tensor, vocab_start: int, kept: bool):
    """One rank: the mean loss, the row maxima and sums as above, and copies of logits and targets (or None) for a backward pass after they have changed."""
    rows, vocab = logits.shape
    mx, packed, each = (torch.empty(*s, dtype=torch.float32, device=logits.device) for s in ((rows,), (2, rows), (rows,)))
    loss = torch.empty((), dtype=torch.float32, device=logits.device)
    lk, tk = (torch.empty_like(logits), torch.empty_like(targets)) if kept else (None, None)
    check(_decl().HcclXentLoss(logits.data_ptr(), targets.data_ptr(), vocab_start, mx.data_ptr(), packed.data_ptr(), each.data_ptr(), lk.data_ptr() if kept else None,
                               tk.data_ptr() if kept else None, loss.data_ptr(), rows, vocab, _stream(logits)), "HcclXentLoss")
    return loss, mx, packed, lk, tk


def _embedding_backward(ids, vocab, hidden, dy):
    return (torch.zeros(vocab, hidden, dtype=dy.dtype, device=dy.device).index_put((ids,), dy, accumulate=True),)


PYTHON_BACKWARD["embedding"] = _embedding_backward


class _Embedding(torch.autograd.Function):
    @staticmethod
    def forward(ctx, w, ids):
        ctx.save_for_backward(ids)
        ctx.shape = tuple(w.shape)
        return w[ids]

    @staticmethod
    def backward(ctx, dy):
        ids, = ctx.saved_tensors
        vocab, hidden = ctx.shape
        grads = _direct((), (dy,))
        if grads is None or not _plain_tensor(ids) or ids.dtype is not torch.int64 or ids.device != dy.device or not ids.is_contiguous() \
                or dy.shape != (*ids.shape, hidden) or not 0 < ids.numel() <= _decl().HcclEmbeddingGradTokens():
            return (*_embedding_backward(ids, vocab, hidden, dy), None)
        dy, = grads
        dw = torch.empty(ctx.shape, dtype=dy.dtype, device=dy.device)
        check(_decl().HcclEmbeddingGrad(ids.data_ptr(), dy.data_ptr(), dw.data_ptr(), ids.numel(), hidden, vocab, _stream(dw)), "HcclEmbeddingGrad")
        return dw, None


def embedding(w: torch.Tensor, ids: torch.Tensor) -> Optional[torch.Tensor]:
    """w[ids] for a vector of few ids, whose gradient then takes one kernel."""
    n = native_nodes(w)
    if (n is None and not _usable(w)) or _functions_watched():
        return None
    if n is not None:
        return n.embedding(w, ids)
    if not (torch.is_grad_enabled() and w.requires_grad) or w.dim() != 2 or w.shape[1] % 8 or not _plain_tensor(ids):
        return None
    if ids.dtype is not torch.int64 or ids.device != w.device or not ids.is_contiguous() or ids.dim() != 1 or not 0 < ids.numel() <= _decl().HcclEmbeddingGradTokens():
        return None
    return _Embedding.apply(w, ids)
