"""Tensor-parallel linear layers whose forward AND backward are the fused matmul+collective kernels.

Megatron-style sequence parallelism: activations between the two linears of a block are sharded along the token
dimension, so the column-parallel linear is AllGather -> matmul and the row-parallel linear is matmul -> ReduceScatter;
their backward passes are the mirrored pair (the gradient of AllGather->matmul is matmul->ReduceScatter and vice versa).
HCCL itself ships only the primitives and the resource-context API for such fusions (reference: include/hccl_mc2.h:25-82;
docs/zh/architecture-brief.md:16 names DP/TP as the intended users); here each direction is ONE sm_100a kernel
(`hccl_b200.ops.mc2`).

CUDA bf16 tensors take the fused kernels. CPU tensors (communicator on the host simulation backend) take the same
algebra written with the plain collectives, which is what the CPU tests compare against a single-process reference.
"""
from __future__ import annotations

import math
from typing import Optional

import torch
import torch.nn as nn

from ..ops import block as _block
from ..ops import gemm as _gemm
from ..ops import mc2 as _mc2


# ---- the three fused primitives with a host path -----------------------------------------------------------------
def _fused_ok(*ts) -> bool:
    return all(t.is_cuda and t.dtype == torch.bfloat16 for t in ts)


_NATIVE_GEMM = True


def use_native_gemm(flag: bool) -> None:
    """False routes the non-fused matmuls (weight gradients) to torch.matmul; used by the NCCL + cuBLAS baseline arm."""
    global _NATIVE_GEMM
    _NATIVE_GEMM = flag
    _tell_nodes()


def _mm_nt(a: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """a[M, K] @ w[N, K].T on the tcgen05 GEMM where its shape rules allow, torch.matmul otherwise."""
    if _NATIVE_GEMM and _fused_ok(a, w) and a.shape[1] % 8 == 0 and w.shape[0] % 8 == 0:
        return _gemm.gemm_bf16(a.contiguous(), w.contiguous())
    return a @ w.t()


def _nn_ok(comm, dy: torch.Tensor, w: torch.Tensor) -> bool:
    """The input gradient dy @ w needs no collective and the tcgen05 GEMM takes it: it reads w as stored, no transposed copy."""
    return comm.size == 1 and _NATIVE_GEMM and getattr(comm, "fused", True) and _fused_ok(dy, w) and w.shape[0] % 8 == 0 and w.shape[1] % 8 == 0 and dy.numel() > 0


_NATIVE_WGRAD = False


def use_native_wgrad(flag: bool) -> None:
    """True computes weight gradients on the tcgen05 GEMM (needs explicit transposes of both operands: its A is K-major, and the form
    that reads B MN-major is used for input gradients only); the default leaves this plain, collective-free GEMM with transposed operands to cuBLAS."""
    global _NATIVE_WGRAD
    _NATIVE_WGRAD = flag
    _tell_nodes()


def _tell_nodes() -> None:
    """The native layers have copies of the switches."""
    n = _block.nodes()
    if n is not None:
        n.set_native_gemm(_NATIVE_GEMM)
        n.set_native_wgrad(_NATIVE_WGRAD)


def _wgrad(dy: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    """dW[N, K] = dy[M, N]^T @ x[M, K]"""
    if _NATIVE_WGRAD:
        return _mm_nt(dy.t().contiguous(), x.t().contiguous())
    return dy.t() @ x


def all_gather_matmul(comm, x_local: torch.Tensor, w: torch.Tensor, want_gathered: bool = False):
    """-> (all_gather_rows(x_local) @ w.T, gathered rows or None)"""
    m, k = x_local.shape
    if getattr(comm, "fused", True) and _fused_ok(x_local, w) and m % 128 == 0 and m <= 8192 and k % 8 == 0 and w.shape[0] % 8 == 0:
        gathered = torch.empty((m * comm.size, k), dtype=x_local.dtype, device=x_local.device) if want_gathered else None
        out = _mc2.all_gather_matmul(comm, x_local.contiguous(), w.contiguous(), gathered=gathered)
        return out, gathered
    gathered = torch.empty((m * comm.size, k), dtype=x_local.dtype, device=x_local.device)
    comm.all_gather(x_local.contiguous(), gathered)
    _sync(comm, x_local)
    return _mm_nt(gathered, w), (gathered if want_gathered else None)


def matmul_reduce_scatter(comm, a: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """-> reduce_scatter_rows(a @ w.T)"""
    m, k = a.shape
    n = w.shape[0]
    if getattr(comm, "fused", True) and _fused_ok(a, w) and m % (128 * comm.size) == 0 and m // comm.size <= 8192 and k % 8 == 0 and n % 8 == 0:
        return _mc2.matmul_reduce_scatter(comm, a.contiguous(), w.contiguous())
    partial = _mm_nt(a, w).contiguous()
    out = torch.empty((m // comm.size, n), dtype=a.dtype, device=a.device)
    comm.reduce_scatter(partial, out)
    _sync(comm, a)
    return out


def matmul_all_reduce(comm, a: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """-> all_reduce(a @ w.T)"""
    if getattr(comm, "fused", True) and _fused_ok(a, w) and a.shape[1] % 8 == 0 and w.shape[0] % 64 == 0:
        return _mc2.matmul_all_reduce(comm, a.contiguous(), w.contiguous())
    out = _mm_nt(a, w).contiguous()
    comm.all_reduce(out)
    _sync(comm, a)
    return out


def _sync(comm, ref: torch.Tensor) -> None:
    if not ref.is_cuda:
        comm.synchronize()      # host backend: operators are queued on a worker


# ---- autograd ------------------------------------------------------------------------------------------------------
class _ColumnSeqParallel(torch.autograd.Function):
    """y[R*m, Nl] = AG(x[m, K]) @ W[Nl, K]^T"""

    @staticmethod
    def forward(ctx, x_local, w, comm):
        out, gathered = all_gather_matmul(comm, x_local, w, want_gathered=True)
        ctx.comm = comm
        ctx.save_for_backward(gathered, w)
        return out

    @staticmethod
    def backward(ctx, dy):
        return (*_column_backward(ctx.comm, *ctx.saved_tensors, dy), None)


def _column_backward(comm, gathered, w, dy):
    dy = dy.contiguous()
    if _nn_ok(comm, dy, w):
        dx = _gemm.gemm_bf16_nn(dy, w.contiguous())
    else:
        dx = matmul_reduce_scatter(comm, dy, w.t().contiguous())              # RS(dy @ W): the mirror of the forward
    return dx, _wgrad(dy, gathered)                                             # dy^T @ AG(x)


class _RowSeqParallel(torch.autograd.Function):
    """y[M/R, N] = RS(x[M, Kl] @ W[N, Kl]^T)"""

    @staticmethod
    def forward(ctx, x, w, comm):
        ctx.comm = comm
        ctx.save_for_backward(x, w)
        return matmul_reduce_scatter(comm, x, w)

    @staticmethod
    def backward(ctx, dy_local):
        return (*_row_backward(ctx.comm, *ctx.saved_tensors, dy_local), None)


def _row_backward(comm, x, w, dy_local):
    dyg = dy_local.contiguous()
    if _nn_ok(comm, dyg, w):
        dx = _gemm.gemm_bf16_nn(dyg, w.contiguous())
    else:
        dx, dyg = all_gather_matmul(comm, dyg, w.t().contiguous(), want_gathered=True)                         # AG(dy) @ W
    return dx, _wgrad(dyg, x)                                                                                  # AG(dy)^T @ x


def _one_rank_backward(backward):
    """The products by single operations where the gradient is itself differentiated, or a tensor is a stand-in (a traced or batched one has no memory for the kernels)."""
    return lambda comm, x, w, dy: (backward(comm, x, w, dy) if not torch.is_grad_enabled() and all([_block._plain_tensor(t) for t in (x, w, dy)])
                                   else (dy @ w, dy.t() @ x))


_block.PYTHON_BACKWARD["column"] = _one_rank_backward(_column_backward)
_block.PYTHON_BACKWARD["row"] = _one_rank_backward(_row_backward)


def _one_rank_linear(x: torch.Tensor, w: torch.Tensor, comm, column: bool, own: bool = False):
    """The sequence-parallel layer of one rank as one native node (the same kernels), or None where it does not apply. own: nobody else has x or will
    change it, so the layer may keep it as it is."""
    if comm.size != 1 or not _NATIVE_GEMM or not getattr(comm, "fused", True):
        return None
    n = _block.native_nodes(x)
    return None if n is None else n.linear(x, w, comm, comm.handle, column, own)


def _mlp_backward(comm, x, w, gu, h, wd, dy):
    """The SwiGLU layer's gradients by its parts; by single operations where something has to see them. What was kept for the kernels alone has no history: a gradient of
    the gradient starts from the input again, or from its copy, which is an output of the node."""
    if torch.is_grad_enabled() or not all([_block._plain_tensor(t) for t in (x, w, gu, h, wd, dy)]):
        return _block._plain_backward(_plain_mlp, [t if t.requires_grad else t.detach().requires_grad_() for t in (x, w, wd)], dy)
    dh, dwd = _row_backward(comm, h, wd, dy)
    dgu, = _block._plain_backward(_plain_swiglu, (gu.detach().requires_grad_(),), dh)
    return (*_column_backward(comm, x, w, dgu), dwd)


def _mlp_traced(x, w, gu, h, wd, dy):
    dgu, = _block.PYTHON_BACKWARD["swiglu traced"](gu, dy @ wd)
    return dgu @ w, dgu.t() @ x, dy.t() @ h


_block.PYTHON_BACKWARD["mlp"] = _mlp_backward
_block.PYTHON_BACKWARD["mlp traced"] = _mlp_traced


class _RowAllReduce(torch.autograd.Function):
    """y[M, N] = AR(x[M, Kl] @ W[N, Kl]^T): the decode-sized variant without sequence sharding."""

    @staticmethod
    def forward(ctx, x, w, comm):
        ctx.comm = comm
        ctx.save_for_backward(x, w)
        return matmul_all_reduce(comm, x, w)

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        dy = dy.contiguous()
        dx = _gemm.gemm_bf16_nn(dy, w.contiguous()) if _nn_ok(ctx.comm, dy, w) else _mm_nt(dy, w.t().contiguous())
        return dx, _wgrad(dy, x), None


class _ColumnReplicatedInput(torch.autograd.Function):
    """y[M, Nl] = x[M, K] @ W[Nl, K]^T with x replicated; the input gradient is all-reduced."""

    @staticmethod
    def forward(ctx, x, w, comm):
        ctx.comm = comm
        ctx.save_for_backward(x, w)
        return _mm_nt(x, w)

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        dy = dy.contiguous()
        dx = _gemm.gemm_bf16_nn(dy, w.contiguous()) if _nn_ok(ctx.comm, dy, w) else matmul_all_reduce(ctx.comm, dy, w.t().contiguous())
        return dx, _wgrad(dy, x), None


def _rows(x: torch.Tensor, width: int) -> torch.Tensor:
    """x as a matrix of rows of that width; a tensor that is one already needs no view of itself."""
    return x if type(x) is torch.Tensor and x.dim() == 2 and x.shape[1] == width else x.reshape(-1, width)


# ---- modules -------------------------------------------------------------------------------------------------------
class ColumnParallelLinear(nn.Module):
    """Weight [out_features / tp, in_features]. sequence_parallel=True: input [tokens / tp, in] -> output [tokens, out / tp]."""

    def __init__(self, comm, in_features: int, out_features: int, *, sequence_parallel: bool = True, dtype=torch.bfloat16, device=None,
                 init_std: float = 0.02, seed: Optional[int] = None):
        super().__init__()
        assert out_features % comm.size == 0
        self.comm, self.sequence_parallel = comm, sequence_parallel
        self.in_features, self.out_features = in_features, out_features
        w = torch.empty(out_features // comm.size, in_features, dtype=dtype, device=device)
        _init_shard(w, init_std, seed, comm.rank, dim=0, full=out_features)
        self.weight = nn.Parameter(w)

    def forward(self, x):
        return self._forward(x, False)

    def _forward(self, x, own: bool):
        lead, x2 = x.shape[:-1], _rows(x, self.in_features)
        if self.sequence_parallel:
            y = _one_rank_linear(x2, self.weight, self.comm, True, own)
            return _ColumnSeqParallel.apply(x2, self.weight, self.comm) if y is None else y
        return _ColumnReplicatedInput.apply(x2, self.weight, self.comm).reshape(*lead, -1)


_COLUMN_FORWARD = ColumnParallelLinear.forward


def is_column(layer: nn.Module) -> bool:
    """A column-parallel layer that is what its class says."""
    return _block.bare(layer, ColumnParallelLinear, _COLUMN_FORWARD)


def column_of_own(layer: nn.Module, x: torch.Tensor) -> torch.Tensor:
    """layer(x) for an x that the caller has made, gives to nobody else and does not change."""
    return layer._forward(x, True) if is_column(layer) else layer(x)


class RowParallelLinear(nn.Module):
    """Weight [out_features, in_features / tp]. sequence_parallel=True: input [tokens, in / tp] -> output [tokens / tp, out]."""

    def __init__(self, comm, in_features: int, out_features: int, *, sequence_parallel: bool = True, dtype=torch.bfloat16, device=None,
                 init_std: float = 0.02, seed: Optional[int] = None):
        super().__init__()
        assert in_features % comm.size == 0
        self.comm, self.sequence_parallel = comm, sequence_parallel
        self.in_features, self.out_features = in_features, out_features
        w = torch.empty(out_features, in_features // comm.size, dtype=dtype, device=device)
        _init_shard(w, init_std, seed, comm.rank, dim=1, full=in_features)
        self.weight = nn.Parameter(w)

    def forward(self, x):
        lead, x2 = x.shape[:-1], _rows(x, self.in_features // self.comm.size)
        if self.sequence_parallel:
            y = _one_rank_linear(x2, self.weight, self.comm, False)
            return _RowSeqParallel.apply(x2, self.weight, self.comm) if y is None else y
        return _RowAllReduce.apply(x2, self.weight, self.comm).reshape(*lead, -1)


_ROW_FORWARD = RowParallelLinear.forward


def _init_shard(w: torch.Tensor, std: float, seed: Optional[int], rank: int, dim: int, full: int) -> None:
    """Every rank draws the FULL matrix from the same seed and keeps its shard, so a TP model equals the unsharded one."""
    if seed is None:
        nn.init.normal_(w, std=std)
        return
    g = torch.Generator().manual_seed(seed)
    shape = list(w.shape)
    shape[dim] = full
    fullw = torch.randn(shape, generator=g, dtype=torch.float32) * std
    n = w.shape[dim]
    w.copy_(fullw.narrow(dim, rank * n, n).to(w.dtype))


class TensorParallelMLP(nn.Module):
    """SwiGLU MLP: gate/up projections column-parallel (one fused AllGather-matmul over their concatenation), down
    projection row-parallel (matmul-ReduceScatter). Input and output are token-sharded [tokens / tp, hidden]."""

    def __init__(self, comm, hidden: int, ffn: int, *, dtype=torch.bfloat16, device=None, seed: Optional[int] = None):
        super().__init__()
        self.comm = comm
        self.ffn_local = ffn // comm.size
        self.gate_up = ColumnParallelLinear(comm, hidden, 2 * ffn, dtype=dtype, device=device, seed=None)
        self.down = RowParallelLinear(comm, ffn, hidden, dtype=dtype, device=device, seed=seed + 1 if seed is not None else None,
                                      init_std=0.02 / math.sqrt(2))
        if seed is not None:   # gate and up drawn separately so that the shard layout [gate_local; up_local] matches an unsharded model
            g = torch.empty(self.ffn_local, hidden, dtype=dtype)
            u = torch.empty(self.ffn_local, hidden, dtype=dtype)
            _init_shard(g, 0.02, seed + 2, comm.rank, 0, ffn)
            _init_shard(u, 0.02, seed + 3, comm.rank, 0, ffn)
            with torch.no_grad():
                self.gate_up.weight.copy_(torch.cat([g, u]).to(self.gate_up.weight.device))

    def forward(self, x_local):
        return self._forward(x_local, False)

    def _one_rank(self, x_local, own: bool):
        """The whole layer as one native node on one rank, or None where it does not apply or a part of it is more than its class says."""
        up, down, comm = self.gate_up, self.down, self.comm
        if comm.size != 1 or not _NATIVE_GEMM or not getattr(comm, "fused", True):
            return None
        n = _block.native_nodes(x_local)
        if n is None or not is_column(up) or not _block.bare(down, RowParallelLinear, _ROW_FORWARD):
            return None
        if not (up.sequence_parallel and down.sequence_parallel and up.comm is comm and down.comm is comm):
            return None
        return n.mlp(_rows(x_local, up.in_features), up.weight, down.weight, comm, comm.handle, own)

    def _forward(self, x_local, own: bool):
        y = self._one_rank(x_local, own)
        if y is not None:
            return y
        gu = column_of_own(self.gate_up, x_local) if own else self.gate_up(x_local)
        h = _block.swiglu(gu, _plain_swiglu)
        return self.down(_plain_swiglu(gu) if h is None else h)


_MLP_FORWARD = TensorParallelMLP.forward


def mlp_of_own(mlp: nn.Module, x_local: torch.Tensor) -> torch.Tensor:
    """mlp(x_local), as `column_of_own`."""
    return mlp._forward(x_local, True) if _block.bare(mlp, TensorParallelMLP, _MLP_FORWARD) else mlp(x_local)


def _plain_swiglu(gu):
    ffn = gu.shape[1] // 2
    return torch.nn.functional.silu(gu[:, :ffn]) * gu[:, ffn:]


def _plain_mlp(x, w, wd):
    return _plain_swiglu(x @ w.t()) @ wd.t()
