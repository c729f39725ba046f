"""Llama-3-architecture decoder (RMSNorm, rotary embeddings, grouped-query attention, SwiGLU) with tensor + sequence
parallelism over a `Communicator`.

Between blocks the residual stream is sharded along the token dimension ([tokens / tp, hidden]); every linear is one of
the fused matmul+collective kernels (`hccl_b200.parallel.tensor_parallel`): QKV and gate/up are AllGather->matmul, the
attention output and down projections are matmul->ReduceScatter, the LM head is AllGather->matmul over a vocabulary
shard followed by a vocabulary-parallel cross entropy (two small all-reduces). With tp == 1 the same module is an
ordinary single-GPU decoder. The reference library has no model code: this module exists for the end-to-end
benchmarks that exercise the TP / DP paths the communication library is written for.
"""
from __future__ import annotations

import functools
import math
from dataclasses import dataclass
from typing import Optional

import torch
import torch.nn as nn
import torch.nn.functional as F

from ..ops import block as _block
from ..parallel.tensor_parallel import ColumnParallelLinear, RowParallelLinear, TensorParallelMLP, column_of_own, is_column, mlp_of_own


@dataclass
class LlamaConfig:
    vocab_size: int = 128256
    hidden: int = 4096
    layers: int = 32
    heads: int = 32
    kv_heads: int = 8
    ffn: int = 14336
    rope_theta: float = 500000.0
    norm_eps: float = 1e-5
    max_seq: int = 8192

    @staticmethod
    def llama3_8b() -> "LlamaConfig":
        return LlamaConfig()

    @staticmethod
    def tiny(vocab=512, hidden=256, layers=2, heads=8, kv_heads=4, ffn=512) -> "LlamaConfig":
        return LlamaConfig(vocab, hidden, layers, heads, kv_heads, ffn, max_seq=512)

    def param_count(self) -> int:
        hd = self.hidden // self.heads
        per_layer = self.hidden * (self.heads + 2 * self.kv_heads) * hd + self.hidden * self.hidden + 3 * self.hidden * self.ffn + 2 * self.hidden
        return self.layers * per_layer + 2 * self.vocab_size * self.hidden + self.hidden

    def flops_per_token(self, seq: int) -> float:
        """Forward + backward matmul FLOPs per token (6 x parameters in the linears + attention scores)."""
        hd = self.hidden // self.heads
        lin = self.layers * (self.hidden * (self.heads + 2 * self.kv_heads) * hd + self.hidden * self.hidden + 3 * self.hidden * self.ffn) \
            + self.vocab_size * self.hidden
        attn = self.layers * 2 * seq * self.hidden          # QK^T and PV, causal halves it, fwd only
        return 6.0 * lin + 6.0 * attn


class RMSNorm(nn.Module):
    def __init__(self, dim: int, eps: float, dtype, device):
        super().__init__()
        self.eps = eps
        self.weight = nn.Parameter(torch.ones(dim, dtype=dtype, device=device))
        self.weight.replicated_under_sequence_parallel = True

    def forward(self, x):
        if not torch.jit.is_scripting():
            y = _block.rms_norm(x, self.weight, self.eps, functools.partial(_plain_rms_norm, eps=self.eps))
            if y is not None:
                return y
        return self._plain(x, self.weight)

    def _plain(self, x, w):
        return _plain_rms_norm(x, w, self.eps)


_NORM_FORWARD = RMSNorm.forward


def _normed(norm, x, d=None):
    """(norm of x, x), or (norm of x + d, x + d), and whether the norm is nobody else's; in one kernel where the module is nothing but a norm."""
    if _block.native_nodes(x) is not None and _block.bare(norm, RMSNorm, _NORM_FORWARD):
        plain = functools.partial(_plain_rms_norm, eps=norm.eps)
        out = _block.rms_norm_kept(x, norm.weight, norm.eps, plain) if d is None else _block.rms_norm_add(x, d, norm.weight, norm.eps, plain)
        if out is not None:
            return *out, True
    x = x if d is None else x + d
    return norm(x), x, False


def _plain_rms_norm(x, w, eps: float):
    v = x.float()
    v = v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + eps)
    return (v * w.float()).to(x.dtype)


def _rope_tables(seq: int, head_dim: int, theta: float, device):
    inv = 1.0 / (theta ** (torch.arange(0, head_dim, 2, device=device, dtype=torch.float32) / head_dim))
    ang = torch.outer(torch.arange(seq, device=device, dtype=torch.float32), inv)
    return ang.cos(), ang.sin()


def _apply_rope(x, cos, sin):
    # x: [B, S, H, D]; rotate pairs (even, odd) halves in the "rotate_half" convention
    d = x.shape[-1] // 2
    x1, x2 = x[..., :d].float(), x[..., d:].float()
    c, s = cos[None, :, None, :], sin[None, :, None, :]
    return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], dim=-1).to(x.dtype)


class Attention(nn.Module):
    def __init__(self, cfg: LlamaConfig, comm, dtype, device, seed):
        super().__init__()
        tp = comm.size
        assert cfg.heads % tp == 0 and cfg.kv_heads % tp == 0, "heads and kv_heads must divide by the tensor-parallel size"
        self.hd = cfg.hidden // cfg.heads
        self.h_local, self.kv_local = cfg.heads // tp, cfg.kv_heads // tp
        self.cfg = cfg
        # one column-parallel weight holding this rank's [q heads; k heads; v heads]
        self.qkv = ColumnParallelLinear(comm, cfg.hidden, (cfg.heads + 2 * cfg.kv_heads) * self.hd, dtype=dtype, device=device, seed=None)
        self.out = RowParallelLinear(comm, cfg.heads * self.hd, cfg.hidden, dtype=dtype, device=device, seed=seed + 1 if seed is not None else None,
                                     init_std=0.02 / math.sqrt(2 * cfg.layers))
        if seed is not None:
            from ..parallel.tensor_parallel import _init_shard
            parts = []
            for i, (nh, nl) in enumerate(((cfg.heads, self.h_local), (cfg.kv_heads, self.kv_local), (cfg.kv_heads, self.kv_local))):
                w = torch.empty(nl * self.hd, cfg.hidden, dtype=dtype)
                _init_shard(w, 0.02, seed + 2 + i, comm.rank, 0, nh * self.hd)
                parts.append(w)
            with torch.no_grad():
                self.qkv.weight.copy_(torch.cat(parts).to(self.qkv.weight.device))

    def forward(self, x_local, batch: int, seq: int, cos, sin):
        return self._forward(x_local, batch, seq, cos, sin, False)

    def _forward(self, x_local, batch: int, seq: int, cos, sin, own: bool):
        qkv = column_of_own(self.qkv, x_local) if own else self.qkv(x_local)                                    # [B*S, (hl + 2 kvl) * hd]
        dims = dict(batch=batch, seq=seq, heads=self.h_local, kv_heads=self.kv_local, hd=self.hd, cos=cos, sin=sin)
        if is_column(self.qkv):                                             # nobody else has the projection
            o = _block.attention(qkv, cos, sin, batch, self.h_local, self.kv_local, self.hd, functools.partial(_plain_attention, **dims))
            if o is not None:
                return self.out(o)
        plain = functools.partial(_rotated, **dims)
        out = _block.rope_qkv(qkv, cos, sin, batch, self.h_local, self.kv_local, self.hd, plain)
        return self.out(_attended(*(plain(qkv) if out is None else out)))   # [B*S / tp, hidden]

    def _rotated(self, qkv, batch, seq, cos, sin):
        return _rotated(qkv, batch, seq, self.h_local, self.kv_local, self.hd, cos, sin)


_ATTENTION_FORWARD = Attention.forward


def _rotated(qkv, batch, seq, heads, kv_heads, hd, cos, sin):
    q, k, v = qkv.split([heads * hd, kv_heads * hd, kv_heads * hd], dim=-1)
    q = _apply_rope(q.reshape(batch, seq, heads, hd), cos, sin)
    k = _apply_rope(k.reshape(batch, seq, kv_heads, hd), cos, sin)
    return q, k, v.reshape(batch, seq, kv_heads, hd)


def _attended(q, k, v):
    batch, seq, heads, hd = q.shape
    o = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), is_causal=True, enable_gqa=heads != k.shape[2])
    return o.transpose(1, 2).reshape(batch * seq, heads * hd)


def _plain_attention(qkv, batch, seq, heads, kv_heads, hd, cos, sin):
    return _attended(*_rotated(qkv, batch, seq, heads, kv_heads, hd, cos, sin))


class Block(nn.Module):
    def __init__(self, cfg: LlamaConfig, comm, dtype, device, seed):
        super().__init__()
        self.attn_norm = RMSNorm(cfg.hidden, cfg.norm_eps, dtype, device)
        self.attn = Attention(cfg, comm, dtype, device, seed)
        self.mlp_norm = RMSNorm(cfg.hidden, cfg.norm_eps, dtype, device)
        self.mlp = TensorParallelMLP(comm, cfg.hidden, cfg.ffn, dtype=dtype, device=device, seed=seed + 10 if seed is not None else None)

    def forward(self, x_local, batch, seq, cos, sin):
        y, x_local, own = _normed(self.attn_norm, x_local)
        if own and _block.bare(self.attn, Attention, _ATTENTION_FORWARD):
            h = self.attn._forward(y, batch, seq, cos, sin, True)
        else:
            h = self.attn(y, batch, seq, cos, sin)
        y, x_local, own = _normed(self.mlp_norm, x_local, h)
        return x_local + (mlp_of_own(self.mlp, y) if own else self.mlp(y))


def _owned(targets, vocab_start, vloc):
    """Which targets this shard owns, and the column of each (any column where it does not)."""
    return (targets >= vocab_start) & (targets < vocab_start + vloc), (targets - vocab_start).clamp(0, vloc - 1)


class _VocabParallelCrossEntropy(torch.autograd.Function):
    """Mean cross entropy over logits sharded along the vocabulary: max and sum-exp are all-reduced, the target logit is
    contributed by the rank that owns it."""

    @staticmethod
    def forward(ctx, logits_local, targets, comm, vocab_start):
        from ..types import ReduceOp
        vloc = logits_local.shape[-1]
        ctx.fused = _block.xent_usable(logits_local, targets)
        if ctx.fused and comm.size == 1:
            loss, mx, packed, logits, kept = _block.xent_loss(logits_local, targets, vocab_start, ctx.needs_input_grad[0])
            ctx.vocab_start = vocab_start
            if ctx.needs_input_grad[0]:
                ctx.save_for_backward(logits, kept, mx, packed)
            return loss
        if ctx.fused:
            mx = _block.xent_row_max(logits_local)
        else:
            lf = logits_local.float()
            mx = lf.max(dim=-1).values.contiguous()
        if comm.size > 1:
            comm.all_reduce(mx, op=ReduceOp.MAX)
            _sync(comm, mx)
        if ctx.fused:
            packed = _block.xent_sums(logits_local, targets, vocab_start, mx)
        else:
            ex = (lf - mx[:, None]).exp()
            mine, idx = _owned(targets, vocab_start, vloc)
            tgt = torch.where(mine, lf.gather(1, idx[:, None])[:, 0] - mx, torch.zeros_like(mx))
            packed = torch.stack([ex.sum(-1), tgt]).contiguous()
        if comm.size > 1:
            comm.all_reduce(packed)
            _sync(comm, packed)
        denom, tgt = packed[0], packed[1]
        loss = (denom.log() - tgt).mean()
        if ctx.fused:
            ctx.vocab_start = vocab_start
            if ctx.needs_input_grad[0]:                                     # copies: the caller may write its tensors before the backward pass
                ctx.save_for_backward(logits_local.clone(), targets.clone(), mx, packed)
        else:
            ctx.save_for_backward(ex / denom[:, None], mine, idx)
        return loss

    @staticmethod
    def backward(ctx, g):
        if ctx.fused:
            logits, targets, mx, packed = ctx.saved_tensors
            if _block.xent_grad_usable(logits, targets, mx, packed, g):
                return _block.xent_grad(logits, targets, ctx.vocab_start, mx, packed, g), None, None, None
            return *_xent_backward(ctx.vocab_start, logits, targets, mx, packed, g), None, None, None
        return _xent_gradient(*ctx.saved_tensors, g), None, None, None


def _xent_gradient(p, mine, idx, g):
    grad = p.clone()
    grad[torch.arange(p.shape[0], device=p.device)[mine], idx[mine]] -= 1.0
    return (grad * (g / p.shape[0])).to(torch.bfloat16 if p.is_cuda else torch.float32)


def _xent_backward(vocab_start, logits, targets, mx, packed, g):
    with torch.no_grad():                                                   # what the plain form keeps
        p = (logits.float() - mx[:, None]).exp() / packed[0][:, None]
        mine, idx = _owned(targets, vocab_start, logits.shape[-1])
    return (_xent_gradient(p, mine, idx, g),)


def _xent_traced(vocab_start, logits, targets, mx, packed, g):
    """Under compiled autograd, where no shape may depend on the targets."""
    hot = torch.arange(logits.shape[-1], device=logits.device) == (targets - vocab_start)[:, None]
    p = (logits.float() - mx[:, None]).exp() / packed[0][:, None]
    return ((torch.where(hot, p - 1.0, p) * (g / p.shape[0])).to(logits.dtype),)


_block.PYTHON_BACKWARD["xent"] = _xent_backward
_block.PYTHON_BACKWARD["xent traced"] = _xent_traced


def _cross_entropy(logits_local, targets, comm, vocab_start):
    """On one rank a native node with the same kernels, where it applies."""
    n = _block.native_nodes(logits_local) if comm.size == 1 else None
    loss = None if n is None else n.xent(logits_local, targets, vocab_start)
    return _VocabParallelCrossEntropy.apply(logits_local, targets, comm, vocab_start) if loss is None else loss


def _sync(comm, t):
    if not t.is_cuda:
        comm.synchronize()


class Llama(nn.Module):
    """`forward(tokens[B, S], targets[B, S]) -> mean next-token loss` (targets given) or vocabulary-sharded logits."""

    def __init__(self, cfg: LlamaConfig, comm, *, dtype=torch.bfloat16, device=None, seed: Optional[int] = 1234):
        super().__init__()
        self.cfg, self.comm = cfg, comm
        tp = comm.size
        assert cfg.vocab_size % tp == 0
        emb = torch.empty(cfg.vocab_size, cfg.hidden, dtype=dtype, device=device)
        if seed is not None:
            emb.copy_((torch.randn(cfg.vocab_size, cfg.hidden, generator=torch.Generator().manual_seed(seed)) * 0.02).to(dtype))
        else:
            nn.init.normal_(emb, std=0.02)
        self.embed = nn.Parameter(emb)
        self.embed.replicated_under_sequence_parallel = True
        self.blocks = nn.ModuleList([Block(cfg, comm, dtype, device, seed + 100 * (i + 1) if seed is not None else None) for i in range(cfg.layers)])
        self.norm = RMSNorm(cfg.hidden, cfg.norm_eps, dtype, device)
        self.lm_head = ColumnParallelLinear(comm, cfg.hidden, cfg.vocab_size, dtype=dtype, device=device, seed=seed + 7 if seed is not None else None)
        self._rope = None

    def forward(self, tokens, targets=None):
        B, S = tokens.shape
        tp, rank = self.comm.size, self.comm.rank
        T = B * S
        assert T % tp == 0
        flat = tokens.reshape(-1)
        ids = flat if tp == 1 else flat[rank * (T // tp):(rank + 1) * (T // tp)]       # this rank's token shard
        x = _block.embedding(self.embed, ids)
        if x is None:
            x = self.embed[ids]
        if self._rope is None or self._rope[0].shape[0] != S or self._rope[0].device != x.device:
            self._rope = _rope_tables(S, self.cfg.hidden // self.cfg.heads, self.cfg.rope_theta, x.device)
        cos, sin = self._rope
        for blk in self.blocks:
            x = blk(x, B, S, cos, sin)
        y, _, own = _normed(self.norm, x)
        logits = column_of_own(self.lm_head, y) if own else self.lm_head(y)                                     # [T, vocab / tp]
        if targets is None:
            return logits
        vloc = self.cfg.vocab_size // tp
        return _cross_entropy(logits, targets.reshape(-1), self.comm, rank * vloc)

    def sync_replicated_grads(self) -> None:
        """Parameters replicated across the tensor-parallel group (embedding, norm scales) see only this rank's tokens:
        their gradients are summed over the group. One flattened all-reduce."""
        if self.comm.size == 1:
            return
        ps = [p for p in self.parameters() if getattr(p, "replicated_under_sequence_parallel", False) and p.grad is not None]
        if not ps:
            return
        flat = torch.cat([p.grad.reshape(-1).float() for p in ps]).contiguous()
        self.comm.all_reduce(flat)
        _sync(self.comm, flat)
        off = 0
        for p in ps:
            n = p.grad.numel()
            p.grad.copy_(flat[off:off + n].reshape(p.grad.shape).to(p.grad.dtype))
            off += n
