"""Performance cases: what programs on one GPU have this library do, through its public entry points.

`listed()` names the cases, `draw(rng)` makes more of the same ranges, `prepare` builds what a program holds before the
call (inputs, weights, handles), `run` is one pass, `work` the bytes and operations that the pass cannot do without,
`exact` the same results in 64 bits with plain torch. Sizes are those of the repository's own configurations and
benchmarks: the Llama-3-70B MLP (hidden 8192, ffn 28672), Llama-3-8B (hidden 4096, ffn 14336, 32 / 8 heads, vocabulary
128256), MoE layers of hidden 7168 with 256 experts and top-8 routing, and the tiny decoder of the smoke test.

With one rank the fused matmul + collective operators run the tcgen05 GEMM they are built on; collectives among several
ranks run as emulated ranks in one cooperative launch.
"""
from __future__ import annotations

import math
import os
import weakref

os.environ.setdefault("HCCL_SYM_HEAP_MB", "6144")     # as the MoE benchmark sets it: a 4096-token layer needs 0.94 GB

import torch
import torch.nn.functional as F

from hccl_b200.comm import Communicator, get_root_info
from hccl_b200.models.llama import Block, Llama, LlamaConfig, _rope_tables
from hccl_b200.ops import gemm, mc2, moe, mxfp8
from hccl_b200.types import ReduceOp
from hccl_b200.utils import emu

BF16 = torch.bfloat16
_COMM = None


def _comm():
    global _COMM
    if _COMM is None:
        torch.cuda.init()
        torch.zeros(1, device="cuda")
        _COMM = Communicator.from_root_info(1, get_root_info(), 0)
    return _COMM


# ---- the cases -------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one decode step's attention output projection (8B): four sequences, the smallest product and the smallest call
        {"name": "decode_out_proj", "kind": "matmul", "op": "matmul_all_reduce", "m": 4, "n": 4096, "k": 4096},
        # a decode batch on a row-parallel shard (70B over eight ranks): the latency-bound MatmulAllReduce
        {"name": "decode_row_shard", "kind": "matmul", "op": "matmul_all_reduce", "m": 128, "n": 8192, "k": 1024},
        # a ragged prompt through the QKV projection (8B)
        {"name": "prompt_qkv_ragged", "kind": "matmul", "op": "all_gather_matmul", "m": 1000, "n": 6144, "k": 4096},
        # logits of a decode batch, 32-bit results
        {"name": "lm_head_fp32", "kind": "matmul", "op": "gemm_fp32", "m": 64, "n": 128256, "k": 4096},
        # the headline step's first half: up projection of the 70B MLP over 8192 tokens, the largest case
        {"name": "mlp_up_70b", "kind": "matmul", "op": "all_gather_matmul", "m": 8192, "n": 28672, "k": 8192},
        # block-scaled prompt: the activations are quantised in the call, the weights were quantised once
        {"name": "mx_prompt_gate_up", "kind": "mx", "op": "all_gather_matmul", "m": 2048, "n": 28672, "k": 4096},
        # block-scaled decode batch, down projection (70B over two ranks)
        {"name": "mx_decode_down", "kind": "mx", "op": "matmul_all_reduce", "m": 32, "n": 8192, "k": 14336},
        # MoE training-size dispatch + combine, bf16 on the wire
        {"name": "moe_4096_tokens", "kind": "moe", "tokens": 4096, "hidden": 7168, "experts": 256, "topk": 8, "mxfp8": False},
        # MoE decode batch, block-scaled dispatch
        {"name": "moe_decode_mx", "kind": "moe", "tokens": 100, "hidden": 7168, "experts": 256, "topk": 8, "mxfp8": True},
        # one decoder block (8B), forward and backward
        {"name": "block_train_8b", "kind": "block", "batch": 1, "seq": 2048, "hidden": 4096, "ffn": 14336, "heads": 32, "kv_heads": 8},
        # a whole tiny decoder, one training step: launches and host time count
        {"name": "tiny_decoder_step", "kind": "model", "batch": 2, "seq": 128, "hidden": 256, "ffn": 512, "heads": 8, "kv_heads": 4, "layers": 2, "vocab": 512},
        # an all-reduce among four ranks (emulated on this GPU), an odd count
        {"name": "allreduce_4_ranks", "kind": "allreduce", "ranks": 4, "count": 1000003, "dtype": "bf16", "alg": "SmAllReduceMesh1DTwoShot"},
    ]


def _log_int(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "matmul", "mx", "mx", "quantize", "moe", "moe", "block", "model", "allreduce"])
    if kind == "matmul":
        m, n, k = _log_int(rng, 1, 8192), _log_int(rng, 512, 28672, 8), _log_int(rng, 512, 16384, 8)
        return {"kind": kind, "op": rng.choice(["matmul_all_reduce", "all_gather_matmul", "matmul_reduce_scatter", "gemm_fp32"]), "m": m, "n": n, "k": k}
    if kind == "mx":
        return {"kind": kind, "op": rng.choice(["matmul_all_reduce", "all_gather_matmul", "matmul_reduce_scatter"]), "m": _log_int(rng, 1, 8192),
                "n": _log_int(rng, 512, 28672, 8), "k": _log_int(rng, 512, 16384, 128)}
    if kind == "quantize":
        return {"kind": kind, "m": _log_int(rng, 1, 16384), "k": _log_int(rng, 512, 16384, 128)}
    if kind == "moe":
        return {"kind": kind, "tokens": _log_int(rng, 1, 4096), "hidden": _log_int(rng, 1024, 7168, 256), "experts": rng.choice([8, 60, 64, 128, 256]),
                "topk": rng.choice([1, 2, 4, 6, 8]), "mxfp8": rng.random() < 0.5}
    if kind == "block":
        hidden = rng.choice([1024, 2048, 4096])
        return {"kind": kind, "batch": rng.choice([1, 2]), "seq": _log_int(rng, 128, 1024), "hidden": hidden, "ffn": hidden * 7 // 2, "heads": hidden // 128,
                "kv_heads": hidden // 512}
    if kind == "model":
        return {"kind": kind, "batch": rng.choice([1, 2, 3]), "seq": _log_int(rng, 16, 512), "hidden": 256, "ffn": 512, "heads": 8, "kv_heads": 4,
                "layers": rng.choice([1, 2, 3]), "vocab": rng.choice([512, 1000, 4096])}
    return {"kind": kind, "ranks": rng.choice([2, 4, 8]), "count": _log_int(rng, 1000, 4000000), "dtype": rng.choice(["bf16", "fp32"]),
            "alg": rng.choice(["SmAllReduceMesh1DOneShot", "SmAllReduceMesh1DTwoShot", "SmAllReducePipelined"])}


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _matmul_inputs(c, seed):
    g = _gen(seed)
    a = torch.randn(c["m"], c["k"], generator=g, device="cuda", dtype=torch.float32).to(BF16)
    w = (torch.randn(c["n"], c["k"], generator=g, device="cuda", dtype=torch.float32) * 0.02).to(BF16)
    return a, w


def _quantize_input(c, seed):
    # activations: channels of different size, a few rows of zeros
    g = _gen(seed)
    x = torch.randn(c["m"], c["k"], generator=g, device="cuda") * torch.exp(torch.randn(c["k"], generator=g, device="cuda"))
    x[:: 97] = 0
    return x.to(BF16)


def _moe_inputs(c, seed):
    T, H, E, K = c["tokens"], c["hidden"], c["experts"], c["topk"]
    g = _gen(seed)
    x = torch.randn(T, H, generator=g, device="cuda").to(BF16)
    bias = 3.0 / torch.arange(1, E + 1, device="cuda").float() ** 1.1           # Zipf-shaped popularity
    logits = torch.randn(T, E, generator=g, device="cuda") + bias[torch.randperm(E, generator=g, device="cuda")]
    top, idx = torch.topk(logits, K, dim=1)
    y = torch.randn(T * K, H, generator=g, device="cuda").to(BF16)              # what the experts returned
    return x, idx.to(torch.int32).contiguous(), torch.softmax(top, dim=1).contiguous(), y


def _block_inputs(c, seed):
    g = _gen(seed)
    t = c["batch"] * c["seq"]
    x = torch.randn(t, c["hidden"], generator=g, device="cuda").to(BF16)
    dy = torch.randn(t, c["hidden"], generator=g, device="cuda").to(BF16)
    return x, dy


def _config(c):
    return LlamaConfig(vocab_size=c.get("vocab", 512), hidden=c["hidden"], layers=c.get("layers", 32), heads=c["heads"], kv_heads=c["kv_heads"], ffn=c["ffn"],
                       max_seq=max(512, c["seq"]))


def _make_block(c, seed):
    with torch.random.fork_rng(devices=[torch.cuda.current_device()]):
        torch.manual_seed(seed)
        blk = Block(_config(c), _comm(), BF16, "cuda", None)
        with torch.no_grad():
            for norm in (blk.attn_norm, blk.mlp_norm):
                norm.weight.add_(torch.randn_like(norm.weight) * 0.1)
    return blk


def _make_model(c, seed):
    return Llama(_config(c), _comm(), dtype=BF16, device="cuda", seed=seed)


def _tokens(c, seed):
    t = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=_gen(seed), device="cuda")
    return t[:, :-1].contiguous(), t[:, 1:].contiguous()


def _allreduce_inputs(c, seed):
    g = _gen(seed)
    dt = BF16 if c["dtype"] == "bf16" else torch.float32
    return [(torch.rand(c["count"], generator=g, device="cuda") * 2 - 1).to(dt) for _ in range(c["ranks"])]


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c, "comm": _comm()}
    if kind == "matmul":
        s["a"], s["w"] = _matmul_inputs(c, seed)
    elif kind == "mx":
        s["a"], w = _matmul_inputs(c, seed)
        s["w"] = mxfp8.quantize(w)
    elif kind == "quantize":
        s["x"] = _quantize_input(c, seed)
    elif kind == "moe":
        s["x"], s["idx"], s["weights"], y = _moe_inputs(c, seed)
        d = moe.MoeDispatcher(s["comm"], c["experts"], c["topk"], c["hidden"], c["tokens"], max_recv_rows=c["tokens"] * c["topk"], mxfp8=c["mxfp8"])
        weakref.finalize(d, moe._decl().HcclMoeDestroy, d._h)
        d.expert_out.copy_(y)
        s["dispatcher"] = d
    elif kind == "block":
        s["x"], s["dy"] = _block_inputs(c, seed)
        s["x"].requires_grad_()
        s["block"] = _make_block(c, seed)
        s["params"] = list(s["block"].parameters())
        s["rope"] = _rope_tables(c["seq"], c["hidden"] // c["heads"], 500000.0, "cuda")
    elif kind == "model":
        s["model"] = _make_model(c, seed)
        s["params"] = list(s["model"].parameters())
        s["tokens"], s["targets"] = _tokens(c, seed)
    else:
        s["xs"] = _allreduce_inputs(c, seed)
        s["outs"] = [torch.empty_like(x) for x in s["xs"]]
        w = emu.EmuWorld(c["ranks"], 32 << 20)
        weakref.finalize(w, w._l.HcclEmuDestroy, w._h)
        s["world"] = w
    return s


# ---- one pass --------------------------------------------------------------------------------------------------------
def run(s):
    c, comm = s["case"], s["comm"]
    kind = c["kind"]
    if kind == "matmul":
        if c["op"] == "gemm_fp32":
            return gemm.gemm_bf16(s["a"], s["w"], out_dtype=torch.float32)
        return getattr(mc2, c["op"])(comm, s["a"], s["w"])
    if kind == "mx":
        return getattr(mxfp8, c["op"])(comm, s["a"], s["w"])
    if kind == "quantize":
        q = mxfp8.quantize(s["x"])
        return q.payload, q.scales
    if kind == "moe":
        d = s["dispatcher"]
        recv_x, recv_scales, counts, src = d.dispatch(s["x"], s["idx"])
        return recv_x, recv_scales, counts, src, d.combine(s["weights"])
    if kind == "block":
        y = s["block"](s["x"], c["batch"], c["seq"], *s["rope"])
        return [y] + list(torch.autograd.grad(y, [s["x"]] + s["params"], s["dy"]))
    if kind == "model":
        loss = s["model"](s["tokens"], s["targets"])
        return [loss] + list(torch.autograd.grad(loss, s["params"]))
    rc = s["world"].run(2, c["alg"], s["xs"], s["outs"], c["count"], s["xs"][0].dtype, ReduceOp.SUM, max_ctas=16)
    if rc:
        raise RuntimeError(f"emulated all-reduce: {rc}")
    return s["outs"]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _block_params(c):
    hd = c["hidden"] // c["heads"]
    return c["hidden"] * (c["heads"] + 2 * c["kv_heads"]) * hd + c["hidden"] * c["hidden"] + 3 * c["hidden"] * c["ffn"]


def work(case):
    c, kind = case, case["kind"]
    if kind == "matmul":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2.0 * (m * k + n * k) + (4.0 if c["op"] == "gemm_fp32" else 2.0) * m * n, "flops": 2.0 * m * n * k}
    if kind == "mx":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2.0 * m * k + n * k * 33 / 32 + 2.0 * m * n, "flops": 2.0 * m * n * k}
    if kind == "quantize":
        return {"bytes": 3.0 * c["m"] * c["k"] + c["m"] * c["k"] / 32.0, "flops": 0}
    if kind == "moe":
        rows, h = c["tokens"] * c["topk"], c["hidden"]
        sent = rows * h * (33 / 32 if c["mxfp8"] else 2.0)
        return {"bytes": 2.0 * c["tokens"] * h + sent + 2.0 * rows * h + 2.0 * c["tokens"] * h + 12.0 * rows, "flops": 2.0 * rows * h}
    if kind in ("block", "model"):
        t, layers, vocab = c["batch"] * c["seq"], c.get("layers", 1), c.get("vocab", 0)
        params = layers * _block_params(c) + vocab * c["hidden"]
        attn = layers * 2 * c["batch"] * c["seq"] ** 2 * c["hidden"]
        return {"bytes": 2.0 * (2 * params + 3 * t * c["hidden"]), "flops": 3.0 * (2 * t * params + attn)}
    return {"bytes": 2.0 * c["ranks"] * c["count"] * (2 if c["dtype"] == "bf16" else 4), "flops": 1.0 * c["ranks"] * c["count"]}


def tolerance(case):
    c, kind = case, case["kind"]
    if kind == "matmul" and c["op"] == "gemm_fp32":
        return {"rel": 4e-5, "max": 4e-4}                    # 32-bit sums of up to 16384 products (1e-5 from the 64-bit result), not rounded
    if kind == "quantize":
        return "exact"                                       # bytes
    if kind in ("block", "model"):
        return {"rel": 5e-2, "max": 0.8}                     # gradients through a dozen tensors kept in 16 bits (3e-2 from the 64-bit result)
    if kind == "allreduce" and c["dtype"] == "fp32":
        return {"rel": 1e-6, "max": 1e-5}
    return {"rel": 7e-3, "max": 1.6e-2}                      # one rounding to bf16 of 32-bit sums


# ---- the same results in 64 bits ---------------------------------------------------------------------------------------
def _mx_quantize64(x):
    """OCP MX rule: scale 2^(floor(log2(amax)) - 8) per 32 values, values rounded to e4m3 with saturation -> (values / scale, biased exponent)."""
    v = x.double().view(x.shape[0], -1, 32)
    amax = v.abs().amax(2)
    e = torch.where(amax > 0, torch.floor(torch.log2(amax.clamp_min(1e-300))), torch.full_like(amax, -127.0))
    se = (e - 8 + 127).clamp(0, 254)
    q = (v * torch.exp2(127 - se)[..., None]).clamp(-448, 448).float().to(torch.float8_e4m3fn)
    return q, se


def _mx_value64(x):
    q, se = _mx_quantize64(x)
    return (q.double() * torch.exp2(se - 127)[..., None]).view(x.shape)


def _quantize64(x):
    q, se = _mx_quantize64(x)
    rows, kb = x.shape[0], x.shape[1] // 32
    padded = (rows + 127) // 128 * 128
    full = torch.full((padded, kb), 127, dtype=torch.uint8, device=x.device)
    full[:rows] = se.to(torch.uint8)
    # atoms of 128 rows x 4 blocks: byte (row % 32) * 16 + (row % 128) / 32 * 4 + block % 4
    atoms = full.view(padded // 128, 4, 32, kb // 4, 4).permute(0, 3, 2, 1, 4).contiguous()
    return q.view(torch.uint8).view(rows, -1), atoms.view(-1)


def _dispatch_mx64(rows):
    """The dispatch's rule: the smallest power of two s with amax / s <= 448; -> e4m3 values and biased exponents."""
    v = rows.double().view(rows.shape[0], -1, 32)
    amax = v.abs().amax(2)
    e = torch.where(amax > 0, torch.ceil(torch.log2((amax / 448).clamp_min(1e-300))), torch.full_like(amax, -8.0))
    se = (e + 127).clamp(0, 254)
    q = (v * torch.exp2(127 - se)[..., None]).float().clamp(-448, 448).to(torch.float8_e4m3fn)
    return q.view(rows.shape[0], -1), se.to(torch.uint8)


def _rms64(x, w, eps=1e-5):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _rope64(x, cos, sin):
    d = x.shape[-1] // 2
    a, b, c, s = x[..., :d], x[..., d:], cos[None, :, None, :], sin[None, :, None, :]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _block64(x, p, c, cos, sin):
    """p: attn_norm, qkv, out, mlp_norm, gate_up, down in that order"""
    b, s, hd, kv = c["batch"], c["seq"], c["hidden"] // c["heads"], c["kv_heads"]
    q, k, v = (_rms64(x, p[0]) @ p[1].t()).split([c["heads"] * hd, kv * hd, kv * hd], -1)
    q = _rope64(q.reshape(b, s, c["heads"], hd), cos, sin).transpose(1, 2)
    k = _rope64(k.reshape(b, s, kv, hd), cos, sin).transpose(1, 2).repeat_interleave(c["heads"] // kv, 1)
    v = v.reshape(b, s, kv, hd).transpose(1, 2).repeat_interleave(c["heads"] // kv, 1)
    mask = torch.ones(s, s, dtype=torch.bool, device=x.device).tril()
    o = torch.softmax((q @ k.transpose(2, 3) / math.sqrt(hd)).masked_fill(~mask, -math.inf), -1) @ v
    x = x + o.transpose(1, 2).reshape(b * s, -1) @ p[2].t()
    g, u = (_rms64(x, p[3]) @ p[4].t()).chunk(2, -1)
    return x + (F.silu(g) * u) @ p[5].t()


def _block_order(prefix, names):
    order = ["attn_norm.weight", "attn.qkv.weight", "attn.out.weight", "mlp_norm.weight", "mlp.gate_up.weight", "mlp.down.weight"]
    return [names.index(prefix + o) for o in order]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "matmul":
        a, w = _matmul_inputs(c, seed)
        return a.double() @ w.double().t()
    if kind == "mx":
        a, w = _matmul_inputs(c, seed)
        return _mx_value64(a) @ _mx_value64(w).t()
    if kind == "quantize":
        return _quantize64(_quantize_input(c, seed))
    if kind == "moe":
        x, idx, weights, y = _moe_inputs(c, seed)
        t, k = idx.shape
        order = torch.argsort(idx.flatten().long(), stable=True)               # rows by expert, then by (token, choice)
        rows = x[order // k]
        slot = torch.empty_like(order)
        slot[order] = torch.arange(t * k, device="cuda")
        out = torch.zeros(t, c["hidden"], dtype=torch.float64, device="cuda")
        for j in range(k):
            out += weights[:, j, None].double() * y[slot.view(t, k)[:, j]].double()
        counts = torch.bincount(idx.flatten().long(), minlength=c["experts"]).to(torch.int32)
        src = (order // k).to(torch.int32)
        if c["mxfp8"]:
            q, se = _dispatch_mx64(rows)
            return q, se, counts, src, out
        return rows, None, counts, src, out
    if kind == "block":
        x, dy = _block_inputs(c, seed)
        blk = _make_block(c, seed)
        names = [n for n, _ in blk.named_parameters()]
        ps = [p.detach().double().requires_grad_() for p in blk.parameters()]
        x = x.double().requires_grad_()
        cos, sin = (t.double() for t in _rope_tables(c["seq"], c["hidden"] // c["heads"], 500000.0, "cuda"))
        y = _block64(x, [ps[i] for i in _block_order("", names)], c, cos, sin)
        return [y.detach()] + list(torch.autograd.grad(y, [x] + ps, dy.double()))
    if kind == "model":
        model = _make_model(c, seed)
        names = [n for n, _ in model.named_parameters()]
        ps = [p.detach().double().requires_grad_() for p in model.parameters()]
        tok, tgt = _tokens(c, seed)
        cos, sin = (t.double() for t in _rope_tables(c["seq"], c["hidden"] // c["heads"], 500000.0, "cuda"))
        x = ps[names.index("embed")][tok.reshape(-1)]
        for i in range(c["layers"]):
            x = _block64(x, [ps[j] for j in _block_order(f"blocks.{i}.", names)], c, cos, sin)
        logits = _rms64(x, ps[names.index("norm.weight")]) @ ps[names.index("lm_head.weight")].t()
        loss = F.cross_entropy(logits, tgt.reshape(-1))
        return [loss.detach()] + list(torch.autograd.grad(loss, ps))
    total = sum(x.double() for x in _allreduce_inputs(c, seed))
    return [total] * c["ranks"]
