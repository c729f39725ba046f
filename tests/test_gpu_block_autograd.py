"""The one-kernel parts of a decoder block under autograd: what the plain operations took has to be taken, with the same meaning."""
import os

import pytest
import torch

pytestmark = pytest.mark.gpu


def _native_nodes():
    """The extension with the native autograd nodes; without it a test of them would compare the Python functions with themselves."""
    from hccl_b200.ops import block
    if os.environ.get("HCCL_B200_LIB"):
        pytest.skip("another flavor of the library runs the Python functions")
    assert block.nodes() is not None
    return block.nodes()


def _is_native(t):
    return t.grad_fn is not None and not isinstance(t.grad_fn, torch.autograd.function.BackwardCFunction)


class _OneRank:
    size, rank = 1, 0


def _close(got, ref, mag, terms):
    """|got - ref| within one rounding to bf16 plus 32-bit arithmetic over `terms` terms of size `mag`."""
    err, bound = (got.double() - ref).abs(), ref.abs() * 2.0 ** -8 + mag * (terms + 16) * 2.0 ** -23
    assert bool((err <= bound + 1e-30).all()), (err - bound).max().item()


def _logits(rows=6, vocab=24):
    g = torch.Generator(device="cuda").manual_seed(rows)
    logits = torch.randn(rows, vocab, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    targets = torch.randint(0, vocab, (rows,), generator=g, device="cuda")
    p = torch.softmax(logits.detach().double(), 1)
    hot = torch.nn.functional.one_hot(targets, vocab).double()
    return logits, targets, (p - hot) / rows, (p + hot) / rows


def test_cross_entropy_gradient_depends_on_the_incoming_gradient():
    """create_graph: the derivative of sum(gradient * c) by the loss's scale; batched and dual incoming gradients."""
    from hccl_b200.models.llama import _VocabParallelCrossEntropy as X
    import torch.autograd.forward_ad as fw
    logits, targets, ref, mag = _logits()
    c = torch.rand(logits.shape, device="cuda")
    scale = torch.tensor(2.0, device="cuda", requires_grad=True)
    g, = torch.autograd.grad(X.apply(logits, targets, _OneRank, 0) * scale, logits, create_graph=True)
    _close(g.detach(), 2 * ref, 2 * mag, logits.shape[1])
    d, = torch.autograd.grad((g.float() * c).sum(), scale)
    # the sum's gradient travels back through bf16: one more rounding of each c
    bound = (ref.abs() * c.double()).sum() * 2.0 ** -7 + (mag * c.double()).sum() * 2.0 ** -16
    assert abs(d.item() - (ref * c.double()).sum().item()) <= bound.item()
    ups = torch.tensor([1.0, -3.0, 0.5], device="cuda")
    gb, = torch.autograd.grad(X.apply(logits, targets, _OneRank, 0), logits, ups, is_grads_batched=True)
    for u, got in zip(ups.tolist(), gb):
        _close(got, u * ref, abs(u) * mag, logits.shape[1])
    loss = X.apply(logits, targets, _OneRank, 0)
    with fw.dual_level():
        gd, = torch.autograd.grad(loss, logits, fw.make_dual(torch.tensor(1.0, device="cuda"), torch.tensor(3.0, device="cuda")))
        _close(fw.unpack_dual(gd).tangent, 3 * ref, 3 * mag, logits.shape[1])


def _op(name, seed=3):
    """(fused function, plain function, inputs) of one part of a block."""
    from hccl_b200.models.llama import Attention, RMSNorm, _rope_tables
    from hccl_b200.ops import block
    g = torch.Generator(device="cuda").manual_seed(seed)
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)
    if name == "rms_norm":
        norm = RMSNorm(64, 1e-5, torch.bfloat16, "cuda")
        return lambda x, w: block.rms_norm(x, w, 1e-5, norm._plain), norm._plain, [draw(5, 64).requires_grad_(), draw(64).requires_grad_()]
    if name == "rope":
        att = Attention.__new__(Attention)
        torch.nn.Module.__init__(att)
        att.h_local, att.kv_local, att.hd = 4, 2, 16
        cos, sin = _rope_tables(3, 16, 10000.0, "cuda")
        plain = lambda t: att._rotated(t, 2, 3, cos, sin)
        return lambda t: block.rope_qkv(t, cos, sin, 2, 4, 2, 16, plain), plain, [draw(6, 128).requires_grad_()]
    plain = lambda t: torch.nn.functional.silu(t[:, :32]) * t[:, 32:]
    return lambda t: block.swiglu(t, plain), plain, [draw(5, 64).requires_grad_()]


def _outs(v):
    return list(v) if isinstance(v, tuple) else [v]


@pytest.mark.parametrize("name", ["rms_norm", "rope", "swiglu"])
def test_backward_takes_what_the_single_operations_took(name):
    """Batched and dual incoming gradients and a dispatch mode of the backward pass alone give what the plain operations give."""
    import torch.autograd.forward_ad as fw
    from torch.utils._python_dispatch import TorchDispatchMode

    fused, plain, ins = _op(name)
    g = torch.Generator(device="cuda").manual_seed(9)
    ups = [torch.randn(3, *o.shape, generator=g, device="cuda").to(torch.bfloat16) for o in _outs(plain(*ins))]
    got, ref = (torch.autograd.grad(_outs(f(*ins)), ins, ups, is_grads_batched=True) for f in (fused, plain))
    for a, b in zip(got, ref):
        assert torch.equal(a, b)

    def tangents(f):
        out = _outs(f(*ins))
        with fw.dual_level():
            d = torch.autograd.grad(out, ins, [fw.make_dual(u[0], u[1]) for u in ups])
            return [fw.unpack_dual(t).tangent for t in d]

    if name != "swiglu":                                 # silu's backward has no forward-mode rule, in the plain form either
        for a, b in zip(tangents(fused), tangents(plain)):
            assert a is not None and torch.equal(a, b)

    class Names(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    out = _outs(fused(*ins))
    with Names() as mode:
        torch.autograd.grad(out, ins, [u[0] for u in ups])
    assert any(s.startswith("aten.mul") for s in mode.seen)


@pytest.mark.parametrize("rows,hidden", [(5, 64), (3, 2048)])
def test_norm_input_and_weight_may_change_before_the_backward_pass(rows, hidden):
    """x += ..., a changed weight and a changed result after the norm: first and second derivatives are those of the values it saw."""
    from hccl_b200.models.llama import RMSNorm
    g = torch.Generator(device="cuda").manual_seed(hidden)
    norm = RMSNorm(hidden, 1e-5, torch.bfloat16, "cuda")
    leaf = torch.randn(rows, hidden, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    dy = torch.randn(rows, hidden, generator=g, device="cuda").to(torch.bfloat16)
    kept = norm.weight.detach().clone()

    def grads(change):
        with torch.no_grad():
            norm.weight.copy_(kept)
        x = leaf * 1
        y = norm(x)
        out = y * 1
        if change:
            with torch.no_grad():
                y.zero_()
                norm.weight.mul_(2)
            x += 1
        first = torch.autograd.grad(out, [x if not change else leaf, norm.weight], dy, create_graph=True)
        return first, torch.autograd.grad(first[0].float().square().sum() + first[1].float().square().sum(), [leaf, norm.weight])

    (a1, a2), (b1, b2) = grads(False), grads(True)
    for a, b in zip(a1 + a2, b1 + b2):
        assert torch.equal(a, b)
    plain = norm._plain(leaf, kept.requires_grad_())
    p1 = torch.autograd.grad(plain, [leaf, kept], dy, create_graph=True)
    p2 = torch.autograd.grad(p1[0].float().square().sum() + p1[1].float().square().sum(), [leaf, kept])
    for a, p in zip(a1 + a2, p1 + p2):                      # the same operations, rounded to bf16 in between at most three times more
        assert (a.double() - p.double()).norm() <= 3 * 2.0 ** -8 * p.double().norm()
    with torch.no_grad():
        assert torch.equal(norm(leaf), norm._plain(leaf, norm.weight)) or (norm(leaf).double() - norm._plain(leaf, norm.weight).double()).norm() < 2.0 ** -8 * plain.norm()


def test_targets_and_logits_may_change_before_the_backward_pass():
    """A token buffer refilled between two losses, logits scaled in place after the loss: the gradient is that of the values it saw."""
    from hccl_b200.models.llama import _VocabParallelCrossEntropy as X
    leaf, targets, ref, mag = _logits()
    logits = leaf * 1
    loss = X.apply(logits, targets, _OneRank, 0)
    logits.mul_(3)
    targets.zero_()
    g, = torch.autograd.grad(loss, leaf)
    _close(g, ref, mag, leaf.shape[1])


def test_rotary_embedding_keeps_nothing_of_the_projection():
    """The rotation is linear: the packed projection is neither kept for the backward pass nor missed when it has changed; the gradient of
    a gradient (by the incoming gradient) is the plain form's."""
    fused, plain, (leaf,) = _op("rope")
    kept = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.append(t.shape) or t, lambda t: t):
        qkv = leaf * 1
        out = fused(qkv)
    assert leaf.shape not in kept
    qkv.zero_()
    ups = [torch.randn(o.shape, device="cuda").to(torch.bfloat16).requires_grad_() for o in out]
    got, = torch.autograd.grad(out, leaf, ups, create_graph=True)
    ref, = torch.autograd.grad(plain(leaf), leaf, ups, create_graph=True)
    assert torch.equal(got, ref)
    c = torch.randn(leaf.shape, device="cuda").to(torch.bfloat16)
    for a, b in zip(torch.autograd.grad(got, ups, c), torch.autograd.grad(ref, ups, c)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name", ["rms_norm", "rope", "swiglu", "xent"])
def test_saved_tensors_that_come_back_changed(name):
    """Hooks that keep 32-bit tensors in 16 bits (and hand those back), or everything transposed: the backward kernels read nothing whose
    type or layout is not what the forward pass saved."""
    from hccl_b200.models.llama import _VocabParallelCrossEntropy as X
    if name == "xent":
        logits, targets, _, _ = _logits()
        f, ins = lambda t: X.apply(t, targets, _OneRank, 0), [logits]
    else:
        f, _, ins = _op(name)
    ref = torch.autograd.grad(_outs(f(*ins)), ins, [torch.ones_like(o) for o in _outs(f(*ins))])
    narrow = (lambda t: t.to(torch.bfloat16) if t.dtype == torch.float32 else t, lambda t: t)
    turned = (lambda t: t.t().contiguous() if t.dim() == 2 else t, lambda t: t.t() if t.dim() == 2 else t)
    for pack, unpack in (narrow, turned):
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            out = _outs(f(*ins))
        for a, b in zip(torch.autograd.grad(out, ins, [torch.ones_like(o) for o in out]), ref):
            assert (a.double() - b.double()).norm() <= 2.0 ** -5 * b.double().norm()


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("name", ["rms_norm", "rope", "swiglu", "xent", "column", "row"])
def test_saved_tensors_of_another_size(name, native, monkeypatch):
    """A hook hands one saved tensor back wider, longer or shorter than it was: the backward pass gives the gradient of what it still knows, or an
    error, and no kernel reads or writes by the sizes of the forward pass."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.models.llama import _cross_entropy
    from hccl_b200.ops import block
    from hccl_b200.parallel import tensor_parallel as tp
    comm = None
    if native:
        _native_nodes()
    else:
        monkeypatch.setattr(block, "_NODES", None)
    try:
        if name == "xent":
            logits, targets, _, _ = _logits()
            f, ins = lambda t: _cross_entropy(t, targets, _OneRank, 0), [logits]
        elif name in ("column", "row"):
            torch.zeros(1, device="cuda")
            comm = Communicator.from_root_info(1, get_root_info(), 0)
            ins = [torch.randn(*s, device="cuda").to(torch.bfloat16).requires_grad_() for s in ((128, 64), (128, 64))]
            cls = tp._ColumnSeqParallel if name == "column" else tp._RowSeqParallel

            def f(x, w):
                y = tp._one_rank_linear(x, w, comm, name == "column")
                assert (y is not None) == native
                return cls.apply(x, w, comm) if y is None else y
        else:
            f, _, ins = _op(name)
        ups = [torch.ones_like(o) for o in _outs(f(*ins))]
        ref = torch.autograd.grad(_outs(f(*ins)), ins, ups)
        saved = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append(t.shape) or t, lambda t: t):
            f(*ins)
        changes = (lambda t: torch.cat([t, t], -1), lambda t: torch.cat([t, t]), lambda t: t[..., :-8].contiguous() if t.shape[-1] > 8 else t[..., :2].contiguous(),
                   lambda t: t[:-1].clone())
        for at in range(len(saved)):
            for change in changes:
                count = [0]

                def pack(t):
                    count[0] += 1
                    return count[0] - 1, t

                with torch.autograd.graph.saved_tensors_hooks(pack, lambda p: change(p[1]) if p[0] == at else p[1]):
                    out = _outs(f(*ins))
                try:
                    got = torch.autograd.grad(out, ins, ups)
                except (RuntimeError, IndexError, ValueError, AssertionError):
                    continue
                for a, b in zip(got, ref):
                    assert a.shape == b.shape and (a.double() - b.double()).norm() <= 2.0 ** -5 * b.double().norm()
        torch.cuda.synchronize()
    finally:
        if comm is not None:
            comm.destroy()


@pytest.mark.parametrize("rows,hidden", [(5, 8), (700, 256), (70, 1000)])
def test_norm_workspace_aligned_to_its_elements(rows, hidden):
    """Up to 1024 columns the backward pass takes a workspace at any multiple of four bytes: the same bits as on whole vectors."""
    from hccl_b200.ops import block
    l = block._decl()
    x, dy, w = [torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((rows, hidden), (rows, hidden), (hidden,))]
    rstd = torch.rsqrt(x.float().square().mean(1) + 1e-5)
    parts = l.HcclRmsNormBwdParts(rows, hidden)

    def run(offset):
        dx, dw, partial = torch.empty_like(x), torch.empty_like(w), torch.empty(parts * hidden + 4, device="cuda")
        assert l.HcclRmsNormBwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr(), dx.data_ptr(), dw.data_ptr(), partial.data_ptr() + offset, rows, hidden,
                                torch.cuda.current_stream().cuda_stream) == 0
        return dx, dw

    for offset in (4, 8, 12):
        assert all(torch.equal(a, b) for a, b in zip(run(0), run(offset)))


@pytest.mark.parametrize("name", ["rms_norm", "rope", "swiglu", "xent", "column", "row"])
def test_compiled_autograd_traces_a_node_once(name):
    """The same step several times under compiled autograd, on new values: the gradients of the single operations and one trace in all. Another first class
    of a vocabulary shard is another trace; the norm's epsilon and the rotary tables are inputs of it."""
    from torch._dynamo import compiled_autograd
    from torch._dynamo.utils import counters
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.models.llama import RMSNorm, _rope_tables, _rotated
    from hccl_b200.ops import block
    from hccl_b200.parallel import tensor_parallel as tp
    nodes = _native_nodes()
    torch.zeros(1, device="cuda")
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    draw = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16).requires_grad_()
    try:
        def case(step):
            """fused outputs, inputs, plain outputs (or gradients) of one step; step 3 has another constant"""
            if name == "rms_norm":
                norm, ins = RMSNorm(64, 1e-5 if step < 3 else 0.5, torch.bfloat16, "cuda"), [draw(5, 64), draw(64)]
                return block.rms_norm(*ins, norm.eps, norm._plain), ins, norm._plain
            if name == "rope":
                cos, sin = _rope_tables(3, 16, 10000.0 + 5000 * step, "cuda")
                plain = lambda t: _rotated(t, 2, 3, 4, 2, 16, cos, sin)
                ins = [draw(6, 128)]
                return block.rope_qkv(*ins, cos, sin, 2, 4, 2, 16, plain), ins, plain
            if name == "swiglu":
                plain, ins = lambda t: torch.nn.functional.silu(t[:, :32]) * t[:, 32:], [draw(5, 64)]
                return block.swiglu(*ins, plain), ins, plain
            if name == "xent":
                ins, targets, start = [draw(6, 24)], torch.randint(0, 24, (6,), device="cuda"), 0 if step < 3 else 4

                def plain(t):
                    lse, mine, idx = t.float().logsumexp(-1), (targets >= start) & (targets < start + 24), (targets - start).clamp(0, 23)
                    return (lse - torch.where(mine, t.float().gather(1, idx[:, None])[:, 0], torch.zeros_like(lse))).mean()

                return nodes.xent(*ins, targets, start), ins, plain
            ins = [draw(128, 64), draw(192, 64)]
            return tp._one_rank_linear(*ins, comm, name == "column"), ins, lambda x, w: x @ w.t()

        def run(step):
            out, ins, plain = case(step)
            ups = [torch.randn_like(o) for o in _outs(out)]
            before = counters["compiled_autograd"]["captures"]
            with compiled_autograd._enable(torch.compile(backend="eager")):
                torch.autograd.backward(_outs(out), ups)
            ref = torch.autograd.grad(_outs(plain(*ins)), ins, ups)
            for t, r in zip(ins, ref):
                assert (t.grad.double() - r.double()).norm() <= 2.0 ** -7 * r.double().norm()
            return counters["compiled_autograd"]["captures"] - before

        counts = [run(step) for step in range(4)]
        assert counts[0] == 1 and counts[1] == 0 and counts[2] == 0, counts
        assert counts[3] == (1 if name == "xent" else 0), counts
    finally:
        comm.destroy()


def _tiny(seed=3):
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.models.llama import Llama, LlamaConfig
    torch.zeros(1, device="cuda")
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    return comm, Llama(LlamaConfig.tiny(), comm, dtype=torch.bfloat16, device="cuda", seed=seed)


@pytest.mark.parametrize("tokens", [(2, 128), (1, 100)])
def test_native_nodes_give_the_bits_of_the_python_functions(tokens, monkeypatch):
    """A whole decoder through both: loss and gradients, on rows that the fused linear takes and on rows that it does not; saved tensors on the
    CPU, a recomputed block, a graph run twice."""
    from torch.utils.checkpoint import checkpoint
    from hccl_b200.models.llama import _rope_tables
    from hccl_b200.ops import block
    _native_nodes()
    comm, model = _tiny()
    try:
        t = torch.randint(0, 512, (tokens[0], tokens[1] + 1), device="cuda")
        params = list(model.parameters())

        def step():
            loss = model(t[:, :-1].contiguous(), t[:, 1:].contiguous())
            assert _is_native(loss) == (block.nodes() is not None)
            first = torch.autograd.grad(loss, params, retain_graph=True)
            return [loss.detach(), *first, *torch.autograd.grad(loss, params)]

        native = step()
        with torch.autograd.graph.save_on_cpu():
            loss = model(t[:, :-1].contiguous(), t[:, 1:].contiguous())
        offloaded = torch.autograd.grad(loss, params)
        x = torch.randn(tokens[0] * tokens[1], 256, device="cuda").to(torch.bfloat16).requires_grad_()
        rope = _rope_tables(tokens[1], 32, 500000.0, "cuda")
        args = (x, *tokens, *rope)
        plain, = torch.autograd.grad(model.blocks[0](*args).sum(), x)
        again, = torch.autograd.grad(checkpoint(model.blocks[0], *args, use_reentrant=False).sum(), x)
        assert torch.equal(plain, again)
        monkeypatch.setattr(block, "_NODES", None)
        for a, b in zip(native, step()):
            assert torch.equal(a, b)
        for a, b in zip(native[1:], offloaded):
            assert torch.equal(a, b)
    finally:
        comm.destroy()


def test_native_nodes_keep_the_engine_s_rules():
    """A graph that was freed and a weight that changed in place are refused; an error of the Python form keeps its type; a module that holds its
    own output is collected."""
    import gc
    import weakref
    from hccl_b200.models.llama import RMSNorm, _rope_tables
    from hccl_b200.ops import block
    _native_nodes()
    comm, model = _tiny()
    try:
        x = torch.randn(256, 256, device="cuda").to(torch.bfloat16).requires_grad_()
        run = lambda: model.blocks[0](x, 2, 128, *_rope_tables(128, 32, 500000.0, "cuda")).sum()
        out = run()
        out.backward()
        with pytest.raises(RuntimeError, match="second time"):
            out.backward()
        out = run()
        with torch.no_grad():
            model.blocks[0].mlp.down.weight.mul_(1)
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            out.backward()

        def failing(x, w):
            raise LookupError("plain form")

        w = torch.ones(256, device="cuda", dtype=torch.bfloat16).requires_grad_()
        y = block.rms_norm(x, w, 1e-5, failing)
        assert _is_native(y)
        with pytest.raises(LookupError, match="plain form"):
            torch.autograd.grad(y.sum(), x, create_graph=True)
        norm = RMSNorm(256, 1e-5, torch.bfloat16, "cuda")
        norm.kept = norm(x)
        gone = weakref.ref(norm)
        del norm
        gc.collect()
        assert gone() is None
    finally:
        comm.destroy()


def _plain_modules(monkeypatch):
    """The decoder's norms one operation after the other: what the fused ones have to give, bit for bit."""
    from hccl_b200.models import llama
    monkeypatch.setattr(llama, "_normed", lambda norm, x, d=None: ((lambda s: (norm(s), s, False))(x if d is None else x + d)))


@pytest.mark.parametrize("rows,hidden", [(1, 8), (9, 264), (300, 1024), (7, 1032), (600, 4096), (5, 4104), (3, 12288)])
def test_norm_of_a_sum(rows, hidden):
    """The sum, its norm and the gradients of both, in every width of the kernels: the bits of the addition and the norm one after the other."""
    from torch._dynamo import compiled_autograd
    from hccl_b200.models.llama import RMSNorm, _normed
    _native_nodes()
    torch._dynamo.reset()                                    # a trace for one row is not one for several
    compiled_autograd.reset()
    g = torch.Generator(device="cuda").manual_seed(hidden)
    norm = RMSNorm(hidden, 1e-5, torch.bfloat16, "cuda")
    with torch.no_grad():
        norm.weight.copy_(torch.randn(hidden, generator=g, device="cuda"))
    x, d = [torch.randn(rows, hidden, generator=g, device="cuda").to(torch.bfloat16).requires_grad_() for _ in range(2)]
    ups = [torch.randn(rows, hidden, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2)]
    for add in (None, d):
        ins = [x, norm.weight] if add is None else [x, d, norm.weight]
        y, s, own = _normed(norm, x, add)
        assert own and _is_native(y)
        ref_s = x * 1 if add is None else x + d
        ref_y = norm(ref_s)
        assert torch.equal(y, ref_y) and torch.equal(s, ref_s)
        for outs, refs, grads in (((y, s), (ref_y, ref_s), ups), ((y,), (ref_y,), ups[:1]), ((s,), (ref_s,), ups[1:])):
            got = torch.autograd.grad(outs, ins, grads, retain_graph=True, allow_unused=True)
            ref = torch.autograd.grad(refs, ins, grads, retain_graph=True, allow_unused=True)
            for a, b in zip(got, ref):
                assert (a is None) == (b is None) and (a is None or torch.equal(a, b))
        first = torch.autograd.grad((y, s), ins, ups, create_graph=True)
        ref1 = torch.autograd.grad((ref_y, ref_s), ins, ups, create_graph=True)
        for a, b in zip(torch.autograd.grad(sum(t.float().square().sum() for t in first), ins), torch.autograd.grad(sum(t.float().square().sum() for t in ref1), ins)):
            assert (a.double() - b.double()).norm() <= 2.0 ** -6 * b.double().norm()
        with compiled_autograd._enable(torch.compile(backend="eager")):        # the traced form keeps 32 bits where the kernel rounds
            torch.autograd.backward(_normed(norm, x, add)[:2], ups)
        ref_s = x * 1 if add is None else x + d
        ref_y = norm(ref_s)
        for t, b in zip(ins, torch.autograd.grad((ref_y, ref_s), ins, ups)):
            assert (t.grad.double() - b.double()).norm() <= 2.0 ** -6 * b.double().norm()
            t.grad = None
        with torch.no_grad():
            y, s, _ = _normed(norm, x, add)
            assert torch.equal(y, ref_y) and torch.equal(s, ref_s)


@pytest.mark.parametrize("tokens", [(2, 128), (3, 37), (1, 1)])
def test_block_with_fused_norms_gives_the_bits_of_the_modules(tokens, monkeypatch):
    """Loss and gradients of a decoder with and without the fused residual additions; saved tensors on the CPU, hooks on the modules (which are all seen)."""
    _native_nodes()
    comm, model = _tiny()
    try:
        t = torch.randint(0, 512, (tokens[0], tokens[1] + 1), device="cuda")
        params = list(model.parameters())

        def step():
            loss = model(t[:, :-1].contiguous(), t[:, 1:].contiguous())
            return [loss.detach(), *torch.autograd.grad(loss, params)]

        fused = step()
        with torch.autograd.graph.save_on_cpu():
            loss = model(t[:, :-1].contiguous(), t[:, 1:].contiguous())
        for a, b in zip(torch.autograd.grad(loss, params), fused[1:]):
            assert torch.equal(a, b)
        seen = []
        hook = lambda m: m.register_forward_hook(lambda m, i, o: seen.append(m))
        projections = [b.attn.qkv for b in model.blocks]
        handles = [hook(m) for m in model.modules() if m is not model and not any(m is p for p in projections)]
        hooked = step()
        handles += [hook(m) for m in projections]                              # then the library's backward pass of the attention: sums in another order
        seen.clear()
        for a, b in zip(step(), fused):
            assert (a.double() - b.double()).norm() <= 2.0 ** -5 * b.double().norm() + 1e-12
        [h.remove() for h in handles]
        assert len(seen) == len(list(model.modules())) - 2                      # but for the model and its list of blocks
        _plain_modules(monkeypatch)
        plain = step()
        for a, b, c in zip(fused, hooked, plain):
            assert torch.equal(a, c) and torch.equal(b, c)
    finally:
        comm.destroy()


def test_block_input_may_change_after_the_pass():
    """The block's input, which its caller may write afterwards, is not what the backward pass reads."""
    from hccl_b200.models.llama import _rope_tables
    comm, model = _tiny()
    try:
        leaf = torch.randn(256, 256, device="cuda").to(torch.bfloat16).requires_grad_()
        up = torch.randn(256, 256, device="cuda").to(torch.bfloat16)

        def grads(change):
            x = leaf * 1
            out = model.blocks[0](x, 2, 128, *_rope_tables(128, 32, 500000.0, "cuda"))
            if change:
                x.zero_()
            return torch.autograd.grad(out, [leaf, *model.blocks[0].parameters()], up)

        for a, b in zip(grads(False), grads(True)):
            assert torch.equal(a, b)
    finally:
        comm.destroy()


def _swiglu_layer(rows, hidden, ffn, seed=1):
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.parallel.tensor_parallel import TensorParallelMLP
    torch.zeros(1, device="cuda")
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    torch.manual_seed(seed)
    mlp = TensorParallelMLP(comm, hidden, ffn, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed)
    x, up = [torch.randn(rows, hidden, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2)]
    return comm, mlp, x.requires_grad_(), up


@pytest.mark.parametrize("rows,hidden,ffn", [(1, 64, 64), (70, 136, 72), (130, 512, 1000), (300, 256, 2056), (513, 520, 1000), (768, 1024, 512), (1030, 264, 3000), (5000, 256, 1536)])
def test_swiglu_layer_gives_the_bits_of_its_parts(rows, hidden, ffn):
    """The products with SwiGLU in their epilogues: every tile width, rows and columns that do not fill a tile, both sides of the choices; result and gradients are those
    of the product and the element-wise kernel one after the other (gate values of all sizes, one of them infinite)."""
    _native_nodes()
    comm, mlp, x, up = _swiglu_layer(rows, hidden, ffn)
    try:
        with torch.no_grad():
            mlp.gate_up.weight.mul_(torch.exp(torch.randn(2 * ffn, 1, device="cuda")).to(torch.bfloat16) * 30)
            mlp.gate_up.weight[0, 0] = float("inf")
        params = list(mlp.parameters())

        def step():
            y = mlp(x)
            return [y.detach(), *torch.autograd.grad(y, [x, *params], up)]

        fused = step()
        assert mlp(x).grad_fn.name() == "_SwiGluMlpBackward"
        handle = mlp.gate_up.register_forward_hook(lambda *a: None)
        parts = step()
        handle.remove()
        for a, b in zip(fused, parts):
            assert torch.equal(a.nan_to_num(3.0, 5.0, 7.0), b.nan_to_num(3.0, 5.0, 7.0))
        with torch.no_grad():
            assert torch.equal(mlp(x).nan_to_num(3.0, 5.0, 7.0), parts[0].nan_to_num(3.0, 5.0, 7.0))
    finally:
        comm.destroy()


@pytest.mark.parametrize("rows,hidden,ffn", [(20, 2016, 64), (40, 1024, 504), (200, 8192, 3584), (300, 16384, 256), (512, 4096, 512), (520, 16384, 512), (700, 4096, 512), (1344, 4184, 1408)])
def test_swiglu_layer_gives_the_bits_of_its_parts_where_they_split_k(rows, hidden, ffn):
    """Long K and few columns on both sides of 512 rows: the products split K, forward or backward or both, which the fused kernels cannot."""
    test_swiglu_layer_gives_the_bits_of_its_parts(rows, hidden, ffn)


def test_swiglu_layer_keeps_the_engine_s_rules():
    """Input that changes after the pass, a gradient's gradient, compiled autograd, batched gradients, saved tensors of another size or on the CPU, a weight that changes in
    place, the switch of the weight gradients."""
    from torch._dynamo import compiled_autograd
    from hccl_b200.parallel import tensor_parallel as tp
    _native_nodes()
    comm, mlp, leaf, up = _swiglu_layer(640, 64, 128)
    try:
        ins = [leaf, *mlp.parameters()]
        ref = torch.autograd.grad(mlp(leaf), ins, up)
        x = leaf * 1
        y = mlp(x)
        x.zero_()
        for a, b in zip(torch.autograd.grad(y, ins, up), ref):
            assert torch.equal(a, b)
        plain = tp._plain_mlp(leaf, mlp.gate_up.weight, mlp.down.weight)
        close = lambda a, b, steps: (a.double() - b.double()).norm() <= steps * 2.0 ** -8 * b.double().norm()
        pg = torch.autograd.grad(plain, ins, up, create_graph=True)
        y = mlp(leaf * 1)
        got = torch.autograd.grad(y, ins, up, create_graph=True)
        assert all(close(a, b, 8) for a, b in zip(got, pg))                     # a dozen roundings to bf16 on the way
        second = torch.autograd.grad(sum(t.float().square().sum() for t in got), ins[1:])
        for a, b in zip(second, torch.autograd.grad(sum(t.float().square().sum() for t in pg), ins[1:])):
            assert close(a, b, 16)
        ups = torch.stack([up, up * 2])
        batched = torch.autograd.grad(mlp(leaf), ins, ups, is_grads_batched=True)
        assert all(close(t[0], b, 8) and close(t[1], 2 * b, 8) for t, b in zip(batched, ref))
        with compiled_autograd._enable(torch.compile(backend="eager")):
            mlp(leaf).backward(up)
        for t, b in zip(ins, ref):
            assert close(t.grad, b, 8)
            t.grad = None
        with torch.autograd.graph.save_on_cpu():
            y = mlp(leaf)
        assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y, ins, up), ref))
        for at in range(5):
            for change in (lambda t: torch.cat([t, t], -1), lambda t: t[:-1].clone(), lambda t: t[:, :-8].contiguous()):
                count = [0]

                def pack(t):
                    count[0] += 1
                    return count[0] - 1, t

                with torch.autograd.graph.saved_tensors_hooks(pack, lambda p: change(p[1]) if p[0] == at else p[1]):
                    y = mlp(leaf)
                assert count[0] == 5
                with pytest.raises((RuntimeError, IndexError, ValueError, AssertionError)):
                    torch.autograd.grad(y, ins, up)
        tp.use_native_wgrad(True)
        assert all(close(a, b, 8) for a, b in zip(torch.autograd.grad(mlp(leaf), ins, up), ref))
        tp.use_native_wgrad(False)
        y = mlp(leaf)
        with torch.no_grad():
            mlp.down.weight.mul_(1)
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            y.sum().backward()
        torch.cuda.synchronize()
    finally:
        tp.use_native_wgrad(False)
        comm.destroy()


@pytest.mark.parametrize("given", ["leaf", "tensor", "away"])
def test_swiglu_layer_second_derivatives_reach_the_input(given):
    """The gradient of every first gradient by every input of the layer: a leaf, a tensor with a history, and one that the caller gives away (kept without a copy). Bounds as above: 16 roundings to bf16
    on the way of both sides."""
    from hccl_b200.parallel import tensor_parallel as tp
    _native_nodes()
    comm, mlp, leaf, up = _swiglu_layer(640, 64, 128)
    try:
        ins = [leaf, *mlp.parameters()]
        layer = {"leaf": lambda: mlp(leaf), "tensor": lambda: mlp(leaf * 1), "away": lambda: tp.mlp_of_own(mlp, leaf * 1)}[given]
        got, plain = (torch.autograd.grad(f(), ins, up, create_graph=True) for f in (layer, lambda: tp._plain_mlp(*ins)))
        square = lambda t: t.float().square().sum()
        for i, (a, b) in enumerate(zip(got, plain)):
            seconds = [torch.autograd.grad(square(t), ins, retain_graph=True, allow_unused=True) for t in (a, b)]
            for c, d in zip(*seconds):
                assert (c is None) == (d is None), i
                assert c is None or (c.double() - d.double()).norm() <= 16 * 2.0 ** -8 * d.double().norm(), i
        square(got[2]).backward()
        assert leaf.grad is not None and (leaf.grad.double() - seconds[1][0].double()).norm() <= 16 * 2.0 ** -8 * seconds[1][0].double().norm()
    finally:
        comm.destroy()


@pytest.mark.parametrize("given", ["leaf", "tensor", "away"])
@pytest.mark.parametrize("column", [True, False])
def test_linear_layer_second_derivatives(column, given):
    """The gradient of every first gradient of a one-rank linear layer by its input and weight, as of the SwiGLU layer: a product each way, four roundings to bf16 on both sides."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.parallel import tensor_parallel as tp
    _native_nodes()
    torch.zeros(1, device="cuda")
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        g = torch.Generator(device="cuda").manual_seed(3)
        ins = [torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16).requires_grad_() for s in ((130, 64), (192, 64))]
        up = torch.randn(130, 192, generator=g, device="cuda").to(torch.bfloat16)
        x = ins[0] if given == "leaf" else ins[0] * 1
        y = tp._one_rank_linear(x, ins[1], comm, column, given == "away")
        got, plain = (torch.autograd.grad(t, ins, up, create_graph=True) for t in (y, ins[0] @ ins[1].t()))
        for i, pair in enumerate(zip(got, plain)):
            seconds = [torch.autograd.grad(t.float().square().sum(), ins, retain_graph=True, allow_unused=True) for t in pair]
            for c, d in zip(*seconds):
                assert (c is None) == (d is None), i
                assert c is None or (c.double() - d.double()).norm() <= 4 * 2.0 ** -8 * d.double().norm(), i
    finally:
        comm.destroy()


def _attention_case(batch, seq, heads, kv_heads, hd, seed=2):
    import functools
    from hccl_b200.models.llama import _plain_attention, _rope_tables
    from hccl_b200.ops import block
    g = torch.Generator(device="cuda").manual_seed(seed)
    qkv, do = [torch.randn(batch * seq, n * hd, generator=g, device="cuda").to(torch.bfloat16) for n in (heads + 2 * kv_heads, heads)]
    cos, sin = _rope_tables(seq, hd, 10000.0, "cuda")
    plain = functools.partial(_plain_attention, batch=batch, seq=seq, heads=heads, kv_heads=kv_heads, hd=hd, cos=cos, sin=sin)
    return lambda t: block.attention(t, cos, sin, batch, heads, kv_heads, hd, plain), plain, qkv.requires_grad_(), do, cos.double(), sin.double()


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("batch,seq,heads,kv_heads,hd", [(1, 2, 8, 4, 32), (3, 63, 2, 1, 32), (2, 64, 4, 4, 32), (1, 65, 8, 2, 32), (2, 200, 6, 3, 32), (1, 1024, 4, 4, 32), (1, 130, 4, 2, 64),
                                                         (2, 128, 8, 2, 64)])
def test_attention_of_short_sequences(batch, seq, heads, kv_heads, hd, native, monkeypatch):
    """The backward kernel: sequences around whole tiles, grouped queries, both widths, against 64 bits from the rotated values as the kernels round them. What the products read is rounded
    to bf16 once: probabilities, their gradients and O in the sum of dO * O, at most 2^-8 of the magnitudes that are added up, and each result once more. The same bits on every run."""
    from hccl_b200.models.llama import _rotated
    from hccl_b200.ops import block
    if native:
        _native_nodes()
    else:
        monkeypatch.setattr(block, "_NODES", None)
    f, _, qkv, do, cos, sin = _attention_case(batch, seq, heads, kv_heads, hd)
    o = f(qkv)
    assert o.grad_fn.name().startswith("_Attention") and _is_native(o) == native
    got, = torch.autograd.grad(o, qkv, do, retain_graph=True)
    assert torch.equal(got, torch.autograd.grad(o, qkv, do)[0])
    group, scale = heads // kv_heads, hd ** -0.5
    q, k, v = (t.double().transpose(1, 2) for t in _rotated(qkv.detach(), batch, seq, heads, kv_heads, hd, cos.float(), sin.float()))
    k, v = k.repeat_interleave(group, 1), v.repeat_interleave(group, 1)
    d = do.double().reshape(batch, seq, heads, hd).transpose(1, 2)
    p = (q @ k.transpose(2, 3) * scale).masked_fill(~torch.ones(seq, seq, dtype=torch.bool, device="cuda").tril(), float("-inf")).softmax(-1)
    ref = p @ v
    flat = lambda t: t.transpose(1, 2).reshape(batch * seq, -1)
    assert bool(((o.double() - flat(ref)).abs() <= flat(p @ v.abs()) * 2.0 ** -8 + flat(ref).abs() * 2.0 ** -8).all())
    dp, dot = d @ v.transpose(2, 3), (d * ref).sum(-1, keepdim=True)
    ds, mag = p * (dp - dot) * scale, p * (dp.abs() + (d.abs() * ref.abs()).sum(-1, keepdim=True)) * scale
    grouped = lambda t: t.reshape(batch, kv_heads, group, seq, hd).sum(2)
    c, s = cos[None, None], sin[None, None]

    def back(t):
        a, b = t[..., :hd // 2], t[..., hd // 2:]
        return torch.cat([a * c + b * s, b * c - a * s], -1)

    def both(t):                                                               # a rotation adds parts of both halves
        return torch.cat([t[..., :hd // 2] + t[..., hd // 2:]] * 2, -1)

    refs = back(ds @ k), back(grouped(ds.transpose(2, 3) @ q)), grouped(p.transpose(2, 3) @ d)
    mags = both(mag @ k.abs()), both(grouped(mag.transpose(2, 3) @ q.abs())), grouped(p.transpose(2, 3) @ d.abs())
    want, bound = torch.cat([flat(t) for t in refs], 1), torch.cat([flat(t) for t in mags], 1)
    assert bool(((got.double() - want).abs() <= bound * 2.0 ** -7 + want.abs() * 2.0 ** -8 + 1e-6).all())


def test_attention_keeps_the_engine_s_rules():
    """Another attention asked for, a projection that changes in place, saved tensors of another size, batched gradients, compiled autograd: the plain form's answers or errors."""
    from torch._dynamo import compiled_autograd
    from torch.nn.attention import SDPBackend, sdpa_kernel
    from hccl_b200.ops import block
    nodes = _native_nodes()
    f, plain, qkv, do, _, _ = _attention_case(2, 100, 4, 2, 32)
    close = lambda a, b: (a.double() - b.double()).norm() <= 2.0 ** -6 * b.double().norm()
    ref, = torch.autograd.grad(plain(qkv), qkv, do)
    assert close(torch.autograd.grad(f(qkv), qkv, do)[0], ref)
    with sdpa_kernel(SDPBackend.MATH):
        assert f(qkv) is None
    with torch.autocast("cuda", dtype=torch.float16):
        assert f(qkv) is None
    batched, = torch.autograd.grad(f(qkv), qkv, torch.stack([do, 2 * do]), is_grads_batched=True)
    assert close(batched[0], ref) and close(batched[1], 2 * ref)
    x = qkv * 1
    o = f(x)
    x.zero_()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(o, qkv, do)
    for at in range(5):
        for change in (lambda t: torch.cat([t, t], -1), lambda t: t[:-1].clone(), lambda t: t[..., :-8].contiguous()):
            count = [0]

            def pack(t):
                count[0] += 1
                return count[0] - 1, t

            with torch.autograd.graph.saved_tensors_hooks(pack, lambda p: change(p[1]) if p[0] == at else p[1]):
                o = f(qkv)
            assert count[0] == 5
            try:
                got, = torch.autograd.grad(o, qkv, do)
            except (RuntimeError, IndexError, ValueError, AssertionError):
                continue
            assert got.shape == ref.shape and close(got, ref)                  # what the plain form does not read may have changed
    with compiled_autograd._enable(torch.compile(backend="eager")):
        f(qkv).backward(do)
    assert close(qkv.grad, ref)
    with torch.no_grad():
        assert f(qkv) is None and nodes is block.nodes()


def test_function_modes_and_a_replaced_attention_see_the_model(monkeypatch):
    """A function mode around the model and another function in the place of the library's attention meet the operations that the model is written with: attention, residual additions, the
    embedding's index. A default device is a mode as well and changes nothing."""
    import torch.nn.functional as F
    from torch.overrides import TorchFunctionMode
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.models.llama import Llama, LlamaConfig
    from hccl_b200.ops import block
    _native_nodes()
    torch.zeros(1, device="cuda")
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        cfg = LlamaConfig.tiny(vocab=512, hidden=256, layers=2, heads=8, kv_heads=4, ffn=512)
        model = Llama(cfg, comm, dtype=torch.bfloat16, device="cuda", seed=3)
        tokens = torch.randint(0, 512, (2, 64), device="cuda")
        seen, calls = [], []

        class See(TorchFunctionMode):
            def __torch_function__(self, func, types, args=(), kwargs=None):
                seen.append(getattr(func, "__name__", ""))
                return func(*args, **(kwargs or {}))

        close = lambda a, b: (a.double() - b.double()).norm() <= 2.0 ** -6 * b.double().norm()
        ref = model(tokens)
        with See():
            assert close(model(tokens), ref)
        assert seen.count("scaled_dot_product_attention") == 2 and "__getitem__" in seen
        assert sum(name in ("add", "__add__") for name in seen) >= 4
        library = F.scaled_dot_product_attention
        monkeypatch.setattr(F, "scaled_dot_product_attention", lambda *a, **k: (calls.append(1), library(*a, **k))[1])
        assert close(model(tokens), ref) and len(calls) == 2
        monkeypatch.undo()
        f, _, qkv, *_ = _attention_case(2, 100, 4, 2, 32)
        with torch.device("cuda"):
            assert f(qkv).grad_fn.name() == "_AttentionBackward"
            assert block.embedding(model.embed, tokens.reshape(-1)).grad_fn.name() == "_EmbeddingBackward"
    finally:
        comm.destroy()


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("tokens,hidden,vocab", [(1, 8, 1), (33, 264, 7), (255, 2056, 300), (257, 256, 512), (2048, 64, 50), (2049, 64, 50)])
def test_embedding_gradient_of_few_tokens(tokens, hidden, vocab, native, monkeypatch):
    """Ids that repeat, ids from the end, both sides of the most tokens that the kernel takes: sums in 32 bits, rounded once (the general form rounds every addition). The gradient of
    the gradient, batched gradients and a changed id buffer are those of the plain index."""
    from torch._dynamo import compiled_autograd
    from hccl_b200.ops import block
    if native:
        _native_nodes()
    else:
        monkeypatch.setattr(block, "_NODES", None)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    w = torch.randn(vocab, hidden, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    ids = torch.randint(-vocab, vocab, (tokens,), generator=g, device="cuda")
    dy = torch.randn(tokens, hidden, generator=g, device="cuda").to(torch.bfloat16)
    y = block.embedding(w, ids)
    if tokens > 2048:
        assert y is None
        return
    assert torch.equal(y, w[ids]) and y.grad_fn.name().startswith("_Embedding") and _is_native(y) == native
    got, = torch.autograd.grad(y, w, dy, retain_graph=True)
    ref, mag = (torch.zeros(vocab, hidden, dtype=torch.float64, device="cuda").index_put((ids,), t, accumulate=True) for t in (dy.double(), dy.double().abs()))
    _close(got, ref, mag, tokens)
    rows = torch.bincount(ids % vocab, minlength=vocab).max().item()
    close = lambda a, b: ((a.double() - b.double()).abs() <= (mag * rows + b.double().abs()) * 2.0 ** -8 + 1e-30).all()      # the plain form rounds as often as an id occurs
    b1, = torch.autograd.grad(y, w, torch.stack([dy, -dy]), is_grads_batched=True, retain_graph=True)
    assert bool(close(b1[0], ref)) and bool(close(b1[1], -ref))
    up = dy.clone().requires_grad_()
    first, = torch.autograd.grad(y, w, up, create_graph=True, retain_graph=True)
    second, = torch.autograd.grad(first, up, torch.ones_like(first))
    assert torch.equal(second, torch.ones_like(dy))
    if native:
        with compiled_autograd._enable(torch.compile(backend="eager")):
            block.embedding(w, ids).backward(dy)
        assert bool(close(w.grad, ref))
        w.grad = None
    ids.zero_()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(y, w, dy)


@pytest.mark.parametrize("tokens,hidden,vocab,common", [(2, 8, 3, 2), (300, 264, 40, 280), (2048, 256, 512, 2048), (2048, 4096, 1000, 1500)])
def test_embedding_gradient_of_a_common_id(tokens, hidden, vocab, common):
    """A batch that is mostly one padding id, at its end: one block adds up its rows, in 32 bits and rounded once; rows of other ids and ids without a token as before."""
    from hccl_b200.ops import block
    _native_nodes()
    g = torch.Generator(device="cuda").manual_seed(tokens + common)
    w = torch.randn(vocab, hidden, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    ids = torch.randint(0, vocab, (tokens,), generator=g, device="cuda")
    ids[tokens - common:] = vocab - 1
    dy = torch.randn(tokens, hidden, generator=g, device="cuda").to(torch.bfloat16)
    got, = torch.autograd.grad(block.embedding(w, ids), w, dy)
    ref, mag = (torch.zeros(vocab, hidden, dtype=torch.float64, device="cuda").index_put((ids,), t, accumulate=True) for t in (dy.double(), dy.double().abs()))
    _close(got, ref, mag, tokens)
    assert not got[torch.bincount(ids, minlength=vocab) == 0].any()


@pytest.mark.parametrize("rows,vocab", [(1, 1), (6, 24), (300, 1000), (1025, 515), (64, 128256)])
def test_cross_entropy_of_one_rank(rows, vocab):
    """The loss against 64 bits, by the native node and the Python function alike: 32-bit sums over a row and over the rows."""
    from hccl_b200.models.llama import _VocabParallelCrossEntropy as X, _cross_entropy
    _native_nodes()
    g = torch.Generator(device="cuda").manual_seed(rows)
    logits = (torch.randn(rows, vocab, generator=g, device="cuda") * 3).to(torch.bfloat16).requires_grad_()
    targets = torch.randint(0, vocab, (rows,), generator=g, device="cuda")
    ref = torch.nn.functional.cross_entropy(logits.double(), targets)
    for loss in (_cross_entropy(logits, targets, _OneRank, 0), X.apply(logits, targets, _OneRank, 0)):
        assert abs(loss.item() - ref.item()) <= 16 * 2.0 ** -23 * (logits.abs().max().item() + ref.item() + 12)
        got, = torch.autograd.grad(loss, logits)
        p = torch.softmax(logits.detach().double(), 1)
        hot = torch.nn.functional.one_hot(targets, vocab).double()
        _close(got, (p - hot) / rows, (p + hot) / rows, 64)
    with torch.no_grad():
        assert torch.equal(_cross_entropy(logits, targets, _OneRank, 0), loss.detach())
        bad = logits.detach().clone()
        bad[rows // 2, vocab // 2] = float("nan")
        assert _cross_entropy(bad, targets, _OneRank, 0).isnan().item()
