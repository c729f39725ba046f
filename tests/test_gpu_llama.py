"""The Llama-architecture decoder on one GPU: linears on the tcgen05 kernels (through a single-rank communicator) against
the same model on torch.matmul."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _NoComm:
    """Single-rank stand-in that routes every linear to torch.matmul."""
    size, rank, fused = 1, 0, False

    def all_gather(self, send, recv, stream=None):
        recv.copy_(send.reshape(recv.shape))

    def reduce_scatter(self, send, recv, op=None, stream=None):
        recv.copy_(send.reshape(recv.shape))

    def all_reduce(self, send, recv=None, op=None, stream=None):
        if recv is not None and recv.data_ptr() != send.data_ptr():
            recv.copy_(send)

    def synchronize(self):
        pass


def test_tiny_llama_matches_torch_matmul_reference():
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.models.llama import Llama, LlamaConfig
    from hccl_b200.ops import gemm
    from hccl_b200.parallel import tensor_parallel

    cfg = LlamaConfig.tiny(vocab=512, hidden=256, layers=2, heads=8, kv_heads=4, ffn=512)
    tok = torch.randint(0, cfg.vocab_size, (2, 129), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        ours = Llama(cfg, comm, dtype=torch.bfloat16, device="cuda", seed=3)
        loss = ours(tok[:, :-1], tok[:, 1:].contiguous())
        loss.backward()
        torch.cuda.synchronize()
        gemm.check_error()
        tensor_parallel.use_native_gemm(False)
        ref = Llama(cfg, _NoComm(), dtype=torch.bfloat16, device="cuda", seed=3)
        rloss = ref(tok[:, :-1], tok[:, 1:].contiguous())
        rloss.backward()
        torch.cuda.synchronize()
    finally:
        tensor_parallel.use_native_gemm(True)
        comm.destroy()
    assert abs(loss.item() - rloss.item()) < 2e-2
    for (n1, p1), (n2, p2) in zip(ours.named_parameters(), ref.named_parameters()):
        a, b = p1.grad.float(), p2.grad.float()
        assert (a - b).abs().max().item() <= 5e-2 * (b.abs().max().item() + 1e-3), n1


def _close(got, ref, mag, terms):
    """|got - ref| within one rounding to bf16 plus 32-bit arithmetic over `terms` terms of size `mag`."""
    err, bound = (got.double() - ref).abs(), ref.abs() * 2.0 ** -8 + mag * (terms + 16) * 2.0 ** -23
    assert bool((err <= bound + 1e-30).all()), (err - bound).max().item()


@pytest.mark.parametrize("rows,hidden", [(1, 8), (9, 264), (300, 1024), (7, 1032), (600, 4096), (3, 12288)])
def test_rms_norm_kernels(rows, hidden):
    """A warp per row up to 1024 columns, a block beyond; rows that do not fill a block; more rows than blocks in the backward pass."""
    from hccl_b200.models.llama import RMSNorm
    g = torch.Generator(device="cuda").manual_seed(rows)
    norm = RMSNorm(hidden, 1e-5, torch.bfloat16, "cuda")
    with torch.no_grad():
        norm.weight.copy_(torch.randn(hidden, generator=g, device="cuda"))
    x = torch.randn(rows, hidden, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    dy = torch.randn(rows, hidden, generator=g, device="cuda").to(torch.bfloat16)
    y = norm(x)
    assert y.grad_fn.name().startswith("_RmsNorm")
    dx, dw = torch.autograd.grad(y, [x, norm.weight], dy)
    xd, wd, gd = x.detach().double(), norm.weight.detach().double(), dy.double()
    r = torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5)
    xh, dg = xd * r, gd * wd
    _close(y, xh * wd, (xh * wd).abs(), hidden)
    _close(dx, r * (dg - xh * (dg * xh).mean(-1, keepdim=True)), r * (dg.abs() + xh.abs() * (dg * xh).abs().mean(-1, keepdim=True)), hidden)
    _close(dw, (gd * xh).sum(0), (gd * xh).abs().sum(0), hidden)
    # the gradient of the gradient, a forward transform and another type go through the plain form
    gx, = torch.autograd.grad(norm(x), x, dy, create_graph=True)
    assert torch.isfinite(torch.autograd.grad(gx.float().square().sum(), x)[0]).all()
    assert torch.func.jvp(lambda t: norm(t), (x.detach(),), (dy,))[1].shape == x.shape
    assert torch.func.vmap(lambda t: norm(t))(x.detach()).shape == x.shape
    assert norm(x.detach()[:0]).shape == (0, hidden)


@pytest.mark.parametrize("batch,seq,heads,kv,hd", [(1, 1, 1, 1, 16), (2, 37, 8, 4, 32), (3, 64, 6, 2, 128)])
def test_rope_qkv_kernels(batch, seq, heads, kv, hd):
    from hccl_b200.models.llama import Attention, _rope_tables
    from hccl_b200.ops import block
    att = Attention.__new__(Attention)
    torch.nn.Module.__init__(att)
    att.h_local, att.kv_local, att.hd = heads, kv, hd
    cos, sin = _rope_tables(seq, hd, 10000.0, "cuda")
    g = torch.Generator(device="cuda").manual_seed(seq)
    qkv = torch.randn(batch * seq, (heads + 2 * kv) * hd, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    out = block.rope_qkv(qkv, cos, sin, batch, heads, kv, hd, lambda t: att._rotated(t, batch, seq, cos, sin))
    ref = att._rotated(qkv, batch, seq, cos, sin)
    gs = [torch.randn(r.shape, generator=g, device="cuda").to(torch.bfloat16) for r in ref]
    gs[0] = gs[0].transpose(1, 2).contiguous().transpose(1, 2)                       # a gradient that is not contiguous
    for a, b in zip(out, ref):
        assert torch.equal(a, b)                                                     # the same two products and one sum per element
    d, = torch.autograd.grad(out, qkv, gs)
    e, = torch.autograd.grad(ref, qkv, gs)
    assert torch.equal(d, e)


@pytest.mark.parametrize("rows,ffn", [(1, 8), (37, 264), (300, 14336)])
def test_swiglu_kernels(rows, ffn):
    from hccl_b200.ops import block
    g = torch.Generator(device="cuda").manual_seed(rows)
    gu = (torch.randn(rows, 2 * ffn, generator=g, device="cuda") * 3).to(torch.bfloat16)
    gu[0, :4] = torch.tensor([-100.0, 100.0, 0.0, -1e30], device="cuda")             # exp overflows, stays finite, is exact
    gu.requires_grad_()
    dh = torch.randn(rows, ffn, generator=g, device="cuda").to(torch.bfloat16)
    h = block.swiglu(gu, None)
    d, = torch.autograd.grad(h, gu, dh)
    gg, uu, s = gu.detach().double()[:, :ffn], gu.detach().double()[:, ffn:], torch.sigmoid(gu.detach().double()[:, :ffn])
    assert torch.equal(h, torch.nn.functional.silu(gu.detach()[:, :ffn]) * gu.detach()[:, ffn:])
    _close(d[:, ffn:], dh.double() * gg * s, (dh.double() * gg).abs() * (s + 2.0 ** -20), 8)
    # the sigmoid's slope s (1 - s) multiplies gate: where 1 - s cancels, the error is that of s
    ref = dh.double() * uu * s * (1 + gg * (1 - s))
    _close(d[:, :ffn][1:], ref[1:], ((dh.double() * uu).abs() * s * (1 + gg.abs()))[1:], 8)
    assert torch.isfinite(d.float()).all()


@pytest.mark.parametrize("rows,vocab,start", [(1, 8, 0), (33, 1000, 0), (20, 1003, 500), (5, 32064, 0)])
def test_cross_entropy_kernels(rows, vocab, start):
    """Vector and scalar widths, a shard that owns only some of the targets."""
    from hccl_b200.ops import block
    g = torch.Generator(device="cuda").manual_seed(rows)
    logits = (torch.randn(rows, vocab, generator=g, device="cuda") * 4).to(torch.bfloat16)
    if vocab > 8:
        logits[0, 3] = -float("inf")
    t = torch.randint(0, vocab + start, (rows,), generator=g, device="cuda")
    ld = logits.double()
    mx = block.xent_row_max(logits)
    assert torch.equal(mx, logits.float().max(1).values)
    packed = block.xent_sums(logits, t, start, mx)
    ex = (ld - mx.double()[:, None]).exp()
    mine = (t >= start) & (t < start + vocab)
    own = (t - start).clamp(0, vocab - 1)
    assert bool(((packed[0].double() - ex.sum(1)).abs() <= ex.sum(1) * (vocab + 64) * 2.0 ** -23).all())
    assert torch.equal(packed[1], torch.where(mine, logits.float().gather(1, own[:, None])[:, 0] - mx, torch.zeros_like(mx)))
    go = torch.tensor(0.7, device="cuda")
    grad = block.xent_grad(logits, t, start, mx, packed, go)
    hot = torch.zeros_like(ld)
    hot[torch.arange(rows, device="cuda")[mine], own[mine]] = 1
    p = ex / ex.sum(1, keepdim=True)
    _close(grad, (p - hot) * 0.7 / rows, (p + hot) * 0.7 / rows, vocab)
