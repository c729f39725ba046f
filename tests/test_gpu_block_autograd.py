"""The one-kernel parts of a decoder block under autograd: what the plain operations took has to be taken, with the same meaning."""
import pytest
import torch

pytestmark = pytest.mark.gpu


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
