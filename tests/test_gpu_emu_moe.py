"""MoE dispatch + combine with all ranks emulated on one GPU (identity experts): every token must come back as
(sum of its top-k weights) * token, and the per-expert receive counts must equal the routing histogram."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nranks,T,E,K,H", [(2, 64, 8, 2, 256), (4, 300, 32, 4, 512), (4, 128, 64, 8, 1024), (8, 96, 64, 8, 256)])
def test_dispatch_combine_round_trip(nranks, T, E, K, H):
    from hccl_b200.ops import moe
    from hccl_b200.utils import emu
    l = moe._decl()
    cfg = moe.HcclMoeConfig(E, K, H, T, nranks * T * K, 0)
    g = torch.Generator(device="cuda").manual_seed(11)
    xs = [torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16) for _ in range(nranks)]
    # skewed routing: a bias makes low expert ids more popular
    bias = -0.3 * torch.arange(E, device="cuda").float().log1p()
    idxs = [torch.topk(torch.randn(T, E, generator=g, device="cuda") + bias, K, dim=1).indices.to(torch.int32).contiguous() for _ in range(nranks)]
    ws = [torch.rand(T, K, generator=g, device="cuda").contiguous() for _ in range(nranks)]
    outs = [torch.zeros(T, H, dtype=torch.bfloat16, device="cuda") for _ in range(nranks)]
    counts = [torch.zeros(E // nranks, dtype=torch.int32, device="cuda") for _ in range(nranks)]
    arena = (4 * nranks * T * K * H * 2 + (8 << 20))
    ctas = max(1, min(16, 148 // nranks))
    with emu.EmuWorld(nranks, 1 << 20, arena_bytes=arena) as w:
        arr = lambda ts: (ctypes.c_void_p * nranks)(*[t.data_ptr() for t in ts])
        for it in range(2):   # the second round reuses buffers, flags and epochs
            rc = l.HcclEmuMoeRoundTrip(w._h, ctypes.byref(cfg), arr(xs), arr(idxs), arr(ws), arr(outs), T, arr(counts), ctas)
            torch.cuda.synchronize()
            assert rc == 0
            hist = torch.zeros(E, dtype=torch.int64, device="cuda")
            for r in range(nranks):
                hist += torch.bincount(idxs[r].flatten().long(), minlength=E)
            got = torch.cat(counts).long()
            assert torch.equal(got, hist)
            for r in range(nranks):
                ref = xs[r].float() * ws[r].sum(1, keepdim=True)
                err = (outs[r].float() - ref).abs().max().item() / (ref.abs().max().item() + 1e-6)
                assert err < 2e-2, err


def test_capacity_overflow_is_reported_not_written():
    from hccl_b200.ops import moe
    from hccl_b200.utils import emu
    l = moe._decl()
    nranks, T, E, K, H = 2, 64, 4, 2, 256
    cfg = moe.HcclMoeConfig(E, K, H, T, 16, 0)      # far too small a receive buffer
    xs = [torch.randn(T, H, device="cuda").to(torch.bfloat16) for _ in range(nranks)]
    idxs = [torch.zeros(T, K, dtype=torch.int32, device="cuda") + torch.tensor([0, 1], dtype=torch.int32, device="cuda") for _ in range(nranks)]
    ws = [torch.ones(T, K, device="cuda") for _ in range(nranks)]
    outs = [torch.zeros(T, H, dtype=torch.bfloat16, device="cuda") for _ in range(nranks)]
    with emu.EmuWorld(nranks, 1 << 20, arena_bytes=8 << 20) as w:
        arr = lambda ts: (ctypes.c_void_p * nranks)(*[t.data_ptr() for t in ts])
        rc = l.HcclEmuMoeRoundTrip(w._h, ctypes.byref(cfg), arr(xs), arr(idxs), arr(ws), arr(outs), T, None, 8)
        torch.cuda.synchronize()
        assert rc == 3     # HCCL_E_MEMORY: reported through the status word, no out-of-bounds write


def _moe_quant_reference(x):
    """The dispatch kernel's block rule in plain PyTorch: per 1 x 32 block the smallest power-of-two scale with amax / scale <= 448,
    values divided by it and rounded to e4m3; returns the dequantised fp32 tensor, the e4m3 bytes and the e8m0 scale bytes."""
    T, H = x.shape
    v = x.float().view(T, H // 32, 32)
    amax = v.abs().amax(2)
    m, e = torch.frexp(amax / 448.0)                       # amax / 448 = m * 2^e, m in [0.5, 1)
    e = torch.where(m == 0.5, e - 1, e)
    biased = torch.where(amax > 0, (e + 127).clamp(0, 254), torch.full_like(e, 127 - 8))
    scale = torch.exp2((biased - 127).float())
    q = (v / scale.unsqueeze(2)).to(torch.float8_e4m3fn)
    return (q.float() * scale.unsqueeze(2)).view(T, H), q.view(torch.uint8).view(T, H), biased.to(torch.uint8)


@pytest.mark.parametrize("nranks,T,E,K,H", [(2, 64, 8, 2, 256), (4, 200, 32, 4, 512), (4, 96, 64, 8, 1024)])
def test_mxfp8_dispatch_round_trip_matches_the_reference_quantiser(nranks, T, E, K, H):
    """Dispatch with the block-scaled payload (e4m3 + e8m0 scale per 32 values): the stand-in experts dequantise what they
    received, so every token must come back as (sum of its top-k weights) * dequantise(quantise(token)) -- the payload and the
    scales both have to be right, for blocks whose magnitudes differ by orders of magnitude."""
    from hccl_b200.ops import moe
    from hccl_b200.utils import emu
    l = moe._decl()
    cfg = moe.HcclMoeConfig(E, K, H, T, nranks * T * K, 1)
    g = torch.Generator(device="cuda").manual_seed(23)
    xs = []
    for _ in range(nranks):
        x = torch.randn(T, H // 32, 32, generator=g, device="cuda") * torch.exp2(torch.randint(-8, 9, (T, H // 32, 1), generator=g, device="cuda").float())
        x = x.view(T, H).to(torch.bfloat16)
        x[0, :32] = 0                                     # an all-zero block
        x[1, 32:64] = 448.0                               # a block exactly at the top of a binade
        xs.append(x.contiguous())
    idxs = [torch.topk(torch.randn(T, E, generator=g, device="cuda"), K, dim=1).indices.to(torch.int32).contiguous() for _ in range(nranks)]
    ws = [torch.rand(T, K, generator=g, device="cuda").contiguous() for _ in range(nranks)]
    outs = [torch.zeros(T, H, dtype=torch.bfloat16, device="cuda") for _ in range(nranks)]
    counts = [torch.zeros(E // nranks, dtype=torch.int32, device="cuda") for _ in range(nranks)]
    arena = (4 * nranks * T * K * H * 2 + (8 << 20))
    ctas = max(1, min(16, 148 // nranks))
    with emu.EmuWorld(nranks, 1 << 20, arena_bytes=arena) as w:
        arr = lambda ts: (ctypes.c_void_p * nranks)(*[t.data_ptr() for t in ts])
        for it in range(2):
            rc = l.HcclEmuMoeRoundTrip(w._h, ctypes.byref(cfg), arr(xs), arr(idxs), arr(ws), arr(outs), T, arr(counts), ctas)
            torch.cuda.synchronize()
            assert rc == 0
            for r in range(nranks):
                deq, _, _ = _moe_quant_reference(xs[r])
                # experts return bf16(dequantised); combine sums K weighted copies in fp32 and rounds to bf16 once more
                ref = deq.to(torch.bfloat16).float() * ws[r].sum(1, keepdim=True)
                err = (outs[r].float() - ref).abs() / (ref.abs() + 1e-30)
                assert float(err[ref.abs() > 0].max()) < 2.0 ** -6, float(err[ref.abs() > 0].max())
                assert bool((outs[r].float()[ref == 0] == 0).all())
                # and the format itself stays within e4m3's half-ulp (2^-4) of the block maximum
                blk = xs[r].float().view(T, H // 32, 32)
                assert bool(((deq.view(T, H // 32, 32) - blk).abs().amax(2) <= blk.abs().amax(2) * 2.0 ** -4 + 1e-30).all())


@pytest.mark.parametrize("T,E,K,H,mxfp8", [(1, 8, 1, 256, False), (3, 60, 6, 1280, False), (700, 256, 8, 512, True), (300, 320, 16, 1024, False), (257, 5, 3, 2304, True)])
def test_one_rank_layout_and_combine(T, E, K, H, mxfp8):
    """One rank (no barrier among CTAs): rows sorted by expert, then by token; few and many tokens per CTA, widths that are not whole
    2 KB pieces, topK 16, the largest expert count."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops.moe import MoeDispatcher
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        g = torch.Generator(device="cuda").manual_seed(T + E)
        x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
        x[0, :32] = 0
        idx = torch.stack([torch.randperm(E, generator=g, device="cuda")[:K] if K <= E else torch.zeros(K, device="cuda") for _ in range(T)]).to(torch.int32).contiguous()
        w = torch.rand(T, K, generator=g, device="cuda")
        d = MoeDispatcher(comm, E, K, H, T, max_recv_rows=T * K, mxfp8=mxfp8)
        rx, rs, counts, src = d.dispatch(x, idx)
        y = torch.randn(T * K, H, generator=g, device="cuda").to(torch.bfloat16)
        d.expert_out.copy_(y)
        out = d.combine(w)
        torch.cuda.synchronize()
        order = torch.argsort(idx.flatten().long(), stable=True)
        assert torch.equal(counts.long(), torch.bincount(idx.flatten().long(), minlength=E))
        assert torch.equal(src.long(), order // K)
        rows = x[order // K]
        if mxfp8:
            val = rx.float().view(T * K, H // 32, 32) * torch.exp2(rs.float() - 127)[..., None]
            amax = rows.float().view(T * K, H // 32, 32).abs().amax(2, keepdim=True)
            assert bool(((val - rows.float().view_as(val)).abs() <= amax * 2.0 ** -4).all())     # 3 mantissa bits, no saturation
        else:
            assert torch.equal(rx, rows)
        slot = torch.empty_like(order)
        slot[order] = torch.arange(T * K, device="cuda")
        terms = w.double()[..., None] * y[slot.view(T, K)].double()
        ref = terms.sum(1)
        assert bool(((out.double() - ref).abs() <= terms.abs().sum(1) * K * 2.0 ** -23 + ref.abs() * 2.0 ** -8).all())
        d.close()
    finally:
        comm.destroy()


@pytest.mark.parametrize("T,E,K,H,mxfp8", [(5, 8, 2, 256, False), (40, 8, 4, 2304, True), (300, 16, 16, 512, False)])
def test_one_rank_ids_outside_the_experts_add_nothing(T, E, K, H, mxfp8):
    """Ids -1 and E are sent and counted nowhere; the combine reads zeros for them, also where an earlier call gave the entry a
    row and whatever the expert outputs hold."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops.moe import MoeDispatcher
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        g = torch.Generator(device="cuda").manual_seed(T)
        x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
        idx = torch.randint(0, E, (T, K), generator=g, device="cuda").to(torch.int32)
        w = torch.rand(T, K, generator=g, device="cuda")
        d = MoeDispatcher(comm, E, K, H, T, max_recv_rows=T * K, mxfp8=mxfp8)
        for step in range(2):                                  # the second routing masks some entries of the first, one token wholly
            if step:
                idx[torch.rand(T, K, generator=g, device="cuda") < 0.3] = -1
                idx[torch.rand(T, K, generator=g, device="cuda") < 0.1] = E
                idx[T // 2] = -1
            ok = (idx >= 0) & (idx < E)
            _, _, counts, src = d.dispatch(x, idx)
            y = torch.randn(T * K, H, generator=g, device="cuda").to(torch.bfloat16)
            y[int(ok.sum()):] = float("nan")                   # no expert wrote these rows
            d.expert_out.copy_(y)
            out = d.combine(w)
            torch.cuda.synchronize()
            flat = idx.flatten().long()
            order = torch.argsort(torch.where(ok.flatten(), flat, E), stable=True)[: int(ok.sum())]
            assert torch.equal(counts.long(), torch.bincount(flat[ok.flatten()], minlength=E))
            assert torch.equal(src[: len(order)].long(), order // K)
            slot = torch.zeros(T * K, dtype=torch.long, device="cuda")
            slot[order] = torch.arange(len(order), device="cuda")
            terms = torch.where(ok[..., None], w.double()[..., None] * y[slot.view(T, K)].double(), 0.0)
            ref = terms.sum(1)
            assert bool(((out.double() - ref).abs() <= terms.abs().sum(1) * K * 2.0 ** -23 + ref.abs() * 2.0 ** -8).all())
        assert bool((out[T // 2] == 0).all())
        d.close()
    finally:
        comm.destroy()


def test_one_rank_overflow_leaves_the_combine_no_rows():
    """More rows than the receive buffer holds, on one rank: reported, nothing moved, and a combine that was already queued behind the
    dispatch writes zeros."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops.moe import MoeDispatcher
    T, E, K, H = 64, 4, 2, 256
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        d = MoeDispatcher(comm, E, K, H, T, max_recv_rows=T * K - 1)
        d.expert_out.fill_(3.0)
        x, idx = torch.ones(T, H, dtype=torch.bfloat16, device="cuda"), torch.zeros(T, K, dtype=torch.int32, device="cuda")
        out, w = torch.ones(T, H, dtype=torch.bfloat16, device="cuda"), torch.ones(T, K, device="cuda")
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)                          # about 10 ms: the combine is queued before the dispatch has run
        rx = d.dispatch(x, idx)[0]
        d.combine(w, out)
        torch.cuda.synchronize()
        assert bool((out == 0).all())
        with pytest.raises(Exception):
            d.dispatch(x, idx)
        assert rx.shape[0] == T * K - 1
    finally:
        comm.destroy()


def test_receive_views_belong_to_their_call():
    """A first dispatch under inference mode leaves later ones trainable, and writing one call's tensor does not mark another's as changed."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops.moe import MoeDispatcher
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        d = MoeDispatcher(comm, 8, 2, 256, 16, max_recv_rows=32)
        x = torch.randn(16, 256, device="cuda").to(torch.bfloat16)
        idx = torch.randint(0, 8, (16, 2), device="cuda", dtype=torch.int32)
        w = torch.randn(256, 64, device="cuda").to(torch.bfloat16).requires_grad_()
        with torch.inference_mode():
            d.dispatch(x, idx)
        first = d.dispatch(x, idx)[0]
        y = first @ w
        second = d.dispatch(x, idx)[0]
        second.mul_(1)
        torch.autograd.backward(y, torch.ones_like(y))
        assert torch.equal(w.grad, first.t() @ torch.ones_like(y))
        d.close()
    finally:
        comm.destroy()


def test_calls_that_the_host_refuses_leave_the_dispatcher_usable():
    """Rows and results that are not 16-byte aligned (they move in such pieces) and a combine before the first dispatch are refused on the host, and the next call is right."""
    from hccl_b200._lib import HcclError
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops.moe import MoeDispatcher
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        d = MoeDispatcher(comm, 8, 2, 256, 16, max_recv_rows=32)
        x = torch.randn(16, 256, device="cuda").to(torch.bfloat16)
        idx = torch.randint(0, 8, (16, 2), device="cuda", dtype=torch.int32)
        weights = torch.rand(16, 2, device="cuda")
        off = torch.empty(16 * 256 + 8, dtype=torch.bfloat16, device="cuda")[1:16 * 256 + 1].view(16, 256)
        with pytest.raises(HcclError):
            d.combine(weights)
        with pytest.raises(HcclError):
            d.dispatch(off.copy_(x), idx)
        recv, _, counts, src = d.dispatch(x, idx)
        assert torch.equal(recv[:32], x[src.long()]) and torch.equal(counts.long(), torch.bincount(idx.flatten().long(), minlength=8))
        d.expert_out.copy_(recv)
        with pytest.raises(HcclError):
            d.combine(weights, out=off)
        want = (x.double()[:, None] * weights.double()[..., None]).sum(1)
        assert bool(((d.combine(weights).double() - want).abs() <= want.abs() * 2.0 ** -8 + x.double().abs() * 2.0 ** -21).all())
        d.close()
    finally:
        comm.destroy()


@pytest.mark.parametrize("T,E,K", [(1, 8, 1), (37, 16, 3), (700, 256, 8)])
def test_one_rank_routing_table_that_is_not_16_byte_aligned(T, E, K):
    """The histogram reads four entries at a time where it can, one at a time from an address that does not allow it."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops.moe import MoeDispatcher
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        g = torch.Generator(device="cuda").manual_seed(T)
        x = torch.randn(T, 256, generator=g, device="cuda").to(torch.bfloat16)
        idx = torch.empty(T * K + 1, dtype=torch.int32, device="cuda")[1:].view(T, K)
        idx.copy_(torch.randint(0, E, (T, K), generator=g, device="cuda"))
        assert idx.data_ptr() % 16
        d = MoeDispatcher(comm, E, K, 256, T, max_recv_rows=T * K)
        rx, _, counts, src = d.dispatch(x, idx)
        torch.cuda.synchronize()
        order = torch.argsort(idx.flatten().long(), stable=True)
        assert torch.equal(counts.long(), torch.bincount(idx.flatten().long(), minlength=E))
        assert torch.equal(src.long(), order // K) and torch.equal(rx, x[order // K])
        d.close()
    finally:
        comm.destroy()


@pytest.mark.parametrize("nranks,T,E,K,H", [(2, 40, 8, 2, 256), (4, 128, 64, 8, 1024)])
def test_ids_outside_the_experts_among_ranks(nranks, T, E, K, H):
    """The same with several ranks and identity experts: a token comes back as the sum of its valid entries' weights times itself, in the
    second routing too, which masks entries that had rows in the first."""
    from hccl_b200.ops import moe
    from hccl_b200.utils import emu
    l = moe._decl()
    cfg = moe.HcclMoeConfig(E, K, H, T, nranks * T * K, 0)
    g = torch.Generator(device="cuda").manual_seed(5)
    xs = [torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16) for _ in range(nranks)]
    idxs = [torch.randint(0, E, (T, K), generator=g, device="cuda").to(torch.int32) for _ in range(nranks)]
    ws = [torch.rand(T, K, generator=g, device="cuda") for _ in range(nranks)]
    outs = [torch.zeros(T, H, dtype=torch.bfloat16, device="cuda") for _ in range(nranks)]
    counts = [torch.zeros(E // nranks, dtype=torch.int32, device="cuda") for _ in range(nranks)]
    with emu.EmuWorld(nranks, 1 << 20, arena_bytes=4 * nranks * T * K * H * 2 + (8 << 20)) as w:
        arr = lambda ts: (ctypes.c_void_p * nranks)(*[t.data_ptr() for t in ts])
        for step in range(2):
            if step:
                for r, idx in enumerate(idxs):
                    idx[torch.rand(T, K, generator=g, device="cuda") < 0.3] = -1 if r % 2 else E
                    idx[r] = -1
            assert l.HcclEmuMoeRoundTrip(w._h, ctypes.byref(cfg), arr(xs), arr(idxs), arr(ws), arr(outs), T, arr(counts), max(1, min(16, 148 // nranks))) == 0
            torch.cuda.synchronize()
            ok = [(i >= 0) & (i < E) for i in idxs]
            assert torch.equal(torch.cat(counts).long(), sum(torch.bincount(i[o].long(), minlength=E) for i, o in zip(idxs, ok)))
            for x, o, wt, out in zip(xs, ok, ws, outs):
                ref = x.double() * torch.where(o, wt, 0.0).double().sum(1, keepdim=True)
                assert bool(((out.double() - ref).abs() <= ref.abs() * (2.0 ** -8 + K * 2.0 ** -23) + 1e-30).all())


@pytest.mark.parametrize("T,E,K,H,mxfp8,ctas", [(512, 256, 8, 256, False, ""), (513, 256, 8, 256, False, ""), (4096, 320, 1, 512, True, ""), (4097, 7, 1, 256, False, ""), (1, 3, 2, 7168, True, ""),
                                                (256, 64, 16, 2304, True, ""), (100, 16, 8, 512, False, "5"), (40, 16, 8, 512, True, "40")])
def test_one_rank_few_tokens(T, E, K, H, mxfp8, ctas, monkeypatch):
    """Both sides of the lines between the dispatch that counts rows directly and the general one (entries in all, entries per CTA), some entries
    without a row: the general kernel's layout, and a combine over it."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops.moe import MoeDispatcher
    if ctas:
        monkeypatch.setenv("HCCL_MOE_CTAS", ctas)
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        g = torch.Generator(device="cuda").manual_seed(T + K)
        x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
        idx = torch.randint(0, E, (T, K), generator=g, device="cuda").to(torch.int32)
        idx[torch.rand(T, K, generator=g, device="cuda") < 0.05] = -1
        w = torch.rand(T, K, generator=g, device="cuda")
        d = MoeDispatcher(comm, E, K, H, T, max_recv_rows=T * K, mxfp8=mxfp8)
        rx, rs, counts, src = d.dispatch(x, idx)
        y = torch.randn(T * K, H, generator=g, device="cuda").to(torch.bfloat16)
        d.expert_out.copy_(y)
        out = d.combine(w)
        torch.cuda.synchronize()
        flat, ok = idx.flatten().long(), (idx >= 0)
        n = int(ok.sum())
        order = torch.argsort(torch.where(ok.flatten(), flat, E), stable=True)[:n]
        assert torch.equal(counts.long(), torch.bincount(flat[ok.flatten()], minlength=E))
        assert torch.equal(src[:n].long(), order // K)
        rows = x[order // K]
        if mxfp8:
            amax = rows.float().view(n, H // 32, 32).abs().amax(2)
            assert torch.equal(rs[:n].long(), torch.ceil(torch.log2(amax.double() / 448)).long() + 127)
            scaled = rows.float().view(n, H // 32, 32) * torch.exp2(127 - rs[:n].float())[..., None]
            assert torch.equal(rx[:n].view(torch.uint8), scaled.to(torch.float8_e4m3fn).view(n, H).view(torch.uint8))
        else:
            assert torch.equal(rx[:n], rows)
        slot = torch.zeros(T * K, dtype=torch.long, device="cuda")
        slot[order] = torch.arange(n, device="cuda")
        terms = torch.where(ok[..., None], w.double()[..., None] * y[slot.view(T, K)].double(), 0.0)
        ref = terms.sum(1)
        assert bool(((out.double() - ref).abs() <= terms.abs().sum(1) * K * 2.0 ** -23 + ref.abs() * 2.0 ** -8).all())
        d.close()
    finally:
        comm.destroy()


@pytest.mark.parametrize("T,E,K,H,mxfp8,ctas", [(700, 64, 16, 512, False, "3"), (700, 64, 14, 768, True, "3"), (513, 320, 13, 256, False, "2"), (4097, 9, 1, 1280, True, "2"), (900, 32, 5, 2304, False, "7"),
                                                (300, 8, 2, 7168, True, ""), (2500, 60, 6, 1024, False, ""), (333, 256, 7, 4352, True, "")])
def test_one_rank_rings(T, E, K, H, mxfp8, ctas, monkeypatch):
    """The rings of the one-rank kernels: several batches of entries per CTA in both directions, every depth, a last piece that is not whole, ragged
    ranges, some entries without a row. Rows and scales are bytes; the combine adds at most 16 products in 32 bits and rounds once."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops.moe import MoeDispatcher
    if ctas:
        monkeypatch.setenv("HCCL_MOE_CTAS", ctas)
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        g = torch.Generator(device="cuda").manual_seed(T + K)
        x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
        idx = torch.randint(0, E, (T, K), generator=g, device="cuda").to(torch.int32)
        idx[torch.rand(T, K, generator=g, device="cuda") < 0.05] = E
        w = torch.rand(T, K, generator=g, device="cuda")
        d = MoeDispatcher(comm, E, K, H, T, max_recv_rows=T * K, mxfp8=mxfp8)
        rx, rs, counts, src = d.dispatch(x, idx)
        y = torch.randn(T * K, H, generator=g, device="cuda").to(torch.bfloat16)
        d.expert_out.copy_(y)
        out = d.combine(w)
        torch.cuda.synchronize()
        flat, ok = idx.flatten().long(), idx < E
        n = int(ok.sum())
        order = torch.argsort(flat, stable=True)[:n]
        assert torch.equal(counts.long(), torch.bincount(flat[ok.flatten()], minlength=E))
        assert torch.equal(src[:n].long(), order // K)
        rows = x[order // K]
        if mxfp8:
            _, q, se = _moe_quant_reference(rows)
            assert torch.equal(rx[:n].view(torch.uint8), q) and torch.equal(rs[:n], se)
        else:
            assert torch.equal(rx[:n], rows)
        slot = torch.zeros(T * K, dtype=torch.long, device="cuda")
        slot[order] = torch.arange(n, device="cuda")
        ref, bound = torch.zeros(T, H, dtype=torch.float64, device="cuda"), torch.zeros(T, H, dtype=torch.float64, device="cuda")
        for j in range(K):
            term = torch.where(ok[:, j, None], w[:, j, None].double() * y[slot.view(T, K)[:, j]].double(), 0.0)
            ref += term
            bound += term.abs()
        assert bool(((out.double() - ref).abs() <= bound * K * 2.0 ** -23 + ref.abs() * 2.0 ** -8).all())
        d.close()
    finally:
        comm.destroy()


@pytest.mark.parametrize("T,E,K,H,mxfp8", [(1, 8, 2, 1024, False), (333, 256, 7, 4352, True), (2500, 60, 6, 1024, False), (700, 64, 16, 512, True)])
def test_one_rank_without_rings(T, E, K, H, mxfp8, monkeypatch):
    """The kernels that move rows through registers, for contexts without the rings' shared memory: the same rows, scales and sums."""
    monkeypatch.setenv("HCCL_MOE_RINGS", "0")
    test_one_rank_rings(T, E, K, H, mxfp8, "", monkeypatch)
