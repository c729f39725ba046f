"""Block-scaled fp8 (MXFP8) kernels: the quantiser against a plain PyTorch restatement of its rule, the tcgen05 block-scaled
GEMM against an fp32 PyTorch product of the DEQUANTISED operands, and the three fused operators on emulated ranks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _wild(shape, seed, base=1.0):
    """bf16 data whose 1 x 32 blocks differ in magnitude by up to 2^12, so a wrong scale byte cannot hide."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rows, k = shape
    x = torch.randn(rows, k // 32, 32, generator=g, device="cuda") * base
    e = torch.randint(-6, 7, (rows, k // 32, 1), generator=g, device="cuda").float()
    return (x * torch.exp2(e)).view(rows, k).to(torch.bfloat16)


def _rel(out, ref):
    return (out.float() - ref).abs().max().item() / (ref.abs().max().item() + 1e-12)


@pytest.mark.parametrize("rows,k", [(128, 128), (200, 256), (1024, 1024), (77, 384)])
def test_quantiser_matches_the_reference_rule(rows, k):
    from hccl_b200.ops import mxfp8 as mx
    x = _wild((rows, k), rows + k)
    x[0, :32] = 0                                   # an all-zero block
    x[1, 32:64] = 448.0 * 2.0 ** 3                  # a block at the top of a binade
    q = mx.quantize(x)
    torch.cuda.synchronize()
    ref = mx.quantize_reference(x)
    assert torch.equal(q.scales, ref.scales)
    assert torch.equal(q.payload, ref.payload)
    # the format loses at most 2^-3 of the block maximum: 3 mantissa bits round to nearest (2^-4), and a block whose scaled
    # maximum lands in (448, 512) saturates at 448
    d = mx.dequantize(q)
    blk = x.float().view(rows, k // 32, 32)
    err = (d.view(rows, k // 32, 32) - blk).abs().amax(2)
    assert bool((err <= blk.abs().amax(2) * 2.0 ** -3 + 1e-30).all())


@pytest.mark.parametrize("m,n,k,tile", [(128, 128, 128, 128), (128, 256, 256, 256), (256, 512, 1024, 128), (384, 768, 512, 256),
                                        (200, 264, 384, 128), (200, 264, 384, 256), (1024, 1024, 2048, 0), (4096, 4096, 512, 0),
                                        # 192-wide tiles: odd tiles start at row 64 of a scale atom; partial last tiles; a single tile
                                        (128, 192, 128, 192), (256, 384, 512, 192), (384, 960, 640, 192), (200, 264, 384, 192), (2048, 8192, 512, 192),
                                        # CTA pairs (2256 / 2192 = 256- / 192-wide pair tiles): one pair, an odd number of row blocks (the second CTA of
                                        # the last pair idles), partial tiles in both directions, many tiles per pair
                                        (256, 256, 128, 2256), (128, 256, 256, 2256), (384, 768, 512, 2256), (200, 264, 384, 2256), (4096, 4096, 512, 2256),
                                        (256, 192, 128, 2192), (384, 960, 640, 2192), (200, 264, 384, 2192), (2048, 8192, 512, 2192)])
def test_block_scaled_gemm_matches_fp32_product_of_dequantised_operands(m, n, k, tile):
    from hccl_b200.ops import gemm as g, mxfp8 as mx
    a, w = mx.quantize(_wild((m, k), 1 + m)), mx.quantize(_wild((n, k), 2 + n, 0.05))
    ref = mx.dequantize(a) @ mx.dequantize(w).t()
    out32 = mx.gemm(a, w, out_dtype=torch.float32, tile_n=tile)
    out16 = mx.gemm(a, w, tile_n=tile)
    torch.cuda.synchronize()
    g.check_error()
    assert _rel(out32, ref) < 2e-3
    assert _rel(out16, ref) < 1e-2


def test_block_scaled_gemm_every_scale_byte_is_used():
    """Scales that differ for every (row, K block): one row of A and one of B get huge scales in single blocks; a kernel that
    picked a neighbouring block's or row's scale would be off by orders of magnitude."""
    from hccl_b200.ops import mxfp8 as mx
    m, n, k = 256, 256, 512
    a, w = torch.ones(m, k, device="cuda"), torch.ones(n, k, device="cuda")
    for kb in range(k // 32):
        a[(7 * kb) % m, kb * 32:(kb + 1) * 32] *= 2.0 ** (kb % 11)
        w[(13 * kb + 5) % n, kb * 32:(kb + 1) * 32] *= 2.0 ** -(kb % 9)
    qa, qw = mx.quantize(a.to(torch.bfloat16)), mx.quantize(w.to(torch.bfloat16))
    ref = mx.dequantize(qa) @ mx.dequantize(qw).t()
    for tile in (128, 192, 256, 2256, 2192):
        out = mx.gemm(qa, qw, out_dtype=torch.float32, tile_n=tile)
        torch.cuda.synchronize()
        assert torch.allclose(out, ref, rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("tile", [256, 192])
@pytest.mark.parametrize("nranks,m_local,N,K", [(2, 128, 256, 256), (4, 256, 512, 512), (2, 384, 776, 1024)])
def test_allgather_matmul_mxfp8(nranks, m_local, N, K, tile, monkeypatch):
    from hccl_b200.ops import mxfp8 as mx
    from hccl_b200.utils import emu
    monkeypatch.setenv("HCCL_MX_TILE_N", str(tile))
    ctas = 148 // nranks
    with emu.EmuWorld(nranks, 1 << 20, arena_bytes=(4 * nranks * m_local * K + (1 << 20))) as w:
        for it in range(3):
            a = [mx.quantize(_wild((m_local, K), 10 * it + r)) for r in range(nranks)]
            b = [mx.quantize(_wild((N, K), 100 + 10 * it + r, 0.05)) for r in range(nranks)]
            out = [torch.zeros(nranks * m_local, N, dtype=torch.bfloat16, device="cuda") for _ in range(nranks)]
            assert w.fused_mx(0, a, b, out, m_local, N, K, ctas, comm_ctas=2) == 0
            full = torch.cat([mx.dequantize(t) for t in a])
            for r in range(nranks):
                assert _rel(out[r], full @ mx.dequantize(b[r]).t()) < 1e-2


@pytest.mark.parametrize("tile", [256, 192])
@pytest.mark.parametrize("nranks,M,N,K", [(2, 256, 256, 256), (4, 512, 512, 384), (2, 512, 776, 256)])
def test_matmul_reduce_scatter_mxfp8(nranks, M, N, K, tile, monkeypatch):
    from hccl_b200.ops import mxfp8 as mx
    from hccl_b200.utils import emu
    monkeypatch.setenv("HCCL_MX_TILE_N", str(tile))
    ctas = 148 // nranks
    with emu.EmuWorld(nranks, 1 << 20, arena_bytes=(4 * M * N + (1 << 20))) as w:
        for it in range(2):
            a = [mx.quantize(_wild((M, K), 20 * it + r)) for r in range(nranks)]
            b = [mx.quantize(_wild((N, K), 200 + 20 * it + r, 0.05)) for r in range(nranks)]
            out = [torch.zeros(M // nranks, N, dtype=torch.bfloat16, device="cuda") for _ in range(nranks)]
            assert w.fused_mx(1, a, b, out, M, N, K, ctas) == 0
            partial = [(mx.dequantize(a[r]) @ mx.dequantize(b[r]).t()).to(torch.bfloat16).float() for r in range(nranks)]
            ref = sum(partial)
            rows = M // nranks
            for r in range(nranks):
                assert _rel(out[r], ref[r * rows:(r + 1) * rows]) < 1.5e-2


@pytest.mark.parametrize("nranks,M,N,K", [(2, 128, 256, 256), (4, 128, 1024, 512), (2, 200, 512, 128)])
def test_matmul_all_reduce_mxfp8(nranks, M, N, K):
    from hccl_b200.ops import mxfp8 as mx
    from hccl_b200.utils import emu
    ctas = min(148 // nranks, ((M + 127) // 128) * (N // 128))
    with emu.EmuWorld(nranks, 1 << 20, arena_bytes=(8 * M * N + (1 << 20))) as w:
        for it in range(2):
            a = [mx.quantize(_wild((M, K), 30 * it + r)) for r in range(nranks)]
            b = [mx.quantize(_wild((N, K), 300 + 30 * it + r, 0.05)) for r in range(nranks)]
            out = [torch.zeros(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(nranks)]
            assert w.fused_mx(2, a, b, out, M, N, K, ctas) == 0
            partial = [(mx.dequantize(a[r]) @ mx.dequantize(b[r]).t()).to(torch.bfloat16).float() for r in range(nranks)]
            ref = sum(partial)
            for r in range(nranks):
                assert _rel(out[r], ref) < 1.5e-2
                assert torch.equal(out[r], out[0])


@pytest.mark.parametrize("m,n,k,bt,split", [(1, 8, 128, 16, 1), (16, 264, 1024, 16, 8), (20, 128, 896, 32, 7), (64, 1000, 512, 64, 2), (200, 264, 384, 64, 3),
                                            (128, 8192, 256, 128, 2), (300, 136, 1024, 256, 4)])
def test_block_scaled_split_k(m, n, k, bt, split):
    """Split-K form: tiles of A that start inside a scale atom (32, 64 rows), two atoms (256), ragged rows and uneven K parts."""
    from hccl_b200.ops import gemm as g, mxfp8 as mx
    a, w = mx.quantize(_wild((m, k), 1 + m)), mx.quantize(_wild((n, k), 2 + n, 0.05))
    da, dw = mx.dequantize(a).double(), mx.dequantize(w).double()
    ref, mag = da @ dw.t(), da.abs() @ dw.abs().t()
    out = mx.gemm(a, w, out_dtype=torch.float32, tile_n=100000 + 1000 * split + bt)
    torch.cuda.synchronize()
    g.check_error()
    assert bool(((out.double() - ref).abs() <= mag * k * 2.0 ** -24 + 1e-30).all())


@pytest.mark.parametrize("m,n,k", [(65, 520, 512), (129, 5432, 1024), (513, 640, 8192), (700, 264, 4096), (1030, 776, 2048), (620, 4160, 512), (334, 6840, 768), (300, 11616, 2048), (1024, 4736, 4096)])
def test_chosen_kernel_of_many_rows(m, n, k):
    """Each kind of kernel that products of more than 64 rows take, ragged: fp32 results within k roundings of the sum of magnitudes, a result in bf16 its rounding."""
    from hccl_b200.ops import gemm as g, mxfp8 as mx
    a, w = mx.quantize(_wild((m, k), 1 + m)), mx.quantize(_wild((n, k), 2 + n, 0.05))
    da, dw = mx.dequantize(a).double(), mx.dequantize(w).double()
    ref, mag = da @ dw.t(), da.abs() @ dw.abs().t()
    out, half = mx.gemm(a, w, out_dtype=torch.float32), mx.gemm(a, w)
    torch.cuda.synchronize()
    g.check_error()
    assert bool(((out.double() - ref).abs() <= mag * k * 2.0 ** -24 + 1e-30).all())
    assert torch.equal(half, out.to(torch.bfloat16))


@pytest.mark.parametrize("m,n,k", [(1, 512, 512), (32, 8192, 1024), (64, 264, 14336), (300, 1024, 2048), (2048, 512, 256)])
def test_one_rank_operators_quantise_in_the_call(m, n, k):
    """bf16 activations on one rank: the bits of quantising first, also where the weights were written by the kernel right before the call
    (the product may read them while the activations are quantised) and where the buffers are reused by the next call."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops import mxfp8
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        xs = [_wild((m, k), 3 + i).to(torch.bfloat16) for i in range(3)]
        ws = [mxfp8.quantize(_wild((n, k), 9 + i).to(torch.bfloat16)) for i in range(3)]
        refs = [mxfp8.gemm(mxfp8.quantize(x), w) for x, w in zip(xs, ws)]
        shared = mxfp8.MxTensor(torch.zeros_like(ws[0].payload), torch.zeros_like(ws[0].scales), n, k)
        torch.cuda.synchronize()
        outs = []
        for op in (mxfp8.matmul_all_reduce, mxfp8.all_gather_matmul, mxfp8.matmul_reduce_scatter):
            for x, w in zip(xs, ws):
                shared.scales.copy_(w.scales)
                shared.payload.copy_(w.payload)
                outs.append(op(comm, x, shared))
        torch.cuda.synchronize()
        for i, out in enumerate(outs):
            assert torch.equal(out, refs[i % 3])
    finally:
        comm.destroy()


def test_one_rank_calls_keep_their_activations_apart():
    """Calls of one shape on two streams and from two threads, back to back: every one has its own quantised activations. Whole bytes and one kernel, so the results are
    those of a call by itself."""
    import threading

    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops import mxfp8
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        w = mxfp8.quantize(torch.randn(1024, 512, device="cuda").to(torch.bfloat16))
        xs = [torch.randn(48, 512, device="cuda").to(torch.bfloat16) for _ in range(16)]
        want = [mxfp8.gemm(mxfp8.quantize(x), w) for x in xs]
        torch.cuda.synchronize()
        streams, got = [torch.cuda.Stream(), torch.cuda.Stream()], [None] * 16

        def calls(part):
            for i in range(part, 16, 2):
                with torch.cuda.stream(streams[i // 2 % 2]):
                    got[i] = mxfp8.matmul_all_reduce(comm, xs[i], w, stream=streams[i // 4 % 2] if i % 3 == 0 else None)

        threads = [threading.Thread(target=calls, args=(p,)) for p in range(2)]
        [t.start() for t in threads]
        [t.join() for t in threads]
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    finally:
        comm.destroy()


def test_activations_of_a_call_on_an_explicit_stream_belong_to_that_stream():
    """Memory that has just become free on the current stream, where a copy that is still to run will read it, is not taken for a call on another stream."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops import mxfp8
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        m, n, k = 256, 512, 4096
        w, a = mxfp8.quantize(torch.randn(n, k, device="cuda").to(torch.bfloat16)), torch.randn(m, k, device="cuda").to(torch.bfloat16)
        want, out, s = mxfp8.gemm(mxfp8.quantize(a), w), torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), torch.cuda.Stream()
        size = m * k + mxfp8.scale_bytes(m, k)
        for stream in (s, torch.cuda.ExternalStream(s.cuda_stream)):
            src, dst = torch.full((size,), 7, dtype=torch.uint8, device="cuda"), torch.empty(size, dtype=torch.uint8, device="cuda")
            out.zero_()
            torch.cuda.synchronize()
            torch.cuda._sleep(20_000_000)                      # about 10 ms: the copy is queued, its source is free
            dst.copy_(src)
            del src
            assert mxfp8.matmul_all_reduce(comm, a, w, out=out, stream=stream) is out
            torch.cuda.synchronize()
            assert bool((dst == 7).all()) and torch.equal(out, want)
    finally:
        comm.destroy()


@pytest.mark.parametrize("m,n,k", [(1, 8, 256), (1, 512, 512), (3, 136, 640), (8, 4096, 4096), (15, 1000, 1152), (16, 14336, 4096), (16, 264, 16384), (17, 4096, 4096), (25, 2056, 2048), (32, 4096, 4096),
                                   (32, 1024, 14336), (33, 4096, 4096)])
def test_products_that_quantise_their_activations(m, n, k):
    """Few rows: the kernel that quantises for itself against the quantiser and the product, on both sides of the choice, rows and columns that do not fill a tile, blocks of zeros, of
    the largest values, of subnormals and with a NaN. The same bits: one rule, one order of sums."""
    from hccl_b200._lib import lib
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops import gemm as g, mxfp8 as mx
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        a, w = _wild((m, k), m + n), mx.quantize(_wild((n, k), n + k, 0.05))
        a[0, :32] = 0
        a[m // 2, 32:64] = 3.0e38
        a[m - 1, 64:96] = 1.0e-39
        for nan in (False, True):
            if nan:
                a[m // 3, 100] = float("nan")
            got = mx.matmul_all_reduce(comm, a, w)
            want = mx.gemm(mx.quantize(a), w)
            torch.cuda.synchronize()
            g.check_error()
            assert torch.equal(got.view(torch.int16), want.view(torch.int16))
        in_one = lib().HcclQuantizeGemmMxfp8InOne
        in_one.argtypes = [__import__("ctypes").c_uint64] * 3
        assert bool(in_one(m, n, k)) == (2 <= k // 128 and (m <= 16 and k >= 512 or 16 < m <= 32 and k >= 2048 and (m, n, k) != (32, 1024, 14336))), in_one(m, n, k)
    finally:
        comm.destroy()
