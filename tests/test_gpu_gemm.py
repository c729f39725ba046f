"""tcgen05 GEMM against a plain PyTorch fp32 reference of the same product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(128, 256, 64), (128, 256, 512), (256, 512, 1024), (384, 768, 200 * 8), (1000, 264, 520),
                                   (128, 8192, 1024), (2048, 3584, 2048), (64, 64, 64)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_matches_fp32_reference(shape, out_dtype):
    from hccl_b200.ops import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    a = torch.randn(M, K, generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32) * 0.05).to(torch.bfloat16)
    out = gemm.gemm_bf16(a, w, out_dtype=out_dtype)
    torch.cuda.synchronize()
    gemm.check_error()
    ref = a.float() @ w.float().t()
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    tol = 2e-2 if out_dtype == torch.bfloat16 else 2e-3
    assert err / scale < tol, f"max err {err} vs scale {scale}"


def test_gemm_back_to_back_is_deterministic():
    from hccl_b200.ops import gemm
    a = torch.randn(512, 1024, device="cuda").to(torch.bfloat16)
    w = torch.randn(1024, 1024, device="cuda").to(torch.bfloat16)
    o1 = gemm.gemm_bf16(a, w)
    o2 = gemm.gemm_bf16(a, w)
    torch.cuda.synchronize()
    assert torch.equal(o1, o2)


@pytest.mark.parametrize("shape", [(256, 256, 64), (256, 512, 512), (512, 768, 1024), (384, 520, 328), (1000, 264, 520), (2048, 3584, 2048),
                                   (100, 256, 128)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_cta_pair_variant(shape, out_dtype):
    """256 x 256 tiles on CTA pairs (tcgen05 cta_group::2): odd row-block counts, ragged N and K tails included."""
    from hccl_b200.ops import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M * 5 + N * 11 + K)
    a = torch.randn(M, K, generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32) * 0.05).to(torch.bfloat16)
    out = gemm.gemm_bf16(a, w, out_dtype=out_dtype, variant=2)
    torch.cuda.synchronize()
    gemm.check_error()
    ref = a.float() @ w.float().t()
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    tol = 2e-2 if out_dtype == torch.bfloat16 else 2e-3
    assert err / scale < tol, f"max err {err} vs scale {scale}"


@pytest.mark.parametrize("shape,bt,split", [((1, 8, 8), 16, 1), ((4, 4096, 520), 16, 8), ((16, 136, 448), 16, 7), ((17, 264, 1032), 32, 5), ((33, 1000, 512), 64, 8),
                                            ((128, 128, 4096), 128, 8), ((100, 72, 200), 128, 3), ((129, 520, 328), 64, 2), ((257, 384, 1024), 256, 4),
                                            ((300, 256, 640), 128, 6), ((64, 8192, 64), 64, 1)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_split_k(shape, bt, split, out_dtype):
    """Rows of A on the narrow side of the instruction, K shared by a cluster: remainders of every tile edge, one k-block per CTA, one row,
    uneven K parts. The reference is a 64-bit product; 32-bit sums of K products err by less than K * 2^-24 of the absolute sum."""
    from hccl_b200.ops import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N * 3 + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M + 1, N), 7.0, device="cuda", dtype=out_dtype)                # a row past the end must stay
    gemm.gemm_bf16(a, w, out[:M], variant=1000 * split + bt)
    torch.cuda.synchronize()
    gemm.check_error()
    ref, mag = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    bound = mag * K * 2.0 ** -24 + (ref.abs() * 2.0 ** -8 if out_dtype == torch.bfloat16 else 0)
    assert bool(((out[:M].double() - ref).abs() <= bound + 1e-30).all())
    assert bool((out[M] == 7.0).all())


@pytest.mark.parametrize("shape,split", [((192, 128, 512), 1), ((193, 264, 520), 2), ((384, 136, 4104), 4), ((577, 520, 2048), 8), ((1, 8, 64), 1), ((384, 4096, 4608), 0), ((300, 2528, 4512), 0)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_split_k_of_192_rows(shape, split, out_dtype):
    """192 rows of A per tile: whole tiles, one row more, one row, uneven K parts, and (0) where the choice takes it."""
    test_gemm_split_k(shape, 192 if split else 0, split, out_dtype)


@pytest.mark.parametrize("shape", [(65, 4088, 5128), (128, 8200, 5000), (129, 1744, 5240), (200, 520, 2048), (257, 3704, 5128), (512, 1448, 5128), (512, 2824, 2048), (300, 5408, 2056)])
def test_gemm_split_k_of_65_to_512_rows(shape):
    """Products that the automatic choice sends to 64-, 128- and 256-row split-K tiles, and the first beyond its lines (bound as above)."""
    from hccl_b200.ops import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N * 3 + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M + 1, N), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm.gemm_bf16(a, w, out[:M])
    torch.cuda.synchronize()
    gemm.check_error()
    ref, mag = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    assert bool(((out[:M].double() - ref).abs() <= mag * K * 2.0 ** -24 + ref.abs() * 2.0 ** -8 + 1e-30).all())
    assert bool((out[M] == 7.0).all())


@pytest.mark.parametrize("shape", [(1, 8, 8), (128, 64, 64), (100, 72, 200), (1000, 264, 520), (384, 768, 1600), (2048, 4104, 1032), (4096, 2560, 264)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_nn(shape, out_dtype):
    """B stored [K, N] and read MN-major: all three tile kernels, ragged edges in every dimension (bound as above)."""
    from hccl_b200.ops import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N * 3 + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(K, N, generator=g, device="cuda").to(torch.bfloat16)
    out = gemm.gemm_bf16_nn(a, w, out_dtype=out_dtype)
    torch.cuda.synchronize()
    gemm.check_error()
    ref, mag = a.double() @ w.double(), a.double().abs() @ w.double().abs()
    bound = mag * K * 2.0 ** -24 + (ref.abs() * 2.0 ** -8 if out_dtype == torch.bfloat16 else 0)
    assert bool(((out.double() - ref).abs() <= bound + 1e-30).all())


@pytest.mark.parametrize("shape,variant", [((256, 192, 64), 192), ((1000, 200, 264), 192), ((300, 392, 128), 224), ((1000, 6144, 512), 0), ((2048, 14336, 256), 0),
                                           ((1500, 3000, 520), 0)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_pair_tile_widths(shape, variant, out_dtype):
    """Pair tiles of 192 and 224 columns (the last staging tile of a 224-wide one stores 32 columns twice), one tile and partial tiles, and
    shapes for which the automatic choice picks them (bound as above)."""
    from hccl_b200.ops import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N * 3 + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M + 1, N), 7.0, device="cuda", dtype=out_dtype)
    gemm.gemm_bf16(a, w, out[:M], variant=variant)
    torch.cuda.synchronize()
    gemm.check_error()
    ref, mag = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    bound = mag * K * 2.0 ** -24 + (ref.abs() * 2.0 ** -8 if out_dtype == torch.bfloat16 else 0)
    assert bool(((out[:M].double() - ref).abs() <= bound + 1e-30).all())
    assert bool((out[M] == 7.0).all())


@pytest.mark.parametrize("shape,variant", [((256, 288, 64), 288), ((8, 8, 8), 512), ((257, 520, 200), 320), ((1000, 6144, 264), 352), ((300, 1000, 136), 416), ((520, 448, 328), 448),
                                           ((700, 3000, 1032), 480), ((2048, 5120, 320), 512), ((2115, 2304, 2344), 0), ((1000, 6144, 4096), 0)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_wide_tiles(shape, variant, out_dtype):
    """Pair tiles of two halves: unequal halves, one k-block and fewer k-blocks than half 0 runs ahead, a second half past the edge, several tiles per
    pair, and shapes for which the automatic choice picks them (bound as above)."""
    from hccl_b200.ops import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N * 3 + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M + 1, N), 7.0, device="cuda", dtype=out_dtype)
    gemm.gemm_bf16(a, w, out[:M], variant=variant)
    torch.cuda.synchronize()
    gemm.check_error()
    ref, mag = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    bound = mag * K * 2.0 ** -24 + (ref.abs() * 2.0 ** -8 if out_dtype == torch.bfloat16 else 0)
    assert bool(((out[:M].double() - ref).abs() <= bound + 1e-30).all())
    assert bool((out[M] == 7.0).all())


@pytest.mark.parametrize("shape", [(2000, 4096, 14344), (4096, 4096, 8200)])
def test_gemm_nn_wide_tiles(shape):
    """B stored [K, N] in 512-wide pair tiles, where the automatic choice takes them; one and two waves (bound as above)."""
    from hccl_b200.ops import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N * 3 + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(K, N, generator=g, device="cuda").to(torch.bfloat16)
    out = gemm.gemm_bf16_nn(a, w)
    torch.cuda.synchronize()
    gemm.check_error()
    ref, mag = a.double() @ w.double(), a.double().abs() @ w.double().abs()
    assert bool(((out.double() - ref).abs() <= mag * K * 2.0 ** -24 + ref.abs() * 2.0 ** -8 + 1e-30).all())


@pytest.mark.parametrize("pairs", ["", "0"])
def test_pairs_can_be_switched_off(pairs):
    """HCCL_GEMM_2CTA=0 keeps both operand layouts off the CTA-pair kernels (the variable is read once per process)."""
    import os
    import subprocess
    import sys
    from pathlib import Path
    prog = """
import torch
from torch.profiler import ProfilerActivity, profile
from hccl_b200.ops import gemm
for fn, shape in ((gemm.gemm_bf16, (4096, 512)), (gemm.gemm_bf16_nn, (512, 4096))):
    a, w = (torch.ones(s, device="cuda", dtype=torch.bfloat16) for s in ((8192, 512), shape))
    fn(a, w)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        out = fn(a, w)
        torch.cuda.synchronize()
    assert bool((out == 512).all())
    print("KERNELS", [e.key for e in p.key_averages() if "Gemm" in e.key])
"""
    env = dict(os.environ, HCCL_GEMM_2CTA=pairs) if pairs else {k: v for k, v in os.environ.items() if k != "HCCL_GEMM_2CTA"}
    res = subprocess.run([sys.executable, "-c", prog], cwd=Path(__file__).resolve().parents[1], env=env, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    lines = [l for l in res.stdout.splitlines() if l.startswith("KERNELS")]
    assert len(lines) == 2 and all(("2Cta" in l) == (pairs != "0") and "GemmKernel" in l for l in lines), lines


@pytest.mark.parametrize("m,variant", [(4, 0), (64, 0), (128, 0), (100, 2064), (1000, 0), (300, 2), (600, 192)])
def test_chained_products_wait_for_one_another(m, variant):
    """Products set up while the kernel before them drains. In a chain each reads the one before and writes the buffer that the one before
    has read; the bits are those of the same chain with a synchronisation after every product, also from a captured graph."""
    from hccl_b200.ops import gemm, mxfp8
    H = 2048
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, H, generator=g, device="cuda").to(torch.bfloat16)
    ws = [(torch.randn(H, H, generator=g, device="cuda") * H ** -0.5).to(torch.bfloat16) for _ in range(3)]
    wq = mxfp8.quantize(ws[2])
    bufs = [torch.empty_like(x), torch.empty_like(x)]

    def chain(sync):
        bufs[0].copy_(x)
        for step in range(12):
            src, dst = bufs[step % 2], bufs[1 - step % 2]
            if step % 4 == 3:
                mxfp8.gemm(src, wq, out=dst)
            elif step % 4 == 1:
                gemm.gemm_bf16_nn(src, ws[1], out=dst)
            else:
                gemm.gemm_bf16(src, ws[0], out=dst, variant=variant)
            if sync:
                torch.cuda.synchronize()
        return bufs[0].clone()

    ref = chain(True)
    assert torch.isfinite(ref.float()).all() and ref.float().abs().max() > 0.1
    for _ in range(5):
        assert torch.equal(chain(False), ref)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        chain(False)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            out = chain(False)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
    gemm.check_error()


@pytest.mark.parametrize("M", [16, 1000])
def test_products_without_the_extension(M, monkeypatch):
    """The ctypes form of the operators (another library chosen, or the extension not built) gives the same bits."""
    from hccl_b200.comm import Communicator, get_root_info
    from hccl_b200.ops import gemm, mc2
    a, w = torch.randn(M, 2048, device="cuda").to(torch.bfloat16), torch.randn(520, 2048, device="cuda").to(torch.bfloat16)
    comm = Communicator.from_root_info(1, get_root_info(), 0)
    try:
        def run():
            gathered = torch.empty_like(a)
            outs = [gemm.gemm_bf16(a, w), gemm.gemm_bf16(a, w, out_dtype=torch.float32), gemm.gemm_bf16_nn(a, w.t().contiguous()),
                    mc2.all_gather_matmul(comm, a, w, gathered=gathered), mc2.matmul_reduce_scatter(comm, a, w), mc2.matmul_all_reduce(comm, a, w)]
            torch.cuda.synchronize()
            return outs + [gathered]

        first = run()
        for module in (gemm, mc2):
            monkeypatch.setattr(module, "_native", lambda: None)
        for x, y in zip(first, run()):
            assert x.dtype == y.dtype and torch.equal(x, y)
    finally:
        comm.destroy()


@pytest.mark.parametrize("M", [16, 1000])
def test_products_as_the_first_call_of_a_thread(M):
    """A product may be the first CUDA call of its thread (autograd's worker thread starts its backward pass with one when the allocator
    has memory at hand): there is no current context yet when the tensor maps are encoded."""
    import threading

    from hccl_b200.ops import gemm, mxfp8
    a, w = torch.randn(M, 2048, device="cuda").to(torch.bfloat16), torch.randn(512, 2048, device="cuda").to(torch.bfloat16)
    wt, qa, qw = w.t().contiguous(), mxfp8.quantize(a), mxfp8.quantize(w)
    calls = [lambda o: gemm.gemm_bf16(a, w, out=o), lambda o: gemm.gemm_bf16_nn(a, wt, out=o), lambda o: gemm.gemm_bf16(a, w, out=o, variant=2),
             lambda o: mxfp8.gemm(qa, qw, out=o), lambda o: mxfp8.gemm(qa, qw, out=o, tile_n=2192)]
    for call in calls:
        ref, out, failed = torch.empty(M, 512, device="cuda", dtype=torch.bfloat16), torch.zeros(M, 512, device="cuda", dtype=torch.bfloat16), []
        call(ref)
        torch.cuda.synchronize()

        def run():
            try:
                call(out)
            except Exception as e:
                failed.append(e)

        t = threading.Thread(target=run)
        t.start()
        t.join()
        torch.cuda.synchronize()
        assert not failed, failed
        assert torch.equal(out, ref)


@pytest.mark.parametrize("shape", [(1, 8, 512), (4, 4096, 1032), (16, 264, 16384), (20, 136, 2056), (64, 1000, 520), (94, 312, 4104), (200, 520, 4104), (300, 392, 8192), (384, 4096, 4608), (548, 2528, 4096)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_nn_split_k(shape, out_dtype):
    """B stored [K, N] read by clusters that share K: every tile height, ragged rows, columns and K. Bound as in test_gemm_split_k."""
    from hccl_b200.ops import gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N * 3 + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(K, N, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M + 1, N), 7.0, device="cuda", dtype=out_dtype)
    gemm.gemm_bf16_nn(a, w, out[:M])
    torch.cuda.synchronize()
    gemm.check_error()
    ref, mag = a.double() @ w.double(), a.double().abs() @ w.double().abs()
    bound = mag * K * 2.0 ** -24 + (ref.abs() * 2.0 ** -8 if out_dtype == torch.bfloat16 else 0)
    assert bool(((out[:M].double() - ref).abs() <= bound + 1e-30).all())
    assert bool((out[M] == 7.0).all())
