"""Argument-blob / resource-context API of the fused-operator interface, and the graph-mode entry points with their
resource queries, on the simulation backend.

Reference behaviour: src/common/hccl_mc2.cc:21-165 (setter validation, context creation is idempotent per
(operator, algorithm config)); src/ops/interface_graph_mode/calc_resource_graph_mode.cc:47-94 (offline / online resource
estimates and algorithm selection from an opaque parameter object); src/ops/all_reduce/all_reduce_op.cc:58-103 (graph-mode
entry addressed by group name and tag).
"""
import ctypes

import numpy as np
import pytest
import torch

from hccl_b200._lib import lib
from hccl_b200.types import DataType, Result
from hccl_b200.utils.sim import run_ranks

vp, u8, u32, u64 = ctypes.c_void_p, ctypes.c_uint8, ctypes.c_uint32, ctypes.c_uint64


class OpResCtx(ctypes.Structure):
    _fields_ = [("magic", u32), ("opType", u32), ("rank", u32), ("nranks", u32), ("srcDataType", u32), ("dstDataType", u32),
                ("reduceType", u32), ("commEngine", u32), ("count", u64), ("heapBytes", u64), ("heap", vp * 32), ("mcHeap", vp),
                ("workspaceOff", u64), ("workspaceBytes", u64), ("flagOff", u64), ("timeoutNs", u64), ("algConfig", ctypes.c_char * 128)]


class OpRes(ctypes.Structure):
    _fields_ = [("scratchBytes", u64), ("streamNum", u32), ("taskNum", u32), ("ctaNum", u32), ("algName", ctypes.c_char * 128), ("engine", u32)]


def _declare():
    l = lib()
    l.HcclKfcAllocOpArgs.argtypes = [ctypes.POINTER(vp)]
    l.HcclKfcFreeOpArgs.argtypes = [vp]
    l.HcclKfcOpArgsSetSrcDataType.argtypes = [vp, u8]
    l.HcclKfcOpArgsSetDstDataType.argtypes = [vp, u8]
    l.HcclKfcOpArgsSetReduceType.argtypes = [vp, u32]
    l.HcclKfcOpArgsSetCount.argtypes = [vp, u64]
    l.HcclKfcOpArgsSetAlgConfig.argtypes = [vp, ctypes.c_char_p]
    l.HcclKfcOpArgsSetCommEngine.argtypes = [vp, u8]
    l.HcclCreateOpResCtx.argtypes = [vp, u8, vp, ctypes.POINTER(vp)]
    for n in ("Create",):
        getattr(l, "HcclOpParamGraphMode" + n).argtypes = [ctypes.POINTER(vp)]
    l.HcclOpParamGraphModeDestroy.argtypes = [vp]
    l.HcclOpParamGraphModeSetOpType.argtypes = [vp, ctypes.c_int]
    l.HcclOpParamGraphModeSetDataCount.argtypes = [vp, u64]
    l.HcclOpParamGraphModeSetDataType.argtypes = [vp, ctypes.c_int]
    l.HcclOpParamGraphModeSetReduceOp.argtypes = [vp, ctypes.c_int]
    l.HcclOpParamGraphModeSetRoot.argtypes = [vp, u32]
    l.HcclOpParamGraphModeSetGroup.argtypes = [vp, ctypes.c_char_p]
    l.HcclCalcOpResOfflineGraphMode.argtypes = [vp, u32, ctypes.POINTER(OpRes)]
    l.HcclCalcOpResOnlineGraphMode.argtypes = [vp, vp, ctypes.POINTER(OpRes)]
    l.HcclSelectAlgGraphMode.argtypes = [vp, vp, ctypes.c_char_p, u32]
    tail = [ctypes.c_char_p, vp, ctypes.c_char_p, ctypes.POINTER(vp), u32, vp, u64]
    l.HcclAllReduceGraphMode.argtypes = [vp, vp, u64, ctypes.c_int, ctypes.c_int] + tail
    l.HcclAllGatherGraphMode.argtypes = [vp, vp, u64, ctypes.c_int] + tail
    l.HcclBroadcastGraphMode.argtypes = [vp, u64, ctypes.c_int, u32] + tail
    return l


def test_op_args_setters_validate():
    l = _declare()
    a = vp()
    assert l.HcclKfcAllocOpArgs(ctypes.byref(a)) == 0 and a.value
    assert l.HcclKfcOpArgsSetSrcDataType(a, int(DataType.BFP16)) == 0
    assert l.HcclKfcOpArgsSetDstDataType(a, int(DataType.FP32)) == 0
    assert l.HcclKfcOpArgsSetSrcDataType(a, 200) != 0
    assert l.HcclKfcOpArgsSetReduceType(a, 0) == 0 and l.HcclKfcOpArgsSetReduceType(a, 9) != 0
    assert l.HcclKfcOpArgsSetCount(a, 1 << 20) == 0
    assert l.HcclKfcOpArgsSetAlgConfig(a, b"AllGather=level0:fullmesh") == 0
    assert l.HcclKfcOpArgsSetAlgConfig(a, b"x" * 200) != 0                 # longer than the 128-character limit
    assert l.HcclKfcOpArgsSetAlgConfig(a, None) == Result.E_PTR
    assert l.HcclKfcOpArgsSetCommEngine(a, 3) == 0 and l.HcclKfcOpArgsSetCommEngine(a, 1) != 0   # only device engines
    assert l.HcclKfcOpArgsSetCount(None, 1) == Result.E_PTR
    junk = ctypes.create_string_buffer(256)
    assert l.HcclKfcOpArgsSetCount(ctypes.cast(junk, vp), 1) == Result.E_PTR   # not a blob made by the allocator
    assert l.HcclKfcFreeOpArgs(a) == 0


def test_resource_context_describes_the_symmetric_heap():
    l = _declare()

    def body(comm, rank):
        a = vp()
        l.HcclKfcAllocOpArgs(ctypes.byref(a))
        l.HcclKfcOpArgsSetSrcDataType(a, int(DataType.FP32))
        l.HcclKfcOpArgsSetDstDataType(a, int(DataType.FP32))
        l.HcclKfcOpArgsSetCount(a, 1000)
        l.HcclKfcOpArgsSetAlgConfig(a, b"mine")
        h = vp(comm.handle)
        ctx1, ctx2 = vp(), vp()
        assert l.HcclCreateOpResCtx(h, 6, a, ctypes.byref(ctx1)) == 0
        assert l.HcclCreateOpResCtx(h, 6, a, ctypes.byref(ctx2)) == 0
        assert ctx1.value == ctx2.value                                    # one context per (operator, algorithm config)
        assert l.HcclCreateOpResCtx(h, 0, a, ctypes.byref(ctx2)) == Result.E_PARA
        assert l.HcclCreateOpResCtx(h, 6, None, ctypes.byref(ctx2)) == Result.E_PTR
        l.HcclKfcOpArgsSetCommEngine(a, 4)
        assert l.HcclCreateOpResCtx(h, 6, a, ctypes.byref(ctx2)) == Result.E_UNAVAIL   # no multicast mapping on the host backend
        c = OpResCtx.from_address(ctx1.value)
        assert c.magic == 0x4332434D and c.rank == rank and c.nranks == comm.size and c.count == 1000
        assert c.workspaceBytes >= 1000 * 4 * comm.size + (64 << 10) and c.flagOff + (64 << 10) == c.workspaceOff + c.workspaceBytes
        # use it the way a custom kernel would: write my rank into every peer's window, then read what the peers wrote
        for r in range(comm.size):
            ctypes.c_uint32.from_address(c.heap[r] + c.workspaceOff + 4 * rank).value = 1000 + rank
        comm.barrier()
        comm.synchronize()
        got = [ctypes.c_uint32.from_address(c.heap[rank] + c.workspaceOff + 4 * r).value for r in range(comm.size)]
        flags_zero = all(ctypes.c_uint32.from_address(c.heap[rank] + c.flagOff + 4 * i).value == 0 for i in range(64))
        l.HcclKfcFreeOpArgs(a)
        return got, flags_zero

    for got, flags_zero in run_ranks(3, body):
        assert got == [1000, 1001, 1002] and flags_zero


def test_graph_mode_resource_queries_and_entry_points():
    l = _declare()
    p = vp()
    assert l.HcclOpParamGraphModeCreate(ctypes.byref(p)) == 0
    res = OpRes()
    assert l.HcclCalcOpResOfflineGraphMode(p, 8, ctypes.byref(res)) == Result.E_PARA      # no operator type set yet
    assert l.HcclOpParamGraphModeSetOpType(p, 2) == 0 and l.HcclOpParamGraphModeSetOpType(p, 0) == Result.E_PARA
    assert l.HcclOpParamGraphModeSetDataCount(p, 1 << 20) == 0
    assert l.HcclOpParamGraphModeSetDataType(p, 11) == 0 and l.HcclOpParamGraphModeSetDataType(p, 99) != 0
    assert l.HcclOpParamGraphModeSetReduceOp(p, 0) == 0
    assert l.HcclCalcOpResOfflineGraphMode(p, 8, ctypes.byref(res)) == 0
    assert res.taskNum >= 1 and res.ctaNum >= 1 and res.algName and res.engine in (3, 4) and res.scratchBytes > 0
    assert l.HcclCalcOpResOfflineGraphMode(p, 1, ctypes.byref(res)) == Result.E_PARA

    def body(comm, rank):
        h = vp(comm.handle)
        q = vp()
        l.HcclOpParamGraphModeCreate(ctypes.byref(q))
        l.HcclOpParamGraphModeSetOpType(q, 2)
        l.HcclOpParamGraphModeSetDataCount(q, 4096)
        l.HcclOpParamGraphModeSetDataType(q, 4)
        l.HcclOpParamGraphModeSetReduceOp(q, 0)
        name = comm.name.encode()
        assert l.HcclOpParamGraphModeSetGroup(q, name) == 0
        r1, r2 = OpRes(), OpRes()
        assert l.HcclCalcOpResOnlineGraphMode(h, q, ctypes.byref(r1)) == 0
        assert l.HcclCalcOpResOnlineGraphMode(None, q, ctypes.byref(r2)) == 0             # resolved through the group name
        alg = ctypes.create_string_buffer(128)
        assert l.HcclSelectAlgGraphMode(h, q, alg, 128) == 0
        assert r1.algName == r2.algName == alg.value and r1.engine == 1
        x = np.full(4096, rank + 1.0, np.float32)
        out = np.empty_like(x)
        assert l.HcclAllReduceGraphMode(x.ctypes.data, out.ctypes.data, 4096, 4, 0, name, None, b"step0_ar", None, 0, None, 0) == 0
        g = np.empty(4096 * comm.size, np.float32)
        assert l.HcclAllGatherGraphMode(x.ctypes.data, g.ctypes.data, 4096, 4, name, None, b"step0_ag", None, 0, None, 0) == 0
        b = x.copy()
        assert l.HcclBroadcastGraphMode(b.ctypes.data, 4096, 4, 1, name, None, b"step0_bc", None, 0, None, 0) == 0
        comm.synchronize()
        assert l.HcclAllReduceGraphMode(x.ctypes.data, out.ctypes.data, 4096, 4, 0, b"no_such_group", None, b"t", None, 0, None, 0) != 0
        assert l.HcclAllReduceGraphMode(x.ctypes.data, out.ctypes.data, 4096, 4, 0, name, None, None, None, 0, None, 0) == Result.E_PTR
        l.HcclOpParamGraphModeDestroy(q)
        return out[0], g[::4096].tolist(), b[0]

    for out, g, b in run_ranks(3, body):
        assert out == 6.0 and g == [1.0, 2.0, 3.0] and b == 2.0
    assert l.HcclOpParamGraphModeDestroy(p) == 0


def test_graph_mode_variable_count_entry_points():
    """AllGatherV / ReduceScatterV / AlltoAllV / AlltoAllVC through the graph-mode entries (group name, tag, helper streams and
    scratch in the tail), against numpy; and the argument checks that differ from the fixed-count forms."""
    l = _declare()
    tail = [ctypes.c_char_p, vp, ctypes.c_char_p, ctypes.POINTER(vp), u32, vp, u64]
    l.HcclAllGatherVGraphMode.argtypes = [vp, vp, u64, vp, vp, ctypes.c_int] + tail
    l.HcclReduceScatterVGraphMode.argtypes = [vp, vp, vp, vp, u64, ctypes.c_int, ctypes.c_int] + tail
    l.HcclAlltoAllVGraphMode.argtypes = [vp, vp, vp, ctypes.c_int, vp, vp, vp, ctypes.c_int] + tail
    l.HcclAlltoAllVCGraphMode.argtypes = [vp, vp, ctypes.c_int, vp, ctypes.c_int] + tail
    n = 3
    counts = np.array([5, 0, 1201], np.uint64)                      # per-rank block sizes of the gather / scatter forms
    displs = np.array([0, 5, 5], np.uint64)
    total = int(counts.sum())
    M = np.array([[2, 0, 7], [300, 1, 0], [4, 5, 6]], np.uint64)    # M[i][j]: elements rank i sends to rank j
    rng = np.random.default_rng(23)
    ag_in = [rng.standard_normal(int(counts[r])).astype(np.float32) for r in range(n)]
    rs_in = [rng.integers(-8, 9, size=total).astype(np.float32) for _ in range(n)]
    a2a_in = [rng.standard_normal(int(M[r].sum())).astype(np.float32) for r in range(n)]
    FP32, SUM = 4, 0

    def body(comm, rank):
        name = comm.name.encode()
        t = lambda tag: (name, None, tag, None, 0, None, 0)
        g = np.zeros(total, np.float32)
        x = ag_in[rank] if counts[rank] else np.zeros(1, np.float32)
        assert l.HcclAllGatherVGraphMode(x.ctypes.data, g.ctypes.data, int(counts[rank]), counts.ctypes.data, displs.ctypes.data, FP32, *t(b"agv")) == 0
        s = np.zeros(max(1, int(counts[rank])), np.float32)
        assert l.HcclReduceScatterVGraphMode(rs_in[rank].ctypes.data, counts.ctypes.data, displs.ctypes.data, s.ctypes.data, int(counts[rank]), FP32, SUM, *t(b"rsv")) == 0
        sc, rc = M[rank].copy(), M[:, rank].copy()
        sd = np.concatenate([[0], np.cumsum(sc)[:-1]]).astype(np.uint64)
        rd = np.concatenate([[0], np.cumsum(rc)[:-1]]).astype(np.uint64)
        o1 = np.zeros(int(rc.sum()), np.float32)
        assert l.HcclAlltoAllVGraphMode(a2a_in[rank].ctypes.data, sc.ctypes.data, sd.ctypes.data, FP32, o1.ctypes.data, rc.ctypes.data, rd.ctypes.data, FP32, *t(b"a2av")) == 0
        o2 = np.zeros(int(rc.sum()), np.float32)
        assert l.HcclAlltoAllVCGraphMode(a2a_in[rank].ctypes.data, M.ctypes.data, FP32, o2.ctypes.data, FP32, *t(b"a2avc")) == 0
        comm.synchronize()
        # argument checks: own count must agree with the array; a product reduction is refused; element sizes must agree
        assert l.HcclAllGatherVGraphMode(x.ctypes.data, g.ctypes.data, int(counts[rank]) + 1, counts.ctypes.data, displs.ctypes.data, FP32, *t(b"bad")) == Result.E_PARA
        assert l.HcclReduceScatterVGraphMode(rs_in[rank].ctypes.data, counts.ctypes.data, displs.ctypes.data, s.ctypes.data, int(counts[rank]), FP32, 1, *t(b"bad")) == Result.E_NOT_SUPPORT
        assert l.HcclAlltoAllVCGraphMode(a2a_in[rank].ctypes.data, M.ctypes.data, FP32, o2.ctypes.data, 3, *t(b"bad")) == Result.E_PARA      # fp16 on the receive side
        assert l.HcclAlltoAllVGraphMode(a2a_in[rank].ctypes.data, None, sd.ctypes.data, FP32, o1.ctypes.data, rc.ctypes.data, rd.ctypes.data, FP32, *t(b"bad")) == Result.E_PTR
        assert l.HcclAllGatherVGraphMode(x.ctypes.data, g.ctypes.data, int(counts[rank]), counts.ctypes.data, displs.ctypes.data, FP32,
                                         b"no_such_group", None, b"t", None, 0, None, 0) != 0
        return g, s[:int(counts[rank])], o1, o2

    res = run_ranks(n, body)
    want_g = np.concatenate(ag_in)
    want_rs = np.sum(np.stack(rs_in).astype(np.float64), axis=0)
    for rank, (g, s, o1, o2) in enumerate(res):
        assert np.array_equal(g, want_g)
        lo = int(displs[rank])
        assert np.array_equal(s.astype(np.float64), want_rs[lo:lo + int(counts[rank])])
        want = np.concatenate([a2a_in[src][int(M[src, :rank].sum()):int(M[src, :rank + 1].sum())] for src in range(n)])
        assert np.array_equal(o1, want) and np.array_equal(o2, want)


def test_misaligned_results_and_scales_are_refused_before_any_launch():
    """The kernel for few rows stores four results at a time and copies block scales in 16-byte pieces: an address that does not allow it
    is a parameter error on the host. The pointers are never read here."""
    l = lib()
    l.HcclGemmBf16.argtypes = [vp, vp, vp, u64, u64, u64, ctypes.c_int, vp]
    l.HcclGemmMxfp8.argtypes = [vp, vp, vp, vp, vp, u64, u64, u64, ctypes.c_int, vp]
    l.HcclGemmMxfp8Variant.argtypes = [vp, vp, vp, vp, vp, u64, u64, u64, ctypes.c_int, ctypes.c_int, vp]
    base = 1 << 20
    para = int(Result.E_PARA)
    for fp32 in (0, 1):
        for off in (2, 4, 8):
            assert l.HcclGemmBf16(base, base, base + off, 4, 4096, 4096, fp32, None) == para
            assert l.HcclGemmMxfp8(base, base, base, base, base + off, 4, 4096, 4096, fp32, None) == para
    for off in (1, 4, 8):
        assert l.HcclGemmMxfp8(base, base + off, base, base, base, 4, 4096, 4096, 0, None) == para
        assert l.HcclGemmMxfp8Variant(base, base, base, base + off, base, 4, 4096, 4096, 0, 128, None) == para


@pytest.mark.parametrize("native", [True, False])
def test_fused_operators_check_shapes_and_results_on_the_host(native, monkeypatch):
    """An operand or result that does not hold what the kernel reads or writes is an error before anything is launched, in the extension and
    in the ctypes form (CPU tensors: a call that passed the checks of shape and type is refused for its device)."""
    from types import SimpleNamespace

    from hccl_b200.ops import gemm, mc2

    if not native:
        monkeypatch.setattr(mc2, "_native", lambda: None)
    elif mc2._native() is None:
        pytest.skip("the extension is not built")
    comm = SimpleNamespace(handle=0, size=2)
    e = lambda *s, dt=torch.bfloat16: torch.empty(*s, dtype=dt)
    a, w = e(8, 16), e(24, 16)
    calls = {"agmm": (mc2.all_gather_matmul, 16), "mmrs": (mc2.matmul_reduce_scatter, 4), "mmar": (mc2.matmul_all_reduce, 8)}
    for fn, rows in calls.values():
        for bad in (e(24, 8), e(24), e(24, 17)):
            with pytest.raises(ValueError, match="matrices"):
                fn(comm, a, bad)
        with pytest.raises(ValueError, match="matrices"):
            fn(comm, e(8, 2, 8), w)
        for out in (e(rows, 23), e(rows * 24 - 1), e(rows, 24, dt=torch.float32), e(24, rows).t()):
            with pytest.raises(ValueError, match="out must be a contiguous"):
                fn(comm, a, w, out=out)
        with pytest.raises(ValueError, match="out must be a CUDA"):
            fn(comm, a, w, out=e(rows + 1, 24))
        for good in (w, e(24, 4, 4)):
            with pytest.raises(ValueError, match="contiguous bf16 CUDA"):
                fn(comm, a, good)
    for gathered in (e(15, 16), e(16, 16, dt=torch.float32)):
        with pytest.raises(ValueError, match="gathered must be"):
            mc2.all_gather_matmul(comm, a, w, gathered=gathered)
    if native:
        ext = mc2._native()
        for out in (e(8, 23), e(8, 24, dt=torch.float16), e(24, 8).t()):
            with pytest.raises(ValueError, match="out must be a contiguous"):
                ext.gemm(a, w, out, False, False, 0, None)
    else:
        with pytest.raises(ValueError, match="bf16 or fp32"):
            gemm.check_result(e(8, 23), 8 * 24, (torch.bfloat16, torch.float32))


def test_block_scaled_and_moe_calls_check_their_memory_on_the_host():
    """What the kernels read or write at an address has to be there: sizes, types and devices are errors before anything is launched (CPU tensors, as above)."""
    from hccl_b200.ops import mxfp8

    ext = mxfp8._native()
    if ext is None:
        pytest.skip("the extension is not built")
    e = lambda *s, dt=torch.bfloat16: torch.empty(*s, dtype=dt)
    byte = lambda *s: e(*s, dt=torch.uint8)
    rows, n, k = 5, 24, 256
    x, payload, scales = e(rows, k), byte(n, k), byte(mxfp8.scale_bytes(n, k))
    for bad, match in (((e(rows, k, 1), payload, scales), "activations"), ((e(k, rows).t(), payload, scales), "activations"), ((e(rows, k, dt=torch.float16), payload, scales), "activations"),
                       ((x, byte(n, k - 1), scales), "payload"), ((x, byte(k, n).t(), scales), "payload"), ((x, payload, scales[:-1]), "scales"),
                       ((e(rows, 2 * k), payload, scales), "payload")):
        with pytest.raises(ValueError, match=match):
            ext.mx_matmul(0, *bad, n, None, None)
    for out in (e(rows, n - 1), e(rows, n, dt=torch.float32), e(n, rows).t()):
        with pytest.raises(ValueError, match="out must be a contiguous"):
            ext.mx_matmul(0, x, payload, scales, n, out, None)
    with pytest.raises(ValueError, match="CUDA"):
        ext.mx_matmul(0, x, payload, scales, n, None, None)
    good = byte(rows, k), byte(mxfp8.scale_bytes(rows, k))
    for bad, match in (((byte(rows, k - 1), good[1]), "payload"), ((good[0], good[1][:-1]), "scales"), ((byte(k, rows).t(), good[1]), "payload"), (good, "CUDA")):
        with pytest.raises(ValueError, match=match):
            ext.mx_quantize(x, *bad, None)
        with pytest.raises(ValueError):
            mxfp8._need(mxfp8.MxTensor(*bad, rows, k), rows, k)
    tokens, hidden, top_k = 6, 256, 2
    xs, idx, weights = e(tokens, hidden), e(tokens, top_k, dt=torch.int32), e(tokens, top_k, dt=torch.float32)
    for bad, match in (((e(tokens, hidden - 1), idx), "x must"), ((xs, idx[:, :1].contiguous()), "topk_idx"), ((xs, idx[:-1]), "topk_idx"), ((xs, idx), "CUDA")):
        with pytest.raises(ValueError, match=match):
            ext.moe_dispatch(0, top_k, hidden, *bad, None, (), ())
    for bad, match in (((weights[:-1], None), "topk_weights"), ((weights, e(tokens, hidden - 1)), "out"), ((weights, e(tokens, hidden, dt=torch.float32)), "out"), ((weights, None), "CUDA")):
        with pytest.raises(ValueError, match=match):
            ext.moe_combine(0, top_k, bad[0], tokens, hidden, bad[1], None)
