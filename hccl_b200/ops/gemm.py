"""tcgen05 GEMM (sm_100a): `gemm_bf16(a, w)` = a @ w.T with bf16 operands and fp32 accumulation in tensor memory."""
from __future__ import annotations

import ctypes

import torch

from .._ext import ops as _native
from .._lib import check, lib


def _decl():
    l = lib()
    if not getattr(l, "_gemm_declared", False):
        l.HcclGemmBf16.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_uint64,
                                   ctypes.c_int, ctypes.c_void_p]
        l.HcclGemmBf16.restype = ctypes.c_int
        l.HcclGemmBf16Variant.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_uint64,
                                          ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
        l.HcclGemmBf16Variant.restype = ctypes.c_int
        l.HcclGemmBf16Nn.argtypes = l.HcclGemmBf16.argtypes
        l.HcclGemmBf16Nn.restype = ctypes.c_int
        l.HcclGemmCheckError.argtypes = []
        l.HcclGemmCheckError.restype = ctypes.c_int
        l._gemm_declared = True
    return l


def check_result(t: torch.Tensor, elems: int, dtypes, what: str = "out") -> None:
    """`elems` results are written at the tensor's address: it has to be that large, dense and of a type the kernels write."""
    if not t.is_contiguous() or t.numel() < elems or t.dtype not in dtypes:
        raise ValueError(f"{what} must be a contiguous tensor of at least {elems} {' or '.join('fp32' if d is torch.float32 else 'bf16' for d in dtypes)} elements")
    if not t.is_cuda:
        raise ValueError(f"{what} must be a CUDA tensor")


def gemm_bf16(a: torch.Tensor, w: torch.Tensor, out: torch.Tensor | None = None, out_dtype: torch.dtype = torch.bfloat16,
              stream=None, variant: int = 0) -> torch.Tensor:
    """a: [M, K] bf16, w: [N, K] bf16 (both row-major) -> [M, N] in `out_dtype` (bf16 or fp32).
    variant: 0 automatic, 2 CTA-pair (cta_group::2) 256 x 256 tiles, 192 / 224 and 288 ... 512 in steps of 32 pair tiles of that width, 1000 * S + BT split-K with BT rows of
    a per tile and S CTAs along K."""
    if not (a.is_cuda and w.is_cuda):
        raise RuntimeError("gemm_bf16 needs CUDA tensors (the tcgen05 kernel has no CPU path)")
    assert a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and a.is_contiguous() and w.is_contiguous()
    M, K = a.shape
    N, K2 = w.shape
    assert K == K2
    n = _native()
    if n is not None and (out is not None or out_dtype in (torch.bfloat16, torch.float32)):
        rc, out = n.gemm(a, w, out, out_dtype == torch.float32, False, variant, None if stream is None else stream.cuda_stream)
        if rc:
            check(rc, "HcclGemmBf16")
        return out
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype, device=a.device)
    check_result(out, M * N, (torch.bfloat16, torch.float32))
    s = torch.cuda.current_stream() if stream is None else stream
    check(_decl().HcclGemmBf16Variant(a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, int(out.dtype == torch.float32), variant, s.cuda_stream),
          "HcclGemmBf16")
    return out


def gemm_bf16_nn(a: torch.Tensor, w: torch.Tensor, out: torch.Tensor | None = None, out_dtype: torch.dtype = torch.bfloat16, stream=None) -> torch.Tensor:
    """a: [M, K] bf16, w: [K, N] bf16 (both row-major) -> a @ w in `out_dtype` (bf16 or fp32); no transposed copy of w is made."""
    if not (a.is_cuda and w.is_cuda):
        raise RuntimeError("gemm_bf16_nn needs CUDA tensors (the tcgen05 kernel has no CPU path)")
    assert a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and a.is_contiguous() and w.is_contiguous()
    M, K = a.shape
    K2, N = w.shape
    assert K == K2
    n = _native()
    if n is not None and (out is not None or out_dtype in (torch.bfloat16, torch.float32)):
        rc, out = n.gemm(a, w, out, out_dtype == torch.float32, True, 0, None if stream is None else stream.cuda_stream)
        if rc:
            check(rc, "HcclGemmBf16Nn")
        return out
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype, device=a.device)
    check_result(out, M * N, (torch.bfloat16, torch.float32))
    s = torch.cuda.current_stream() if stream is None else stream
    check(_decl().HcclGemmBf16Nn(a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, int(out.dtype == torch.float32), s.cuda_stream), "HcclGemmBf16Nn")
    return out


def check_error() -> None:
    check(_decl().HcclGemmCheckError(), "HcclGemmCheckError")
