"""bf16 GEMM on the tcgen05 tile engine (``csrc/gemm``), with a torch fallback for CPU runs.

Three layouts cover a linear layer without transposed copies:

* :func:`mm_nt`  ``y[M,N] = x[M,K] @ w[N,K]^T``      forward
* :func:`mm_nn`  ``dx[M,K] = dy[M,N] @ w[N,K]``       input gradient
* :func:`mm_tn`  ``dw[N,K] = dy[T,N]^T @ x[T,K]``     weight gradient (optionally accumulated in fp32)

and the grouped variants (:func:`grouped_mm_nt`, :func:`grouped_mm_nn`, :func:`grouped_mm_tn`) run every
expert of an MoE layer in one persistent launch with device-resident group offsets.
"""
from __future__ import annotations

import ctypes
from typing import Optional

import torch

from . import _lib

DENSE, GROUPED_M, GROUPED_K = 0, 1, 2
_c_ll = ctypes.c_longlong
_c_int = ctypes.c_int


def _use_cuda(*ts) -> bool:
    return all(t is None or t.is_cuda for t in ts) and ts[0].dtype == torch.bfloat16 and _lib.available()


_RESULT_TYPES = (None, torch.bfloat16, torch.float32)


def _native(a, b, bias, out_dtype):
    """The module that forms the product in one call, where the kernels cover the operands."""
    if a.is_cuda and a.dtype == torch.bfloat16 and b.is_cuda and out_dtype in _RESULT_TYPES \
            and (bias is None or bias.is_cuda):
        return _lib.native_if_enabled()
    return None


_entry = None


def _gemm_entry():
    """The C entry point with its argument types declared once: plain integers then pass through, where wrapping each of
    the 28 arguments of every call was a large part of a small GEMM's time on the host."""
    global _entry
    if _entry is None:
        f = _lib.lib().mcb_gemm_bf16
        p, ll, i, fl = ctypes.c_void_p, _c_ll, _c_int, ctypes.c_float
        f.argtypes = [p, ll, ll, ll, i, p, ll, ll, ll, i, p, ll, ll, i, i, i, i, i, fl, p, i, i, p, i, p, i, i, p]
        _entry = f
    return _entry


def _launch(a, a_inner, a_outer, lda, a_mn, b, b_inner, b_outer, ldb, b_mn, c, ldc, c_group_stride, M, N, K, alpha,
            bias, accumulate, mode=DENSE, num_groups=0, offsets=None, b_group_rows=0, max_sms=0, force_bn=0):
    rc = _gemm_entry()(
        a.data_ptr(), a_inner, a_outer, lda, int(a_mn), b.data_ptr(), b_inner, b_outer, ldb, int(b_mn),
        c.data_ptr(), ldc, c_group_stride, int(c.dtype == torch.float32), int(accumulate), M, N, K, alpha,
        None if bias is None else bias.data_ptr(), mode, num_groups, None if offsets is None else offsets.data_ptr(),
        b_group_rows, _lib.status_word(a.device).data_ptr(), max_sms, force_bn, _lib.stream_ptr())
    _lib.check_rc(rc, 'mcb_gemm_bf16')


def _lib_mm(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """``a @ b`` for the paths without the in-tree kernels, returned in fp32.  On the CPU (the oracle of the tests) the
    product is formed in fp32; on a GPU with the kernels switched off it is the library's GEMM in the operands' own
    dtype (bf16 inputs, fp32 accumulation), which is what a stack built on cuBLAS would run."""
    if a.is_cuda and a.dtype == b.dtype and a.dtype in (torch.bfloat16, torch.float16):
        return torch.matmul(a, b).float()
    return torch.matmul(a.float(), b.float())


def _row_major_2d(t: torch.Tensor) -> torch.Tensor:
    """Returns a 2-D view whose last dim is contiguous and whose row stride is TMA-compatible."""
    if t.dim() != 2:
        t = t.reshape(-1, t.shape[-1])
    if t.stride(1) != 1 or t.stride(0) % 8 != 0 or t.data_ptr() % 16 != 0:
        t = t.contiguous()
    return t


def _out(out, shape, dtype, device, accumulate):
    if out is None:
        assert not accumulate, 'accumulate needs an output tensor'
        return torch.empty(shape, dtype=dtype, device=device)
    assert tuple(out.shape) == tuple(shape) and out.stride(-1) == 1, (out.shape, shape, out.stride())
    return out


def _deliver(y, x, out, accumulate):
    """The 2-D result ``y`` of a product with ``x [..., K]``: into ``out`` where that is given."""
    if out is None:
        return y if x.dim() == 2 else y.view(*x.shape[:-1], y.shape[-1])
    if accumulate:
        out.add_(y.view(out.shape))
    else:
        out.copy_(y.view(out.shape))
    return out


def mm_nt(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None,
          out_dtype: Optional[torch.dtype] = None, accumulate: bool = False, alpha: float = 1.0,
          max_sms: int = 0, force_bn: int = 0) -> torch.Tensor:
    """``x[..., K] @ w[N, K]^T (+ bias)``."""
    nat = _native(x, w, bias, out_dtype)
    if nat is not None:
        y = nat.mm(0, x, w, bias, out, out_dtype == torch.float32, accumulate, alpha, max_sms, force_bn)
        if out is not None:
            return out
        return y if x.dim() == 2 else y.view(*x.shape[:-1], w.shape[0])   # no alias for the common case
    K = x.shape[-1]
    assert w.shape[1] == K
    y = _lib_mm(x.reshape(-1, K), w.t()) * alpha
    if bias is not None:
        y = y + bias.float()
    return _deliver(y.to(out_dtype or x.dtype), x, out, accumulate)


def mm_nn(dy: torch.Tensor, w: torch.Tensor, out: Optional[torch.Tensor] = None,
          out_dtype: Optional[torch.dtype] = None, accumulate: bool = False, alpha: float = 1.0,
          max_sms: int = 0, force_bn: int = 0) -> torch.Tensor:
    """``dy[..., N] @ w[N, K]`` -> ``[..., K]``."""
    nat = _native(dy, w, None, out_dtype)
    if nat is not None:
        y = nat.mm(1, dy, w, None, out, out_dtype == torch.float32, accumulate, alpha, max_sms, force_bn)
        if out is not None:
            return out
        return y if dy.dim() == 2 else y.view(*dy.shape[:-1], w.shape[1])
    N = dy.shape[-1]
    assert w.shape[0] == N
    y = (_lib_mm(dy.reshape(-1, N), w) * alpha).to(out_dtype or dy.dtype)
    return _deliver(y, dy, out, accumulate)


def mm_tn(dy: torch.Tensor, x: torch.Tensor, out: Optional[torch.Tensor] = None,
          out_dtype: Optional[torch.dtype] = None, accumulate: bool = False, alpha: float = 1.0,
          max_sms: int = 0, force_bn: int = 0) -> torch.Tensor:
    """``dy[T, N]^T @ x[T, K]`` -> ``[N, K]`` (weight gradient)."""
    nat = _native(dy, x, None, out_dtype)
    if nat is not None:
        return nat.mm(2, dy, x, None, out, out_dtype == torch.float32, accumulate, alpha, max_sms, force_bn)
    y = _lib_mm(dy.reshape(-1, dy.shape[-1]).t(), x.reshape(-1, x.shape[-1])) * alpha
    if out is None:
        return y.to(out_dtype or dy.dtype)
    return out.add_(y.to(out.dtype)) if accumulate else out.copy_(y.to(out.dtype))


# ------------------------------------------------------------------ grouped (MoE experts)
def _check_offsets(offsets: torch.Tensor):
    assert offsets.dtype == torch.int32 and offsets.dim() == 1


def grouped_mm_nt(x: torch.Tensor, w: torch.Tensor, offsets: torch.Tensor, bias: Optional[torch.Tensor] = None,
                  out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``y[r] = x[r] @ w[g(r)]^T`` for rows grouped by expert.

    ``x`` is ``[R, K]`` with group ``g`` owning rows ``offsets[g]:offsets[g+1]`` (every offset a multiple of
    128; rows past ``offsets[-1]`` are ignored), ``w`` is ``[G, N, K]``.
    """
    _check_offsets(offsets)
    G, N, K = w.shape
    R = x.shape[0]
    if not _use_cuda(x, w, offsets):
        y = torch.zeros(R, N, dtype=x.dtype, device=x.device) if out is None else out
        off = offsets.tolist()
        for g in range(G):
            s, e = off[g], off[g + 1]
            if e > s:
                r = _lib_mm(x[s:e], w[g].t())
                if bias is not None:
                    r = r + bias[g].float()
                y[s:e] = r.to(y.dtype)
        return y
    x2 = _row_major_2d(x)
    w2 = w.contiguous().view(G * N, K)
    c = _out(out, (R, N), torch.bfloat16, x.device, False)
    _launch(x2, K, R, x2.stride(0), False, w2, K, G * N, K, False, c, c.stride(0), 0, R, N, K, 1.0, bias, False,
            mode=GROUPED_M, num_groups=G, offsets=offsets, b_group_rows=N)
    return c


def grouped_mm_nn(dy: torch.Tensor, w: torch.Tensor, offsets: torch.Tensor,
                  out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``dx[r] = dy[r] @ w[g(r)]`` with ``dy [R, N]``, ``w [G, N, K]`` -> ``[R, K]``."""
    _check_offsets(offsets)
    G, N, K = w.shape
    R = dy.shape[0]
    if not _use_cuda(dy, w, offsets):
        y = torch.zeros(R, K, dtype=dy.dtype, device=dy.device) if out is None else out
        off = offsets.tolist()
        for g in range(G):
            s, e = off[g], off[g + 1]
            if e > s:
                y[s:e] = _lib_mm(dy[s:e], w[g]).to(y.dtype)
        return y
    assert N % 64 == 0, 'grouped dgrad needs the contraction (N) to be a multiple of 64'
    d2 = _row_major_2d(dy)
    w2 = w.contiguous().view(G * N, K)
    c = _out(out, (R, K), torch.bfloat16, dy.device, False)
    _launch(d2, N, R, d2.stride(0), False, w2, K, G * N, K, True, c, c.stride(0), 0, R, K, N, 1.0, None, False,
            mode=GROUPED_M, num_groups=G, offsets=offsets, b_group_rows=N)
    return c


def grouped_mm_tn(dy: torch.Tensor, x: torch.Tensor, offsets: torch.Tensor, out: Optional[torch.Tensor] = None,
                  out_dtype: Optional[torch.dtype] = None, accumulate: bool = False) -> torch.Tensor:
    """``dw[g] = dy[rows g]^T @ x[rows g]`` -> ``[G, N, K]``; padded rows inside a group must be zero."""
    _check_offsets(offsets)
    G = offsets.numel() - 1
    N, K = dy.shape[-1], x.shape[-1]
    if not _use_cuda(dy, x, offsets):
        y = torch.zeros(G, N, K, dtype=torch.float32, device=dy.device)
        off = offsets.tolist()
        for g in range(G):
            s, e = off[g], off[g + 1]
            if e > s:
                y[g] = _lib_mm(dy[s:e].t(), x[s:e])
        if out is not None:
            if accumulate:
                out.add_(y.to(out.dtype))
            else:
                out.copy_(y.to(out.dtype))
            return out
        return y.to(out_dtype or dy.dtype)
    d2, x2 = _row_major_2d(dy), _row_major_2d(x)
    R = d2.shape[0]
    c = _out(out, (G, N, K), out_dtype or torch.bfloat16, dy.device, accumulate)
    assert c.is_contiguous()
    _launch(d2, N, R, d2.stride(0), True, x2, K, R, x2.stride(0), True, c, K, N * K, N, K, 0, 1.0, None, accumulate,
            mode=GROUPED_K, num_groups=G, offsets=offsets)
    return c
