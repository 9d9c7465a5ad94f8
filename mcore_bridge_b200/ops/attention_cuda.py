"""Binding of the in-tree sm_100a attention kernels (``csrc/attention``).

Forward: ``attn_fwd_sm100.cu`` (tcgen05 / TMEM, online softmax in two warp groups).  Backward:
``attn_bwd_sm100.cu`` (delta, dQ and dK/dV kernels; the dK/dV kernel can split the query heads of a GQA group over
several CTAs when the grid would not fill the GPU).
"""
from __future__ import annotations

import ctypes
import math
from typing import Optional

import torch

from . import _lib

_ll, _int, _f = ctypes.c_longlong, ctypes.c_int, ctypes.c_float


def unsupported_reason(q, k, v, causal, window, sinks, softcap) -> Optional[str]:
    """``None`` when the in-tree kernel covers the call, else what it lacks (used for the one-time warning)."""
    if not causal:
        return 'non-causal attention'
    if window is not None and (window[0] is None or int(window[0]) < 0):
        window = None
    if softcap:
        return 'soft-capped scores'
    if q.dtype != torch.bfloat16:
        return f'dtype {q.dtype}'
    if q.shape[-1] not in (64, 128):
        return f'head size {q.shape[-1]}'
    if v.shape[-1] != q.shape[-1]:
        return f'value head size {v.shape[-1]} != query head size {q.shape[-1]}'
    if q.shape[1] % k.shape[1] != 0 or q.shape[0] != k.shape[0]:
        return 'query / key token counts or head counts that do not match'
    return None


def supported(q, k, v, causal, window, sinks, softcap) -> bool:
    return unsupported_reason(q, k, v, causal, window, sinks, softcap) is None and _lib.available()


def _here(t: torch.Tensor, device) -> bool:
    """Whether a CUDA tensor is on ``device``, where ``cuda`` is the current one."""
    device = torch.device(device)
    index = torch.cuda.current_device() if device.type == 'cuda' and device.index is None else device.index
    return device.type == 'cuda' and t.device.index == index


def seq_start_from_cu(cu_seqlens: Optional[torch.Tensor], T: int, device) -> torch.Tensor:
    """``[T]`` int32: index of the first token of the packed sequence each token belongs to."""
    if cu_seqlens is None:
        return torch.zeros(T, dtype=torch.int32, device=device)
    if cu_seqlens.is_cuda and _here(cu_seqlens, device) and cu_seqlens.numel() >= 2 \
            and cu_seqlens.dtype in (torch.int32, torch.int64) and cu_seqlens.dim() == 1 and _lib.cuda_enabled():
        return _lib.native().seq_starts(cu_seqlens, T)
    cu = cu_seqlens.to(device=device, dtype=torch.int64)
    seg = torch.searchsorted(cu[1:].contiguous(), torch.arange(T, device=device), right=True)
    return cu[:-1][seg.clamp(max=cu.numel() - 2)].to(torch.int32)


def _row_starts(seq_start: torch.Tensor, T: int, device, one_each: bool) -> torch.Tensor:
    """``seq_start`` as the kernels read it: ``T`` int32 on ``device``, one after the other.  A single value counts for
    every token; more than ``T`` are refused with ``one_each``."""
    if seq_start.dtype == torch.int32 and seq_start.shape == (T,) and seq_start.device == device:
        return seq_start.contiguous()
    n = seq_start.numel()
    if n != 1 and (n < T or (one_each and n != T)):
        raise RuntimeError(f'seq_start has {n} elements for {T} tokens')
    if seq_start.is_floating_point() or seq_start.is_complex():
        raise RuntimeError(f'seq_start is {seq_start.dtype}: whole numbers are wanted')
    if seq_start.device != device and seq_start.dim() > 0:
        raise RuntimeError(f'seq_start is on {seq_start.device}, the queries are on {device}')
    seq_start = seq_start.to(device=device, dtype=torch.int32).reshape(-1)
    return (seq_start.expand(T) if n == 1 else seq_start[:T]).contiguous()


def attention(q, k, v, cu_seqlens, max_seqlen, scale, seq_start: Optional[torch.Tensor] = None, window=None,
              sinks: Optional[torch.Tensor] = None):
    """Packed causal self-attention.  ``window = (left, _)`` limits every query to its ``left`` most recent
    predecessors (plus itself); ``sinks [nq]`` adds a learnable per-head logit to every row's softmax."""
    T, nq, d = q.shape
    if scale is None:
        scale = 1.0 / math.sqrt(d)
    if seq_start is None:
        seq_start = seq_start_from_cu(cu_seqlens, T, q.device)
    left = None if window is None or window[0] is None or int(window[0]) < 0 else int(window[0])
    seq_start = _row_starts(seq_start, T, q.device, left is not None)
    if left is None and sinks is None:
        return _lib.native().attention(q, k, v, seq_start, None, None, None, None, scale)[0]
    k_lo = seq_start
    if left is not None:
        # still non-decreasing, so the kernels' causal fast paths (k_hi = the query itself) apply unchanged
        k_lo = _lib.native().attn_window_starts(seq_start, left)
    o, _ = attention_ranges(q, k, v, k_lo, None, None, None, scale, sinks)
    return o


# ---------------------------------------------------------------------------------------------------------------
# general masks: per-query inclusive key ranges (context-parallel attention, non-causal packed attention)
# ---------------------------------------------------------------------------------------------------------------
def ranges_supported(q, k, v) -> bool:
    d = q.shape[-1]
    return (q.is_cuda and q.dtype == torch.bfloat16 and d in (64, 128) and v.shape[-1] == d and k.shape[-1] == d
            and q.shape[1] % k.shape[1] == 0 and _lib.available())


def fwd_ranges_raw(q, k, v, k_lo, k_hi, scale: float):
    """One forward launch without autograd: ``(o [T, nq, d], lse [nq, T])`` of the queries over their key ranges in
    ``k`` / ``v`` (rows with an empty range: ``o = 0``, ``lse = -inf``).  Building block of ring attention."""
    T, nq, d = q.shape
    o = torch.empty_like(q)
    lse = torch.empty((nq, T), dtype=torch.float32, device=q.device)
    rc = _lib.lib().mcb_attn_fwd_ranges(_lib.ptr(q), _lib.ptr(k), _lib.ptr(v), _lib.ptr(k_lo), _lib.ptr(k_hi), None,
                                        _lib.ptr(o), _lib.ptr(lse), _int(T), _int(k.shape[0]), _int(nq),
                                        _int(k.shape[1]), _int(d), _f(scale), _lib.ptr(_lib.status_word(q.device)),
                                        _lib.stream_ptr())
    _lib.check_rc(rc, 'mcb_attn_fwd_ranges')
    return o, lse


def bwd_ranges_raw(q, k, v, o, do, lse, delta, k_lo, k_hi, q_lo, q_hi, scale: float):
    """One backward launch without autograd, with the log-sum-exp and ``delta = rowsum(o * do)`` of the *whole*
    attention given (``[nq, T]`` fp32): ``(dq, dk, dv)`` of this block of keys."""
    T, nq, d = q.shape
    Tk, nkv = k.shape[0], k.shape[1]
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    splits = _lib.native().attn_dkv_splits(Tk, nq, nkv)
    partial = torch.empty((2, splits, Tk, nkv, d), dtype=torch.float32, device=q.device) if splits > 1 else None
    rc = _lib.lib().mcb_attn_bwd_ranges(
        _lib.ptr(q), _lib.ptr(k), _lib.ptr(v), _lib.ptr(o), _lib.ptr(do), _lib.ptr(lse), _lib.ptr(delta), _int(1),
        _lib.ptr(k_lo), _lib.ptr(k_hi), _lib.ptr(q_lo), _lib.ptr(q_hi), _lib.ptr(dq), _lib.ptr(dk), _lib.ptr(dv),
        _int(T), _int(Tk), _int(nq), _int(nkv), _int(d), _f(scale), _lib.ptr(partial), _int(splits),
        _lib.ptr(_lib.status_word(q.device)), _lib.stream_ptr())
    _lib.check_rc(rc, 'mcb_attn_bwd_ranges')
    return dq, dk, dv


def attention_ranges(q, k, v, k_lo, k_hi, q_lo, q_hi, scale: Optional[float] = None,
                     sinks: Optional[torch.Tensor] = None):
    """``o[i] = softmax over keys k_lo[i]..k_hi[i] of q[i] k^T * scale`` applied to ``v``; queries ``[T, nq, d]`` and
    keys / values ``[Tk, nkv, d]`` may be different token sets.  ``q_lo`` / ``q_hi`` ``[Tk]`` bound, per key, the
    queries that can see it (they only limit the loops of the dK/dV kernel).

    Returns ``(o [T, nq, d], lse [nq, T])``; all four range tensors are int32 on the device (``k_hi`` / ``q_lo`` /
    ``q_hi`` may all be ``None`` for masks of the causal family: ``k_hi[i] = i`` and a non-decreasing ``k_lo``)."""
    if scale is None:
        scale = 1.0 / math.sqrt(q.shape[-1])
    return _lib.native().attention(q, k, v, k_lo, k_hi, q_lo, q_hi, sinks, scale)
