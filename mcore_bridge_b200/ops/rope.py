"""Rotary embedding application and the fused QKV post-processing op.

* :func:`apply_rope` — rotate the first ``rot`` dims of ``[T, heads, d]`` with per-token tables
  (rotate-half or interleaved pairs; inverse rotation by negating ``sin``).
* :func:`qkv_split_norm_rope` — split a packed QKV projection per query group, per-head RMSNorm on
  q/k, rope, and write separate q/k/v(/gate) tensors in one pass (CUDA: ``csrc/elementwise/qkv_rope.cu``).

The tables are per token, ``[T, rot/2]`` fp32, so packed sequences, context-parallel chunks, MRoPE
sections and attention scaling (``mscale`` folded into cos/sin, reference
``src/mcore_bridge/model/modules/transformer_layer.py:249-278``) are the table builder's business.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import _lib
from .norm import rmsnorm_ref


def apply_rope_ref(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, interleaved: bool = False) -> torch.Tensor:
    """``x``: ``[T, heads, d]``; ``cos``/``sin``: ``[T, rot/2]``.  Dims past ``rot`` pass through."""
    rot = cos.shape[-1] * 2
    xr, xp = x[..., :rot].float(), x[..., rot:]
    c, s = cos[:, None, :].float(), sin[:, None, :].float()
    if interleaved:
        x1, x2 = xr[..., 0::2], xr[..., 1::2]
        o = torch.stack((x1 * c - x2 * s, x2 * c + x1 * s), dim=-1).flatten(-2)
    else:
        x1, x2 = xr[..., :rot // 2], xr[..., rot // 2:]
        o = torch.cat((x1 * c - x2 * s, x2 * c + x1 * s), dim=-1)
    return torch.cat((o.to(x.dtype), xp), dim=-1)


def apply_rope(x, cos, sin, interleaved: bool = False, inverse: bool = False):
    if inverse:
        sin = -sin
    return apply_rope_ref(x, cos, sin, interleaved)


def qkv_split_norm_rope_ref(qkv, wq, wk, cos, sin, ng, qpg, d, has_gate, interleaved, eps, zero_centered):
    T = qkv.shape[0]
    per_group = qpg * (2 if has_gate else 1) + 2
    x = qkv.reshape(T, ng, per_group, d)
    nqs = qpg * (2 if has_gate else 1)
    qs = x[:, :, :nqs]
    k = x[:, :, nqs]
    v = x[:, :, nqs + 1]
    gate = None
    if has_gate:
        gate = qs[:, :, 1::2].reshape(T, ng * qpg, d)
        q = qs[:, :, 0::2].reshape(T, ng * qpg, d)
    else:
        q = qs.reshape(T, ng * qpg, d)
    if wq is not None:
        q = rmsnorm_ref(q, wq, eps, zero_centered)
        k = rmsnorm_ref(k, wk, eps, zero_centered)
    if cos is not None:
        q = apply_rope_ref(q, cos, sin, interleaved)
        k = apply_rope_ref(k, cos, sin, interleaved)
    return q.contiguous(), k.contiguous(), v.contiguous(), (gate.contiguous() if gate is not None else None)


def qkv_split_norm_rope(qkv: torch.Tensor, wq: Optional[torch.Tensor], wk: Optional[torch.Tensor],
                        cos: Optional[torch.Tensor], sin: Optional[torch.Tensor], num_groups: int,
                        q_per_group: int, head_dim: int, has_gate: bool = False, interleaved: bool = False,
                        eps: float = 1e-6, zero_centered: bool = False
                        ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, Optional[torch.Tensor]]:
    """Packed ``[T, ng*(qpg(+gates)+2)*d]`` -> ``q [T,nq,d]``, ``k [T,ng,d]``, ``v [T,ng,d]``, ``gate``."""
    if (qkv.is_cuda and qkv.dtype == torch.bfloat16 and head_dim <= 256 and head_dim % 8 == 0 and _lib.available()
            and (wq is None or wq.dtype == torch.bfloat16)):
        if cos is not None:
            cos, sin = cos.float().contiguous(), sin.float().contiguous()
        return _lib.native().qkv(qkv, wq, wk, cos, sin, num_groups, q_per_group, head_dim, has_gate, interleaved, eps,
                                 zero_centered)
    return qkv_split_norm_rope_ref(qkv, wq, wk, cos, sin, num_groups, q_per_group, head_dim, has_gate, interleaved,
                                   eps, zero_centered)
