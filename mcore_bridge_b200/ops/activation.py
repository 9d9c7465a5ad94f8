"""Gated activations: SwiGLU, quick-GEGLU (clamped, offset — gpt-oss), GEGLU-tanh; forward + backward.

Input is ``[rows, 2F]`` laid out ``[gate | up]`` (the fc1 layout the bridge writes); output ``[rows, F]``.
An optional per-row probability multiplies the output (MoE experts weight their output by the router
probability before the second GEMM, so the combine is a plain sum).
CUDA: ``csrc/elementwise/norm_act.cu``.
"""
from __future__ import annotations

from typing import Optional

import torch
import torch.nn.functional as F

from . import _lib

KINDS = {'swiglu': 0, 'quick_geglu': 1, 'geglu_tanh': 2}


def glu_ref(x, kind='swiglu', probs=None, clamp: float = 0.0, offset: float = 0.0):
    g, u = x.float().chunk(2, dim=-1)
    if clamp and clamp > 0:
        g = g.clamp(max=clamp)
        u = u.clamp(min=-clamp, max=clamp)
    if kind == 'swiglu':
        a = F.silu(g)
    elif kind == 'quick_geglu':
        a = g * torch.sigmoid(1.702 * g)
    else:
        a = F.gelu(g, approximate='tanh')
    y = a * (u + offset)
    if probs is not None:
        y = y * probs.float().unsqueeze(-1)
    return y.to(x.dtype)


class _GluCuda(torch.autograd.Function):

    @staticmethod
    def forward(ctx, x, probs, kind, clamp, offset):
        pr = None if probs is None else probs.reshape(-1).float().contiguous()
        out, x2 = _lib.native().glu_fwd(x, pr, kind, clamp, offset)
        ctx.save_for_backward(x2, pr)
        ctx.args = (kind, clamp, offset, x.shape, None if probs is None else (probs.shape, probs.dtype))
        return out if x.dim() == 2 else out.view(*x.shape[:-1], out.shape[-1])

    @staticmethod
    def backward(ctx, dout):
        x2, pr = ctx.saved_tensors
        kind, clamp, offset, shape, pmeta = ctx.args
        din, dpr = _lib.native().glu_bwd(dout, x2, pr, kind, clamp, offset)
        return din.view(shape), None if pmeta is None else dpr.view(pmeta[0]).to(pmeta[1]), None, None, None


def glu(x: torch.Tensor, kind: str = 'swiglu', probs: Optional[torch.Tensor] = None, clamp: float = 0.0,
        offset: float = 0.0) -> torch.Tensor:
    clamp = float(clamp or 0.0)
    if x.is_cuda and x.dtype == torch.bfloat16 and (x.shape[-1] // 2) % 8 == 0 and _lib.available():
        return _GluCuda.apply(x, probs, KINDS[kind], clamp, float(offset))
    return glu_ref(x, kind, probs, clamp, offset)


def swiglu(x: torch.Tensor, probs: Optional[torch.Tensor] = None) -> torch.Tensor:
    return glu(x, 'swiglu', probs)
