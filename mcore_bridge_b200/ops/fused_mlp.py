"""Activation-lean fused blocks for the single-rank (no tensor parallel) dense path.

``norm_linear``:  ``y = rmsnorm(x) @ W^T`` that keeps ``x`` and the per-row ``rstd`` for backward instead of the
normalised activation, which the norm's backward kernel forms again for the weight gradient.
``glu_linear``:   ``y = glu(h) @ W^T`` that keeps ``h`` only; the gated activation comes out of its backward kernel.

Per Qwen3-8B layer and 8192 tokens this drops 2 x 67 MB (normalised inputs of QKV and FC1) and 201 MB (SwiGLU output)
from what autograd holds, about 30 % of a layer's activations, which is what lets a single 180 GB GPU keep almost all
layers' activations instead of recomputing a third of the forward pass.  Results are bit-identical to the unfused
sequence (the recomputed tensors are the same expressions of the same inputs, written over the gradient they follow).
"""
from __future__ import annotations

import torch

from . import _lib
from .linear import _weight_grad


class _NormLinearFn(torch.autograd.Function):

    @staticmethod
    def forward(ctx, x, ln_w, weight, eps, zc):
        y, x2, rstd = _lib.native().norm_linear_fwd(x, ln_w, weight, eps, zc)
        ctx.save_for_backward(x2, ln_w, rstd, weight)
        ctx.eps, ctx.zc, ctx.shape = eps, zc, x.shape
        return y if x.dim() == 2 else y.view(*x.shape[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, ln_w, rstd, weight = ctx.saved_tensors
        need_dw = ctx.needs_input_grad[2]
        dx, dlw, dy2, xn = _lib.native().norm_linear_bwd(dy, x2, ln_w, rstd, weight, ctx.eps, ctx.zc, need_dw)
        return dx.view(ctx.shape), dlw, _weight_grad(weight, dy2, xn) if need_dw else None, None, None


class _GluLinearFn(torch.autograd.Function):

    @staticmethod
    def forward(ctx, h, weight, kind, clamp, offset):
        y, h2 = _lib.native().glu_linear_fwd(h, weight, kind, clamp, offset)
        ctx.save_for_backward(h2, weight)
        ctx.args = (kind, clamp, offset, h.shape)
        return y if h.dim() == 2 else y.view(*h.shape[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, dy):
        h2, weight = ctx.saved_tensors
        kind, clamp, offset, shape = ctx.args
        need_dw = ctx.needs_input_grad[1]
        dh, dy2, a = _lib.native().glu_linear_bwd(dy, h2, weight, kind, clamp, offset, need_dw)
        return dh.view(shape), _weight_grad(weight, dy2, a) if need_dw else None, None, None, None


def usable(x: torch.Tensor, weight: torch.Tensor) -> bool:
    return (x.is_cuda and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and _lib.available()
            and x.shape[-1] % 8 == 0)


def norm_linear(x, ln_w, weight, eps, zero_centered):
    return _NormLinearFn.apply(x, ln_w, weight, float(eps), bool(zero_centered))


def glu_linear(h, weight, kind: int, clamp: float, offset: float):
    return _GluLinearFn.apply(h, weight, int(kind), float(clamp or 0.0), float(offset))
