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


def usable(x: torch.Tensor, weight: torch.Tensor) -> bool:
    return (x.is_cuda and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and _lib.available()
            and x.shape[-1] % 8 == 0)


def norm_linear(x, ln_w, weight, eps, zero_centered, keep: bool = False):
    """With ``keep`` returns ``x`` as well: a residual taken from there has its gradient added to the norm's by the
    norm's backward kernel."""
    return _lib.native().norm_linear(x, ln_w, weight, eps, zero_centered, keep)


def glu_linear(h, weight, kind: int, clamp: float, offset: float, residual=None):
    """``residual`` (of the result's shape) is added in the product's epilogue."""
    return _lib.native().glu_linear(h, weight, kind, clamp or 0.0, offset, residual)
