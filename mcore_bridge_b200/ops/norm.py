"""RMSNorm (plain / zero-centred gamma / per-head), forward + backward.

CUDA: ``csrc/elementwise/norm_act.cu``.  The torch path is the CPU oracle; its math follows the
zero-centred definition the reference spells out in ``src/mcore_bridge/model/gpts/qwen3_next.py:87-95``
(``x * rsqrt(mean(x^2) + eps) * (1 + w)`` computed in fp32).
"""
from __future__ import annotations

import torch

from . import _lib


def rmsnorm_ref(x: torch.Tensor, w: torch.Tensor, eps: float, zero_centered: bool = False) -> torch.Tensor:
    xf = x.float()
    y = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps)
    wf = w.float() + 1.0 if zero_centered else w.float()
    return (y * wf).to(x.dtype)


def rmsnorm(x: torch.Tensor, w: torch.Tensor, eps: float = 1e-6, zero_centered: bool = False) -> torch.Tensor:
    """Normalises the last dimension.  ``x`` may be ``[..., H]`` (per-head norm: pass ``[..., heads, d]``)."""
    if x.is_cuda and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0 \
            and x.shape[-1] <= 16384 and _lib.available():
        return _lib.native().rmsnorm(x, w, eps, zero_centered)
    return rmsnorm_ref(x, w, eps, zero_centered)


def layernorm_ref(x, w, b, eps):
    return torch.nn.functional.layer_norm(x.float(), (x.shape[-1],), w.float(), None if b is None else b.float(),
                                          eps).to(x.dtype)


def l2norm(x: torch.Tensor, eps: float = 1e-6) -> torch.Tensor:
    """``x / sqrt(sum(x^2) + eps)`` over the last dim (q/k normalisation of gated DeltaNet)."""
    xf = x.float()
    return (xf * torch.rsqrt(xf.pow(2).sum(-1, keepdim=True) + eps)).to(x.dtype)
