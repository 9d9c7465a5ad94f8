"""Chunked linear-attention kernels (simple GLA, gated delta rule) at the edges of their chunks, against fp64
recurrences: single tokens, whole chunks, one token more, sequences that end inside a chunk, empty sequences."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp(min=1e-30)).item()


def _spans(T, cuts):
    return list(zip([0] + cuts, cuts + [T]))


def _inputs(T, h, d, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randn(T, h, d, generator=gen, device=DEV).bfloat16() for _ in range(4)], gen


@pytest.mark.parametrize('T,h,d,cuts', [(1, 1, 64, []), (5, 2, 128, [2, 2]), (127, 2, 64, []), (128, 3, 128, []),
                                        (129, 2, 128, [1]), (700, 4, 64, [3, 130, 131, 600]), (800, 2, 128, [128, 384])])
def test_simple_gla_chunk_edges(T, h, d, cuts):
    from mcore_bridge_b200.ops.gdn import simple_gla
    (q, k, v, dy), _ = _inputs(T, h, d, 1)
    decay = -torch.tensor([0.02, 3.0, 0.2, 0.001], device=DEV)[:h]
    cu = torch.tensor([0] + cuts + [T], dtype=torch.int32, device=DEV)
    leaves = [t.requires_grad_() for t in (q, k, v)]
    o = simple_gla(*leaves, decay, cu)
    grads = torch.autograd.grad(o, leaves, dy)
    wide = [t.detach().double().requires_grad_() for t in leaves]
    out = []
    for s, e in _spans(T, cuts):
        n = torch.arange(e - s, device=DEV, dtype=torch.float64)
        gap = n[:, None] - n[None]
        mix = torch.exp(decay.double()[:, None, None] * gap.clamp(min=0)) * (gap >= 0) * d ** -0.5
        att = torch.einsum('ihd,jhd->hij', wide[0][s:e], wide[1][s:e]) * mix
        out.append(torch.einsum('hij,jhd->ihd', att, wide[2][s:e]))
    ref = torch.cat(out)
    # fp32 products and states (16-bit-mantissa terms): what remains is the rounding of the result to bf16, 2^-9
    for a, b in zip([o, *grads], [ref, *torch.autograd.grad(ref, wide, dy.double())]):
        assert _rel(a, b) < 2 ** -8
