"""Attention kernels at the edges of their tiles: one to a few 128-row query tiles and key blocks, every way the forward
kernel fills a CTA (two heads of a group, two row tiles, one tile with its keys split), windows, sinks and ranges with gaps, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = 'cuda'

CASES = [   # queries, keys, query heads, kv heads, head size, mask
    (1, 1, 1, 1, 64, 'causal'), (127, 127, 4, 2, 64, 'packed'), (128, 128, 3, 1, 128, 'causal'),
    (129, 129, 6, 2, 128, 'packed'), (1100, 1100, 32, 8, 128, 'packed'),       # paired heads
    (1300, 1300, 24, 8, 64, 'window'),                                         # paired rows (odd group size)
    (2100, 2100, 9, 3, 128, 'window'), (2000, 2000, 64, 8, 64, 'sinks'),
    (700, 1300, 32, 4, 128, 'ranges'), (1300, 700, 30, 10, 64, 'ranges'), (900, 2000, 24, 8, 128, 'gaps'),
    # few enough tiles for one CTA each: the key blocks of a tile alternate between the two softmax groups
    (1500, 1500, 4, 2, 128, 'causal'), (1500, 1500, 2, 1, 64, 'packed'), (1000, 1000, 6, 2, 64, 'window'),
    (1100, 1100, 8, 1, 128, 'sinks'), (600, 1700, 4, 4, 128, 'ranges'), (300, 2000, 6, 2, 64, 'gaps'),
]


def _mask(T, Tk, kind, gen):
    """Per-query inclusive key ranges (lo, hi or None = own index) and, for general ranges, per-key query bounds."""
    i = torch.arange(T, device=DEV, dtype=torch.int32)
    lo, hi, ql, qh = torch.zeros_like(i), None, None, None
    if kind in ('packed', 'window', 'sinks'):
        from mcore_bridge_b200.ops.attention_cuda import seq_start_from_cu
        cu = torch.tensor(sorted({0, T // 7, T // 3, T // 3 + 5, T}), dtype=torch.int32, device=DEV)
        lo = seq_start_from_cu(cu, T, DEV)
    if kind in ('window', 'sinks'):
        lo = torch.maximum(lo, i - 100)
    if kind == 'ranges':        # arbitrary, some empty
        lo = torch.randint(0, Tk, (T,), generator=gen, device=DEV, dtype=torch.int32)
        hi = (lo + torch.randint(-20, Tk // 2, (T,), generator=gen, device=DEV, dtype=torch.int32)).clamp(max=Tk - 1)
    if kind == 'gaps':          # tiles of one CTA see key blocks far apart
        lo = torch.where(i % 300 < 150, 0, Tk - 200).int()
        hi = lo + 150
    keys = torch.arange(Tk, device=DEV)
    vis = (keys[None] >= lo[:, None]) & (keys[None] <= (i if hi is None else hi)[:, None])
    if hi is not None:
        seen = vis.any(0)
        ql = torch.where(seen, vis.int().argmax(0), 1).int()
        qh = torch.where(seen, T - 1 - vis.flip(0).int().argmax(0), 0).int()
    return lo.contiguous(), hi, ql, qh, vis


@pytest.mark.parametrize('sharp', [1.0, 6.0])       # 6: row maxima grow past the lazy-rescale threshold
@pytest.mark.parametrize('T,Tk,nq,nkv,d,kind', CASES)
def test_tile_edges_match_fp64(T, Tk, nq, nkv, d, kind, sharp):
    from mcore_bridge_b200.ops import _lib
    from mcore_bridge_b200.ops.attention_cuda import attention_ranges
    gen = torch.Generator(device=DEV).manual_seed(3)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device=DEV)

    q, k, v = (rand(T, nq, d) * sharp).bfloat16(), rand(Tk, nkv, d).bfloat16(), rand(Tk, nkv, d).bfloat16()
    sinks = rand(nq) * 3 if kind == 'sinks' else None
    leaves = [t.requires_grad_() for t in ([q, k, v] + ([sinks] if sinks is not None else []))]
    lo, hi, ql, qh, vis = _mask(T, Tk, kind, gen)
    o, lse = attention_ranges(q, k, v, lo, hi, ql, qh, d ** -0.5, sinks)
    dy = rand(T, nq, d).bfloat16()
    grads = torch.autograd.grad(o, leaves, dy)
    _lib.check_status()

    wide = [t.detach().double().requires_grad_() for t in leaves]
    qw, kw, vw = (t.transpose(0, 1) for t in wide[:3])
    kw, vw = (t.repeat_interleave(nq // nkv, 0) for t in (kw, vw))
    s = (qw @ kw.transpose(1, 2) * d ** -0.5).masked_fill(~vis[None], -1e30)
    if sinks is not None:
        s = torch.cat([s, wide[3].view(nq, 1, 1).expand(nq, T, 1)], -1)
    p = torch.softmax(s, -1)[..., :Tk] * vis[None]
    ref = (p @ vw).transpose(0, 1)
    want = torch.autograd.grad(ref, wide, dy.double())

    def rel(a, b):
        return ((a.double() - b).norm() / b.norm().clamp(min=1e-30)).item()

    # bf16 probabilities and a bf16 result: at most 2^-9 relative each; the gradients add bf16 dS, dO sums and results
    assert rel(o, ref) < 2 ** -8
    for a, b in zip(grads, want):
        assert rel(a, b) < 2 ** -7
    some = vis.any(1) if sinks is None else torch.ones(T, dtype=torch.bool, device=DEV)
    exact = torch.logsumexp(s, -1)
    assert (lse[:, some].double() - exact[:, some]).abs().max() < 1e-4      # fp32 sums of up to 2100 terms, |lse| < 100
    assert torch.isneginf(lse[:, ~some]).all() and (o[~some] == 0).all()


@pytest.mark.parametrize('T,d', [(1100, 128), (4000, 64)])
def test_probabilities_keep_their_precision_over_many_blocks(T, d):
    """The bf16 probabilities are rounded against a reference that follows the row's maximum: the result is no further from
    fp64 than with the final maximum as the reference, for which the largest probabilities lie just below 1."""
    from mcore_bridge_b200.ops.attention import attention
    gen = torch.Generator(device=DEV).manual_seed(4)
    q, k, v = (torch.randn(T, 2, d, generator=gen, device=DEV).bfloat16() for _ in range(3))
    o = attention(q, k, v, torch.tensor([0, T], dtype=torch.int32, device=DEV), T)
    qw, kw, vw = (t.double().transpose(0, 1) for t in (q, k, v))
    hide = torch.ones(T, T, dtype=torch.bool, device=DEV).triu(1)
    s = (qw @ kw.transpose(1, 2) * d ** -0.5).masked_fill(hide, float('-inf'))
    p = torch.exp(s - s.amax(-1, keepdim=True))
    ref = (p / p.sum(-1, keepdim=True)) @ vw
    rounded = ((p.bfloat16().double() @ vw) / p.sum(-1, keepdim=True)).bfloat16().double()
    # 4000 x 128 (1100 x 256) independent roundings: the two errors agree to far less than half a per cent by chance
    assert (o.transpose(0, 1).double() - ref).norm() <= 1.005 * (rounded - ref).norm()


@pytest.mark.parametrize('nq,nkv,d', [(6, 2, 64), (5, 1, 128), (8, 2, 128)])
@pytest.mark.parametrize('left', [0, 1, 31, 32, 33, 64, 127, 128, 129])
def test_windows_at_the_edges_of_pieces(nq, nkv, d, left):
    """The mask is looked at in pieces of 32 x 32: windows that end on, before and behind them; group sizes of 3 and 5, whose dK and
    dV are summed from as many parts."""
    from mcore_bridge_b200.ops.attention import attention
    T, cuts = 420, [0, 33, 160, 420]
    gen = torch.Generator(device=DEV).manual_seed(5)
    q, k, v, dy = (torch.randn(T, n, d, generator=gen, device=DEV).bfloat16() for n in (nq, nkv, nkv, nq))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    o = attention(*leaves, torch.tensor(cuts, dtype=torch.int32, device=DEV), 260, window=(left, 0))
    grads = torch.autograd.grad(o, leaves, dy)
    i = torch.arange(T, device=DEV)
    seq = torch.bucketize(i, torch.tensor(cuts[1:], device=DEV), right=True)
    vis = (seq[:, None] == seq[None]) & (i[None] <= i[:, None]) & (i[None] >= i[:, None] - left)
    wide = [t.detach().double().requires_grad_() for t in leaves]
    kw, vw = (t.transpose(0, 1).repeat_interleave(nq // nkv, 0) for t in wide[1:])
    s = (wide[0].transpose(0, 1) @ kw.transpose(1, 2) * d ** -0.5).masked_fill(~vis[None], float('-inf'))
    ref = (torch.softmax(s, -1) @ vw).transpose(0, 1)
    want = torch.autograd.grad(ref, wide, dy.double())
    # as above: one bf16 rounding of probabilities and result, two more in the gradients (with one visible key dq and dk are zero
    # but for the rounding of dP - delta, whose terms are sums of d products of size 1)
    assert (o.double() - ref).norm() < 2 ** -8 * ref.norm()
    for a, b in zip(grads, want):
        assert (a.double() - b).norm() < 2 ** -7 * max(b.norm().item(), 2 ** -8 * a.numel() ** 0.5)
