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
                                        (129, 2, 128, [1]), (700, 4, 64, [3, 130, 131, 600]),
                                        (800, 2, 128, [128, 384])])
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


def _delta_rule(q, k, v, g, beta, spans):
    out = []
    for s, e in spans:
        S = torch.zeros(q.shape[1], q.shape[2], q.shape[2], dtype=torch.float64, device=DEV)
        for t in range(s, e):
            S = S * g[t].exp()[:, None, None]
            write = (v[t] - torch.einsum('hkv,hk->hv', S, k[t])) * beta[t][:, None]
            S = S + k[t][:, :, None] * write[:, None, :]
            out.append(torch.einsum('hkv,hk->hv', S, q[t]) * q.shape[2] ** -0.5)
    return torch.stack(out)


@pytest.mark.parametrize('T,h,d,cuts', [(1, 1, 64, []), (5, 2, 128, [2, 2]), (63, 2, 64, []), (64, 3, 128, []),
                                        (65, 2, 128, [1]), (300, 4, 64, [3, 130, 131]), (270, 2, 128, [128])])
def test_gated_delta_rule_chunk_edges(T, h, d, cuts):
    from mcore_bridge_b200.ops.gdn import chunk_gated_delta_rule, l2norm
    (q, k, v, dy), gen = _inputs(T, h, d, 2)
    q, k = l2norm(q), l2norm(k)
    g = -torch.rand(T, h, generator=gen, device=DEV) * torch.tensor([0.05, 8.0, 0.5, 0.001], device=DEV)[:h]
    beta = torch.rand(T, h, generator=gen, device=DEV)
    cu = torch.tensor([0] + cuts + [T], dtype=torch.int32, device=DEV)
    leaves = [t.requires_grad_() for t in (q, k, v, g, beta)]
    o = chunk_gated_delta_rule(*leaves, cu)
    grads = torch.autograd.grad(o, leaves, dy)
    wide = [t.detach().double().requires_grad_() for t in leaves]
    ref = _delta_rule(*wide, _spans(T, cuts))
    # fp32 throughout (operands with 16 mantissa bits): bf16 results are rounded once, g and beta gradients not at all
    for a, b in zip([o, *grads], [ref, *torch.autograd.grad(ref, wide, dy.double())]):
        assert _rel(a, b) < (2 ** -8 if a.dtype == torch.bfloat16 else 2 ** -12)


def test_gated_delta_rule_outside_every_sequence_is_zero():
    from mcore_bridge_b200.ops.gdn import chunk_gated_delta_rule
    (q, k, v, dy), _ = _inputs(100, 2, 64, 3)
    leaves = [t.requires_grad_() for t in (q, k, v)]
    g, beta = -torch.rand(100, 2, device=DEV), torch.rand(100, 2, device=DEV)
    o = chunk_gated_delta_rule(*leaves, g, beta, torch.tensor([0, 70], dtype=torch.int32, device=DEV))
    grads = torch.autograd.grad(o, leaves, dy)
    assert all((t[70:] == 0).all() and (t[:70] != 0).any() for t in (o, *grads))


def test_gated_delta_rule_differentiates_twice():
    """With ``create_graph`` the gradient comes from the torch evaluation: same values, and differentiable again."""
    from mcore_bridge_b200.ops.gdn import chunk_gated_delta_rule, l2norm
    (q, k, v, dy), _ = _inputs(80, 2, 64, 5)
    q, k = l2norm(q), l2norm(k)
    g, beta = -torch.rand(80, 2, device=DEV), torch.rand(80, 2, device=DEV)
    leaves = [t.requires_grad_() for t in (q, k, v, g, beta)]
    first = torch.autograd.grad(chunk_gated_delta_rule(*leaves), leaves, dy)
    again = torch.autograd.grad(chunk_gated_delta_rule(*leaves), leaves, dy, create_graph=True)
    for a, b in zip(first, again):
        assert _rel(a, b.double()) < 2 ** -8
    second = torch.autograd.grad(again[2].float().square().sum(), beta)[0]
    assert torch.isfinite(second).all() and (second != 0).any()


@pytest.mark.parametrize('T,groups,ratio,d,cuts', [(1, 1, 1, 64, []), (3, 2, 2, 128, [1]), (16, 1, 4, 64, [13, 15]),
                                                   (65, 3, 2, 128, [62, 64]), (130, 2, 4, 128, []),
                                                   (257, 2, 1, 64, [1, 2, 3]),
                                                   # sequences that begin between whole groups of four rows
                                                   (300, 1, 2, 128, [100, 201, 203, 240]), (299, 2, 1, 128, [74])])
def test_gdn_inputs_walk_edges(T, groups, ratio, d, cuts):
    """Projection -> inputs of the delta rule in one pass, at the edges of a warp's walk (16 / 32 tokens) and of
    sequences."""
    import torch.nn.functional as F
    from mcore_bridge_b200.ops.attention_cuda import seq_start_from_cu
    from mcore_bridge_b200.ops.gdn import gdn_inputs
    gen = torch.Generator(device=DEV).manual_seed(4)
    S, h = 2 + ratio, groups * ratio

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device=DEV).bfloat16()

    proj, w = rand(T, groups * (2 * d + 2 * ratio * d + 2 * ratio)), rand(groups * S * d, 4) * 0.5
    A_log, dt = rand(h), rand(h)
    cu = torch.tensor([0] + cuts + [T], dtype=torch.int32, device=DEV)
    leaves = [t.requires_grad_() for t in (proj, w, A_log, dt)]
    out = gdn_inputs(*leaves, seq_start_from_cu(cu, T, DEV), groups, ratio, d)
    cot = [rand(*t.shape).to(t.dtype) for t in out]
    grads = torch.autograd.grad(out, leaves, cot)

    wide = [t.detach().double().requires_grad_() for t in leaves]
    qkv, z, b, a = wide[0].view(T, groups, -1).split([S * d, ratio * d, ratio, ratio], dim=-1)
    qkv, pieces = qkv.reshape(T, -1), []
    for s, e in _spans(T, cuts):
        xs = F.pad(qkv[s:e], (0, 0, 3, 0))
        pieces.append(sum(xs[j:j + e - s] * wide[1][:, j] for j in range(4)))
    q, k, v = F.silu(torch.cat(pieces)).view(T, groups, -1).split([d, d, ratio * d], dim=-1)
    q, k = (t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (t.repeat_interleave(ratio, dim=1) for t in (q, k))
    ref = [q, k, v.reshape(T, h, d), z.reshape(T, h, d),
           -wide[2].exp() * F.softplus(a.reshape(T, h) + wide[3]), torch.sigmoid(b.reshape(T, h))]
    want = torch.autograd.grad(ref, wide, [c.double() for c in cot])
    # bf16 results, q and k rounded once more before their norm: 2^-9 each; g and beta are fp32
    for x, y in zip(out, ref):
        assert _rel(x, y) < (2 ** -8 if x.dtype == torch.bfloat16 else 1e-5)
    for x, y in zip(grads, want):
        assert _rel(x, y) < 2 ** -7


def _gates(T, d, gen):
    """A projection whose gate columns run from one infinity to the other (one group, four value heads)."""
    proj = torch.randn(T, 2 * d + 8 * d + 8, generator=gen, device=DEV)
    wide = torch.cat([torch.linspace(-100, 100, T - 2, device=DEV), torch.tensor([-1e-3, 1e-3], device=DEV)])
    b, a = proj[:, -8:-4], proj[:, -4:]
    b[:, 0], a[:, 3], b[:, 3] = wide, wide, -wide
    b[::3, 1], b[1::3, 1], a[::2, 1] = float('inf'), -float('inf'), -float('inf')
    A_log = torch.tensor([2.0, 0.5, -float('inf'), -3.0], device=DEV)
    dt = torch.tensor([1.0, -0.5, 0.25, 0.0], device=DEV)
    return proj.bfloat16(), A_log.bfloat16(), dt.bfloat16()


def test_gdn_gates_over_their_whole_range():
    """beta = sigmoid(b) and g = -exp(A_log) softplus(a + dt) element by element, infinite gates included."""
    import torch.nn.functional as F
    from mcore_bridge_b200.ops.gdn import gdn_inputs
    T, d = 64, 64
    gen = torch.Generator(device=DEV).manual_seed(6)
    proj, A_log, dt = _gates(T, d, gen)
    w = torch.randn(6 * d, 4, generator=gen, device=DEV).bfloat16()
    leaves = [t.requires_grad_() for t in (proj, A_log, dt)]
    out = gdn_inputs(leaves[0], w, leaves[1], leaves[2], torch.zeros(T, dtype=torch.int32, device=DEV), 1, 4, d)
    g, beta = out[4], out[5]
    dg, dbeta = (torch.randn(T, 4, generator=gen, device=DEV) for _ in range(2))
    grads = torch.autograd.grad([g, beta], leaves, [dg, dbeta])
    wide = [t.detach().double().requires_grad_() for t in (proj[:, -8:-4], proj[:, -4:], A_log, dt)]
    ref_b, ref_g = torch.sigmoid(wide[0]), -wide[2].exp() * F.softplus(wide[1] + wide[3])
    want = torch.autograd.grad([ref_g, ref_b], wide, [dg.double(), dbeta.double()])
    # CUDA's bounds: expf and log1pf 2 ulp each, sums, quotient and product 1/2 ulp each: under 8 ulp = 2^-21 (below the
    # smallest normal number the spacing is absolute)
    for x, ref in ((g, ref_g), (beta, ref_b)):
        assert ((x.double() - ref).abs() <= 2 ** -21 * ref.abs() + 2 ** -126).all()
    got = [grads[0][:, -8:-4], grads[0][:, -4:], grads[1], grads[2]]
    for x, ref in zip(got, want):                       # rounded to bf16; sums of 64 fp32 terms before that
        assert ((x.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5).all()


@pytest.mark.parametrize('op', ['gla', 'rule'])
@pytest.mark.parametrize('bounds,same,report', [
    ([0, 150, 400], [0, 150, 300], True), ([0, 300, 900], [0, 300, 300], True), ([-70, 150, 300], [0, 150, 300], True),
    ([0, 150, 300, 0, 0], [0, 150, 300], False),            # ends before it starts: empty
    ([0, 300, 0, 300, 0, 300], None, False)])               # overlapping: more chunks than the workspaces have rows
def test_boundaries_only_the_device_knows(op, bounds, same, report):
    """Boundaries outside of the batch that the host cannot see are clipped and reported; whatever they are, the kernels stay
    inside their buffers."""
    from mcore_bridge_b200.ops import _lib
    from mcore_bridge_b200.ops.gdn import chunk_gated_delta_rule, l2norm, simple_gla
    (q, k, v, dy), gen = _inputs(300, 2, 64, 7)
    q, k = l2norm(q), l2norm(k)
    g, beta = -torch.rand(300, 2, generator=gen, device=DEV), torch.rand(300, 2, generator=gen, device=DEV)

    def run(cu):
        leaves = [t.detach().requires_grad_() for t in (q, k, v)]
        args = (-torch.rand(2, device=DEV).fill_(0.1),) if op == 'gla' else (g, beta)
        o = (simple_gla if op == 'gla' else chunk_gated_delta_rule)(*leaves, *args, cu)
        return [o, *torch.autograd.grad(o, leaves, dy)]

    _lib.check_status()
    out = run(torch.tensor(bounds, dtype=torch.int32, device=DEV))
    if report:
        with pytest.raises(_lib.KernelError, match='bad argument'):
            _lib.check_status()
    if same is not None:
        for a, b in zip(out, run(torch.tensor([[c, -1] for c in same], dtype=torch.int32, device=DEV)[:, 0])):
            assert torch.equal(a, b)
    _lib.check_status()


@pytest.mark.parametrize('op', ['gla', 'rule'])
def test_views_off_a_16_byte_boundary_give_the_same_bits(op):
    from mcore_bridge_b200.ops.gdn import chunk_gated_delta_rule, l2norm, simple_gla
    (q, k, v, dy), gen = _inputs(150, 2, 64, 8)
    g, beta = -torch.rand(150, 2, generator=gen, device=DEV), torch.rand(150, 2, generator=gen, device=DEV)

    def shifted(t):
        return torch.empty(t.numel() + 8, dtype=t.dtype, device=DEV)[1:t.numel() + 1].view(t.shape).copy_(t)

    def run(lay):
        leaves = [lay(t).requires_grad_() for t in (l2norm(q), l2norm(k), v)]
        o = simple_gla(*leaves, -beta[0]) if op == 'gla' else chunk_gated_delta_rule(*leaves, lay(g), lay(beta))
        return [o, *torch.autograd.grad(o, leaves, lay(dy))]

    for a, b in zip(run(torch.clone), run(shifted)):
        assert torch.equal(a, b)


@pytest.mark.parametrize('d', [64, 128])
@pytest.mark.parametrize('decays,key', [((0.05, 8.0), 1.0), ((1e-5, 0.0), 1.0), ((30.0, 100.0), 1.0), ((-500.0, -50.0), 1.0),
                                        ((0.3, 0.02), 1.35)])
def test_gated_delta_rule_fp32_gradients(decays, key, d):
    """dg and dbeta are fp32 results of fp32 arithmetic: no, weak and strong decays, single tokens that forget everything
    (negative: one token in twenty), and keys longer than 1, for which the chunk's inverse grows."""
    from mcore_bridge_b200.ops.gdn import chunk_gated_delta_rule, l2norm
    T, h, cuts = 400, 2, [150]
    (q, k, v, dy), gen = _inputs(T, h, d, 9)
    q, k = l2norm(q), (l2norm(k).float() * key).bfloat16()
    rate = torch.tensor(decays, device=DEV)
    g = -torch.rand(T, h, generator=gen, device=DEV) * rate.abs()
    g = torch.where((rate < 0) & (torch.rand(T, h, generator=gen, device=DEV) > 0.05), g * 1e-4, g)
    beta = torch.rand(T, h, generator=gen, device=DEV)
    cu = torch.tensor([0] + cuts + [T], dtype=torch.int32, device=DEV)
    leaves = [t.requires_grad_() for t in (q, k, v, g, beta)]
    got = torch.autograd.grad(chunk_gated_delta_rule(*leaves, cu), leaves, dy)[3:]
    wide = [t.detach().double().requires_grad_() for t in leaves]
    want = torch.autograd.grad(_delta_rule(*wide, _spans(T, cuts)), wide, dy.double())[3:]
    # sums of at most 2 d products, each cut at most once per 16 of them at 2^-24: 16 cuts = 2^-20, were they all one way
    for a, b in zip(got, want):
        assert _rel(a, b) < 2 ** -20


def test_gated_delta_rule_without_writes():
    """beta = 0 writes nothing: zero results and state, and the gradient of beta that the unwritten value would have had."""
    from mcore_bridge_b200.ops.gdn import chunk_gated_delta_rule, l2norm
    T = 150
    (q, k, v, dy), gen = _inputs(T, 2, 64, 10)
    q, k, g = l2norm(q), l2norm(k), -torch.rand(T, 2, generator=gen, device=DEV) * 0.1
    beta = torch.rand(T, 2, generator=gen, device=DEV)
    beta[:, 0] = 0
    beta[::3, 1] = 0
    leaves = [t.requires_grad_() for t in (q, k, v, g, beta)]
    o = chunk_gated_delta_rule(*leaves)
    got = torch.autograd.grad(o, leaves, dy)
    assert (o[:, 0] == 0).all() and (got[3][:, 0] == 0).all()
    wide = [t.detach().double().requires_grad_() for t in leaves]
    want = torch.autograd.grad(_delta_rule(*wide, [(0, T)]), wide, dy.double())
    assert _rel(got[3], want[3]) < 2 ** -20 and _rel(got[4], want[4]) < 2 ** -20
    for a, b in zip(got[:3], want[:3]):
        assert _rel(a, b) < 2 ** -8


@pytest.mark.parametrize('T,d,lengths', [(64, 64, [4]), (64, 64, [5, 3]), (160, 128, [16]), (160, 128, [15]),
                                         (300, 64, [1]), (2100, 64, [40, 1, 1, 1, 1, 1]), (700, 128, [130, 0, 2, 3, 1]),
                                         (1700, 64, [17, 16]), (5200, 64, [1, 2, 3, 150, 0, 1])])
def test_simple_gla_short_sequences(T, d, lengths):
    """On both sides of the line between the token and the chunk kernels (16 tokens a sequence on average), more than the 64
    sequences one step of the chunk search reads a lane at a time, and empty ones."""
    from mcore_bridge_b200.ops.gdn import simple_gla
    ends, n = [], 0
    while not ends or ends[-1] < T:
        ends.append(min(T, (ends[-1] if ends else 0) + lengths[n % len(lengths)]))
        n += 1
    (q, k, v, dy), _ = _inputs(T, 2, d, 11)
    decay = -torch.tensor([0.02, 0.5], device=DEV)
    leaves = [t.requires_grad_() for t in (q, k, v)]
    o = simple_gla(*leaves, decay, torch.tensor([0] + ends, dtype=torch.int32, device=DEV))
    grads = torch.autograd.grad(o, leaves, dy)
    wide = [t.detach().double().requires_grad_() for t in leaves]
    seq = torch.bucketize(torch.arange(T, device=DEV), torch.tensor(ends, device=DEV), right=True)
    n = torch.arange(T, device=DEV, dtype=torch.float64)
    gap = n[:, None] - n[None]
    mix = torch.exp(decay.double()[:, None, None] * gap.clamp(min=0)) * (gap >= 0) * (seq[:, None] == seq[None]) * d ** -0.5
    ref = torch.einsum('hij,jhd->ihd', torch.einsum('ihd,jhd->hij', wide[0], wide[1]) * mix, wide[2])
    for a, b in zip([o, *grads], [ref, *torch.autograd.grad(ref, wide, dy.double())]):
        assert _rel(a, b) < 2 ** -8


@pytest.mark.parametrize('T,cuts', [(200, []), (200, [130]), (40, [10, 20, 30])])
def test_simple_gla_that_forgets_everything(T, cuts):
    """decay = -inf: exp(-inf) = 0, every token sees itself alone."""
    from mcore_bridge_b200.ops.gdn import simple_gla
    (q, k, v, dy), _ = _inputs(T, 2, 64, 12)
    leaves = [t.requires_grad_() for t in (q, k, v)]
    decay = torch.tensor([-float('inf'), -200.0], device=DEV)       # exp(-200) is zero in fp32 too
    o = simple_gla(*leaves, decay, torch.tensor([0] + cuts + [T], dtype=torch.int32, device=DEV))
    grads = torch.autograd.grad(o, leaves, dy)
    wide = [t.detach().double().requires_grad_() for t in leaves]
    ref = (wide[0] * wide[1]).sum(-1, keepdim=True) * 64 ** -0.5 * wide[2]
    for a, b in zip([o, *grads], [ref, *torch.autograd.grad(ref, wide, dy.double())]):
        assert _rel(a, b) < 2 ** -8


def test_gdn_inputs_differentiate_twice():
    """With ``create_graph`` the gradient comes from torch operations: same values, and differentiable again."""
    from mcore_bridge_b200.ops.attention_cuda import seq_start_from_cu
    from mcore_bridge_b200.ops.gdn import gdn_inputs
    gen = torch.Generator(device=DEV).manual_seed(13)
    T, d = 40, 64
    proj = torch.randn(T, 2 * (2 * d + 4 * d + 4), generator=gen, device=DEV).bfloat16()
    w = (torch.randn(2 * 4 * d, 4, generator=gen, device=DEV) * 0.5).bfloat16()
    leaves = [t.requires_grad_() for t in (proj, w, *(torch.randn(4, generator=gen, device=DEV).bfloat16() for _ in range(2)))]
    out = gdn_inputs(*leaves, seq_start_from_cu(torch.tensor([0, 13, T], device=DEV), T, DEV), 2, 2, d)
    cot = [torch.randn(t.shape, generator=gen, device=DEV).to(t.dtype) for t in out]
    first = torch.autograd.grad(out, leaves, cot, retain_graph=True)
    again = torch.autograd.grad(out, leaves, cot, create_graph=True)
    for a, b in zip(first, again):
        assert _rel(a, b.double()) < 2 ** -7
    # g = -exp(A) softplus(a + dt): its second derivative by A is g itself
    second = torch.autograd.grad(again[2], leaves[2], torch.ones_like(again[2]), retain_graph=True)[0]
    assert _rel(second, (out[4].detach() * cot[4]).sum(0).double()) < 2 ** -7
    assert all(torch.isfinite(t).all() and (t != 0).any()
               for t in torch.autograd.grad(again[0].float().square().sum(), leaves))


def test_gated_delta_rule_with_hundreds_of_sequences():
    """More sequences than one step of the chunk search reads (256), short, empty and of more than a chunk."""
    from mcore_bridge_b200.ops.gdn import chunk_gated_delta_rule, l2norm
    lengths = ([1, 2, 0, 1] * 80 + [70])[:321]
    ends = torch.tensor(lengths).cumsum(0)
    T = int(ends[-1])
    (q, k, v, dy), gen = _inputs(T, 2, 64, 14)
    q, k = l2norm(q), l2norm(k)
    g, beta = -torch.rand(T, 2, generator=gen, device=DEV), torch.rand(T, 2, generator=gen, device=DEV)
    leaves = [t.requires_grad_() for t in (q, k, v, g, beta)]
    o = chunk_gated_delta_rule(*leaves, torch.cat([torch.zeros(1), ends]).int().to(DEV))
    grads = torch.autograd.grad(o, leaves, dy)
    wide = [t.detach().double().requires_grad_() for t in leaves]
    ref = _delta_rule(*wide, _spans(T, ends[:-1].tolist()))
    for a, b in zip([o, *grads], [ref, *torch.autograd.grad(ref, wide, dy.double())]):
        assert _rel(a, b) < (2 ** -8 if a.dtype == torch.bfloat16 else 2 ** -20)


@pytest.mark.parametrize('T,h,cuts', [(1300, 16, [1, 130, 130, 700]), (1300, 16, list(range(100, 1300, 100))),
                                      (130, 150, []), (257, 80, [129])])
def test_simple_gla_one_result_per_block(T, h, cuts):
    """More chunks x heads than SMs take kernels with one result a block, half of the heads at a time do not: equal bits."""
    from mcore_bridge_b200.ops.gdn import simple_gla
    tensors, gen = _inputs(T, h, 128, 3)
    decay = -torch.rand(h, generator=gen, device=DEV)
    cu = torch.tensor([0] + cuts + [T], dtype=torch.int32, device=DEV)

    def run(s):
        leaves = [t[:, s].contiguous().requires_grad_() for t in tensors[:3]]
        o = simple_gla(*leaves, decay[s].contiguous(), cu)
        return [o.detach(), *torch.autograd.grad(o, leaves, tensors[3][:, s].contiguous())]

    parts = [run(slice(0, h // 2)), run(slice(h // 2, h))]
    for got, *want in zip(run(slice(0, h)), *parts):
        assert torch.equal(got, torch.cat(want, dim=1))


@pytest.mark.parametrize('T,d,cuts', [(300, 64, [128, 130, 256]), (400, 128, [5, 127, 129, 380]), (129, 64, [128]),
                                      (1000, 128, list(range(7, 1000, 25))), (520, 64, [0, 384, 384, 500])])
def test_simple_gla_tiles_shared_by_sequences(T, d, cuts):
    """Sequences that begin and end anywhere in the tiles of 128 tokens, fewer and more of them than edges between tiles.  What
    is infinite in one sequence stays there: every other token has the bits it has without it."""
    from mcore_bridge_b200.ops.gdn import simple_gla
    (q, k, v, dy), _ = _inputs(T, 2, d, 21)
    decay = -torch.tensor([0.02, 0.5], device=DEV)
    cu = torch.tensor([0] + cuts + [T], dtype=torch.int32, device=DEV)

    def run(*tensors):
        leaves = [t.detach().requires_grad_() for t in tensors[:3]]
        o = simple_gla(*leaves, decay, cu)
        return [o.detach(), *torch.autograd.grad(o, leaves, tensors[3])]

    clean = run(q, k, v, dy)
    wide = [t.double().requires_grad_() for t in (q, k, v)]
    out = []
    for s, e in _spans(T, cuts):
        n = torch.arange(e - s, device=DEV, dtype=torch.float64)
        gap = n[:, None] - n[None]
        mix = torch.exp(decay.double()[:, None, None] * gap.clamp(min=0)) * (gap >= 0) * d ** -0.5
        out.append(torch.einsum('hij,jhd->ihd', torch.einsum('ihd,jhd->hij', wide[0][s:e], wide[1][s:e]) * mix, wide[2][s:e]))
    ref = torch.cat(out)
    for a, b in zip(clean, [ref, *torch.autograd.grad(ref, wide, dy.double())]):
        assert _rel(a, b) < 2 ** -8
    first, last = max(_spans(T, cuts), key=lambda s: s[1] - s[0])
    hit = [t.clone() for t in (q, k, v, dy)]
    for t, value in zip(hit, (float('inf'), float('nan'), -float('inf'), float('inf'))):
        t[(first + last) // 2, :, 3] = value
    others = torch.ones(T, dtype=torch.bool, device=DEV)
    others[first:last] = False
    for a, b in zip(run(*hit), clean):
        assert torch.equal(a[others], b[others])
        assert not a[first:last].isfinite().all()


@pytest.mark.parametrize('T,d,lengths', [(64, 64, [13]), (2048, 128, [12]), (2047, 64, [8, 3, 17]), (1000, 128, [15])])
def test_simple_gla_short_sequences_in_full_fp32_precision(T, d, lengths):
    """fp32 sums of d products are off by about 2^-25 sqrt(d) < 2^-21 of themselves, bf16 results 2^-8 .. 2^-7 apart: they are the
    exact ones' nearest but for 2^-12 of them.  Operands of 16 bits would move eight times as many."""
    from mcore_bridge_b200.ops.gdn import simple_gla
    ends, n, h = [0], 0, 32
    while ends[-1] < T:
        ends.append(min(T, ends[-1] + lengths[n % len(lengths)]))
        n += 1
    (q, k, v, dy), _ = _inputs(T, h, d, 31)
    decay = -(2.0 ** (-8.0 * torch.arange(1, h + 1, device=DEV) / h))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    o = simple_gla(*leaves, decay, torch.tensor(ends, dtype=torch.int32, device=DEV))
    grads = torch.autograd.grad(o, leaves, dy)
    wide = [t.detach().double().requires_grad_() for t in leaves]
    out = []
    for s, e in zip(ends[:-1], ends[1:]):
        n = torch.arange(e - s, device=DEV, dtype=torch.float64)
        gap = n[:, None] - n[None]
        mix = torch.exp(decay.double()[:, None, None] * gap.clamp(min=0)) * (gap >= 0) * d ** -0.5
        out.append(torch.einsum('hij,jhd->ihd', torch.einsum('ihd,jhd->hij', wide[0][s:e], wide[1][s:e]) * mix, wide[2][s:e]))
    ref = torch.cat(out)
    for a, b in zip([o, *grads], [ref, *torch.autograd.grad(ref, wide, dy.double())]):
        assert (a != b.bfloat16()).double().mean() < 2 ** -11


@pytest.mark.parametrize('T,d,cuts,at', [(40, 64, [], 17), (128, 128, [], 100), (300, 64, [], 130), (400, 128, [128], 250),
                                         (64, 128, list(range(8, 64, 8)), 21), (300, 64, [20], 290)])
def test_simple_gla_what_is_not_finite_stays_with_the_tokens_that_see_it(T, d, cuts, at):
    """One infinite channel of one token: the other results of its sequence have the bits they have without it."""
    from mcore_bridge_b200.ops.gdn import simple_gla
    tensors, _ = _inputs(T, 2, d, 23)
    decay = -torch.tensor([0.02, 0.001], device=DEV)
    cu = torch.tensor([0] + cuts + [T], dtype=torch.int32, device=DEV)

    def run(tensors):
        leaves = [t.detach().requires_grad_() for t in tensors[:3]]
        o = simple_gla(*leaves, decay, cu)
        return [o.detach(), *torch.autograd.grad(o, leaves, tensors[3])]

    clean = run(tensors)
    first, last = next(s for s in _spans(T, cuts) if s[0] <= at < s[1])
    t, c = torch.arange(T, device=DEV), 3
    own, later, earlier = t == at, (t >= at) & (t < last), (t <= at) & (t >= first)
    channel = torch.zeros(d, dtype=torch.bool, device=DEV)
    channel[c] = True
    none, row = torch.zeros(T, d, dtype=torch.bool, device=DEV), torch.ones(d, dtype=torch.bool, device=DEV)

    def where(rows, columns):
        return rows[:, None] & columns[None]

    # of q, k, v and dy: the parts of o, dq, dk and dv it enters
    reach = [(where(own, row), none, where(earlier, channel), where(earlier, row)),
             (where(later, row), where(later, channel), none, where(own, row)),
             (where(later, channel), where(later, row), where(own, row), none),
             (none, where(own, row), where(earlier, row), where(earlier, channel))]
    for i, value in enumerate((float('inf'), float('nan'), -float('inf'), float('inf'))):
        hit = [x.clone() for x in tensors]
        hit[i][at, :, c] = value
        for a, b, r in zip(run(hit), clean, reach[i]):
            r = r[:, None].expand(a.shape)
            assert torch.equal(a[~r], b[~r])
            assert not a[r].isfinite().any()
