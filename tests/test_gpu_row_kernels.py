"""Row-wise kernels at the edges of how they walk: one vector, a pair of heads or of rows at a time, with the next in flight."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def _rand(*shape, seed=0):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, generator=gen, device=DEV).bfloat16()


@pytest.mark.parametrize('rows,F', [(1, 8), (3, 264), (33, 256), (700, 104), (5, 8192)])
@pytest.mark.parametrize('kind,clamp,offset', [('swiglu', 0.0, 0.0), ('quick_geglu', 2.0, 1.0), ('geglu_tanh', 0.0, 0.0)])
def test_gated_activation(rows, F, kind, clamp, offset):
    from mcore_bridge_b200.ops.activation import glu, glu_ref
    x, dy = _rand(rows, 2 * F), _rand(rows, F, seed=1)
    probs = torch.rand(rows, device=DEV)
    for pr in (None, probs):
        leaves = [t.clone().requires_grad_() for t in (x, pr) if t is not None]
        got = torch.autograd.grad(glu(leaves[0], kind, leaves[1] if pr is not None else None, clamp, offset), leaves, dy)
        out = glu(x, kind, pr, clamp, offset)
        wide = [t.detach().double().requires_grad_() for t in leaves]
        ref = glu_ref(wide[0], kind, wide[1] if pr is not None else None, clamp, offset)
        want = torch.autograd.grad(ref, wide, dy.double())
        # rounded once; fp32: sums of F products, and the hardware's tanh, within 2^-11, enters g (1 + tanh) / 2
        tanh = 2 ** -12 * (x[:, :F] * x[:, F:] * dy).double().abs().sum(-1).norm() if kind == 'geglu_tanh' else 0.0
        for a, b in zip([out, *got], [ref, *want]):
            assert _rel(a, b) < (2 ** -8 if a.dtype == torch.bfloat16 else 2 ** -17 + tanh / b.norm())


@pytest.mark.parametrize('rows,H', [(593, 104), (1190, 2048), (601, 4096), (300, 8192), (1201, 1024)])
def test_norm_backward_with_the_next_rows_in_flight(rows, H):
    # more rows than the grid takes at once: every row has the bits it has alone, with and without the residual's gradient
    from mcore_bridge_b200.ops import _lib
    lib, ptr, ll = _lib.lib(), lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr()), ctypes.c_longlong
    x, dy, res, w = _rand(rows, H), _rand(rows, H, seed=1), _rand(rows, H, seed=2), _rand(H, seed=3)
    rstd = torch.rsqrt(x.float().pow(2).mean(-1) + 1e-6)

    def backward(first, last, res, with_y):
        n = last - first
        part = torch.empty(lib.mcb_rmsnorm_bwd_partial_rows(ll(n), H), H, device=DEV)
        d, dx, dw = dy[first:last].clone(), torch.empty_like(dy[first:last]), torch.empty_like(w)
        f = lib.mcb_rmsnorm_bwd_det_y if with_y else lib.mcb_rmsnorm_bwd_det
        assert f(ptr(d), ptr(x[first:]), ptr(w), ptr(rstd[first:]), ptr(None if res is None else res[first:]), ptr(dx), ptr(dw),
                 1, ptr(part), ll(n), H, ll(H), ctypes.c_float(1e-6), 0, _lib.stream_ptr()) == 0
        return dx, dw, d

    dx, dw, _ = backward(0, rows, None, False)
    for first, last in ((0, 1), (0, 100), (rows - 101, rows)):
        assert torch.equal(backward(first, last, None, False)[0], dx[first:last])
    dxr, dwr, y = backward(0, rows, res, True)
    assert torch.equal(dxr, dx + res) and torch.equal(dwr, dw)
    assert _rel(y, x.double() * rstd.double()[:, None] * w.double()) < 2 ** -8
    wide = x.double().requires_grad_(), w.double().requires_grad_()
    ref = wide[0] * torch.rsqrt(wide[0].pow(2).mean(-1, keepdim=True) + 1e-6) * wide[1]
    for a, b in zip((dx, dw), torch.autograd.grad(ref, wide, dy.double())):
        assert _rel(a, b) < 2 ** -8


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason='needs 2 GPUs')
def test_norm_backward_on_one_device_after_the_other():
    from mcore_bridge_b200.ops.norm import rmsnorm
    grads = []
    for index in (0, 1):
        with torch.cuda.device(index):
            x, w = (t.to(index).requires_grad_() for t in (_rand(1190, 2048), _rand(2048, seed=3)))
            grads.append(torch.autograd.grad(rmsnorm(x, w), [x, w], _rand(1190, 2048, seed=1).to(index)))
    for a, b in zip(*grads):
        assert torch.equal(a.cpu(), b.cpu())


@pytest.mark.parametrize('rows,H', [(1, 8), (9500, 136), (20000, 256), (2500, 264), (1300, 4096), (1200, 8192)])
@pytest.mark.parametrize('zero_centered', [False, True])
def test_norm_forward_with_the_next_row_in_flight(rows, H, zero_centered):
    from mcore_bridge_b200.ops.norm import rmsnorm
    x, w = _rand(rows, H), _rand(H, seed=3)
    y = rmsnorm(x, w, 1e-6, zero_centered)
    wide = x.double()
    ref = wide * torch.rsqrt(wide.pow(2).mean(-1, keepdim=True) + 1e-6) * (w.double() + (1 if zero_centered else 0))
    assert _rel(y, ref) < 2 ** -8                                        # rounded once
    for rows_of in (slice(0, 1), slice(rows - 3, rows)):                 # every row has the bits it has alone
        assert torch.equal(rmsnorm(x[rows_of], w, 1e-6, zero_centered), y[rows_of])


@pytest.mark.parametrize('T,ng,qpg,gate', [(1, 1, 1, False), (2, 16, 3, False), (333, 1, 2, True), (7, 300, 1, False), (2500, 3, 1, False)])
@pytest.mark.parametrize('norm', [False, True])
def test_heads_of_128(T, ng, qpg, gate, norm):
    from mcore_bridge_b200.ops.rope import qkv_split_norm_rope, qkv_split_norm_rope_ref
    W = ng * (qpg * (2 if gate else 1) + 2) * 128
    cos, sin = torch.rand(T, 64, device=DEV), torch.rand(T, 64, device=DEV)
    buf = _rand(T * W + 2)
    ws = [_rand(128, seed=s) for s in (1, 2)] if norm else [None, None]

    def run(qkv, f, ws):
        leaves = [t.requires_grad_() for t in (qkv, *ws) if t is not None]
        outs = f(qkv, ws[0], ws[1], cos.to(qkv.dtype), sin.to(qkv.dtype), ng, qpg, 128, gate, False, 1e-6, False)
        outs = [t for t in outs if t is not None]
        gen = torch.Generator(device=DEV).manual_seed(5)
        seeds = [torch.randn(t.shape, generator=gen, device=DEV).bfloat16().to(t.dtype) for t in outs]
        return outs + list(torch.autograd.grad(outs, leaves, seeds))

    def single(qkv, wq, wk, cos, sin, *rest):
        return qkv_split_norm_rope(qkv, wq, wk, cos.float(), sin.float(), *rest)

    qkv = buf[:T * W].view(T, W)
    got = run(qkv.detach().clone(), single, [None if w is None else w.clone() for w in ws])
    cos, sin = cos.double(), sin.double()
    want = run(qkv.double(), qkv_split_norm_rope_ref, [None if w is None else w.double() for w in ws])
    for a, b in zip(got, want):
        assert _rel(a, b) < 2 ** -8                                      # rounded once
    cos, sin = cos.float(), sin.float()
    buf[2:] = buf[:-2].clone()                                           # four bytes from any wider boundary
    for a, b in zip(run(buf[2:].view(T, W).detach(), single, ws), got):
        assert torch.equal(a, b)


@pytest.mark.parametrize('rows,D', [(1, 128), (77, 64), (9001, 128), (5, 256), (3001, 256), (20001, 64)])
def test_gated_norm(rows, D):
    from mcore_bridge_b200.ops import gdn
    x, z, dy, w = _rand(rows, D), _rand(rows, D, seed=1), _rand(rows, D, seed=2), _rand(D, seed=3)

    def run(x, z, w, dy):
        leaves = [t.detach().requires_grad_() for t in (x, z, w)]
        y = gdn.gated_rmsnorm(*leaves, 1e-6)
        return [y, *torch.autograd.grad(y, leaves, dy)]

    wide = [t.double().requires_grad_() for t in (x, z, w)]
    ref = wide[0] * torch.rsqrt(wide[0].pow(2).mean(-1, keepdim=True) + 1e-6) * wide[2] * torch.nn.functional.silu(wide[1])
    got = run(x, z, w, dy)
    for a, b in zip(got, [ref, *torch.autograd.grad(ref, wide, dy.double())]):
        assert _rel(a, b) < 2 ** -7                                      # rounded once, and the normalised value before it
    odd = [torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape) for t in (x, z, w, dy)]      # two bytes from a wider boundary
    for i, (a, b) in enumerate(zip(run(*odd), got)):
        assert torch.equal(a, b) or (i == 3 and _rel(a, b) < 2 ** -8)    # the weight's gradient is summed with atomics


@pytest.mark.parametrize('T,k,H', [(1, 1, 8), (100, 2, 264), (7, 3, 2048), (33, 5, 512), (300, 8, 520), (9, 9, 256)])
def test_combined_rows(T, k, H):
    from mcore_bridge_b200.ops import _lib
    rows = T * k
    y, idx = _rand(rows, H), torch.zeros(T, k, dtype=torch.int32, device=DEV)
    gen = torch.Generator(device=DEV).manual_seed(4)
    sent = torch.randperm(rows, generator=gen, device=DEV).view(T, k).int()
    sent[torch.rand(T, k, generator=gen, device=DEV) < 0.1] = -1                         # entries that were not sent
    scalars, out, probs = torch.rand(rows, device=DEV), torch.empty(T, H, device=DEV).bfloat16(), torch.empty(T, k, device=DEV)
    tables = [(ctypes.c_void_p * 1)(t.data_ptr()) for t in (y, scalars)]
    assert _lib.lib().mcb_moe_combine(*tables, *map(ctypes.c_int, (1, T, k, 4, H)), _lib.ptr(idx), _lib.ptr(sent), _lib.ptr(out),
                                      _lib.ptr(probs), _lib.stream_ptr()) == 0
    want = torch.zeros(T, H, device=DEV)
    for j in range(k):
        want += torch.where(sent[:, j, None] >= 0, y[sent[:, j].clamp(min=0).long()].float(), 0.0)
    assert torch.equal(out, want.bfloat16())
    assert torch.equal(probs, torch.where(sent >= 0, scalars[sent.clamp(min=0).long()], 0.0))


@pytest.mark.parametrize('T,ng,qpg,d,gate', [(1, 2, 2, 128, False), (333, 2, 4, 128, True), (70, 3, 2, 64, False)])
def test_heads_in_columns_of_a_wider_tensor(T, ng, qpg, d, gate):
    """The gradient of such columns is dense: the bits of a contiguous copy's, and of nothing beside it."""
    from mcore_bridge_b200.ops.rope import qkv_split_norm_rope
    W = ng * (qpg * (2 if gate else 1) + 2) * d
    wide, ws = _rand(T, W + 40), [_rand(d, seed=s) for s in (1, 2)]
    cos, sin = torch.rand(T, d // 2, device=DEV), torch.rand(T, d // 2, device=DEV)

    def run(qkv):
        leaves = [qkv.detach().requires_grad_(), *(w.clone().requires_grad_() for w in ws)]
        outs = [t for t in qkv_split_norm_rope(*leaves, cos, sin, ng, qpg, d, gate, False, 1e-6, False) if t is not None]
        return outs + list(torch.autograd.grad(outs, leaves, [_rand(*t.shape, seed=5) for t in outs]))

    for a, b in zip(run(wide[:, :W]), run(wide[:, :W].clone())):
        assert a.shape == b.shape and torch.equal(a, b)


@pytest.mark.parametrize('rows,H', [(5, 104), (700, 2048), (3, 8192), (7, 8200), (300, 16384)])
def test_norm_backward_adds_a_residual_gradient_once_rounded(rows, H):
    from mcore_bridge_b200.ops import _lib
    lib, ptr, ll = _lib.lib(), lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr()), ctypes.c_longlong
    x, dy, w = _rand(rows, H), _rand(rows, H, seed=1), _rand(H, seed=3)
    wide = x.double()
    r = torch.rsqrt(wide.pow(2).mean(-1, keepdim=True) + 1e-6)
    g, xh = dy.double() * w.double(), wide * r
    dx = r * (g - xh * (g * xh).mean(-1, keepdim=True))
    res = (_rand(rows, H, seed=2) * 2 ** -6 - dx).bfloat16()           # the sum is small beside its two terms
    part = torch.empty(lib.mcb_rmsnorm_bwd_partial_rows(ll(rows), H), H, device=DEV)
    dw, acc = torch.empty_like(w), torch.zeros(H, device=DEV)
    for f, extra in ((lib.mcb_rmsnorm_bwd_det, (ptr(dw), 1, ptr(part))), (lib.mcb_rmsnorm_bwd, (ptr(acc),))):
        out = torch.empty_like(x)
        assert f(ptr(dy), ptr(x), ptr(w), None, ptr(res), ptr(out), *extra, ll(rows), H, ll(H), ctypes.c_float(1e-6), 0,
                 _lib.stream_ptr()) == 0
        # half a unit of the last of the result's 8 bits, 2^-8 of it at most, and fp32 arithmetic on terms of the size of g and of xh
        # times the mean: sums of up to 16384 terms over 256 chains, some 20 roundings of 2^-24 for the mean
        size = r * (g.abs() + xh.abs() * (g * xh).abs().mean(-1, keepdim=True))
        assert ((out.double() - (dx + res.double())).abs() <= 2 ** -8 * (dx + res.double()).abs() + 2 ** -18 * size).all()


def _odd(t):
    """The same values, contiguous, two bytes behind a 16-byte boundary."""
    return torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape)


@pytest.mark.parametrize('name', ['rmsnorm', 'norm_linear', 'glu', 'glu_linear', 'heads of 64', 'heads of 128', 'conv'])
def test_tensors_off_a_16_byte_boundary_give_the_same_bits(name):
    from mcore_bridge_b200.ops import fused_mlp, gdn
    from mcore_bridge_b200.ops.activation import glu
    from mcore_bridge_b200.ops.norm import rmsnorm
    from mcore_bridge_b200.ops.rope import qkv_split_norm_rope
    d = 128 if name == 'heads of 128' else 64
    cos, sin = torch.rand(50, d // 2, device=DEV), torch.rand(50, d // 2, device=DEV)
    x, w = _rand(50, 256), _rand(96, 256, seed=2)
    # inputs, and whether they and the results' gradients may lie anywhere: products read neither weights nor gradients that do
    fn, inputs, odd, odd_grads = {
        'rmsnorm': (rmsnorm, [x, _rand(256, seed=1)], (1, 1), (1,)),
        'norm_linear': (lambda x, l, w: fused_mlp.norm_linear(x, l, w, 1e-6, False, True), [x, _rand(256, seed=1), w], (1, 1, 0), (0, 1)),
        'glu': (glu, [x], (1,), (1,)),
        'glu_linear': (lambda h, w: fused_mlp.glu_linear(h, w, 0, 0.0, 0.0), [_rand(50, 512), w], (1, 0), (0,)),
        'conv': (lambda x, w: gdn.causal_conv1d_silu(x, w), [x, _rand(256, 4, seed=1)], (1, 1), (1,)),
    }.get(name) or (lambda x, a, b: qkv_split_norm_rope(x, a, b, cos, sin, 2, 2, d)[:3],
                    [_rand(50, 8 * d), _rand(d, seed=1), _rand(d, seed=2)], (1, 1, 1), (1, 1, 1))

    def run(lay):
        leaves = [(lay if o else torch.clone)(t).detach().requires_grad_() for t, o in zip(inputs, odd)]
        y = fn(*leaves)
        y = [y] if torch.is_tensor(y) else list(y)
        return y + list(torch.autograd.grad(y, leaves, [(lay if o else torch.clone)(_rand(*t.shape, seed=9)) for t, o in zip(y, odd_grads)]))

    for i, (a, b) in enumerate(zip(run(torch.clone), run(_odd))):
        assert torch.equal(a, b) or (name == 'conv' and i == 2 and _rel(a, b) < 2 ** -7)   # summed with atomics
