"""The operations whose autograd nodes are native: what torch's machinery expects of a node (shapes, gradients that are not wanted,
saved-tensor hooks, in-place checks, second passes, `main_grad`), and the transforms they refuse."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16 = 'cuda', torch.bfloat16


def _rand(*shape, seed=1, scale=1.0):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=gen, device=DEV) * scale).to(BF16)


def _ops():
    from mcore_bridge_b200.ops import fused_mlp
    from mcore_bridge_b200.ops.attention import attention
    from mcore_bridge_b200.ops.linear import linear
    from mcore_bridge_b200.ops.norm import rmsnorm
    from mcore_bridge_b200.ops.rope import qkv_split_norm_rope
    cu = torch.tensor([0, 30, 70], dtype=torch.int32, device=DEV)
    return dict(
        linear=(lambda x, w, b: linear(x, w, b), [_rand(70, 64), _rand(96, 64, seed=2), _rand(96, seed=3)]),
        linear3=(lambda x, w: linear(x, w), [_rand(2, 35, 64), _rand(96, 64, seed=2)]),
        rmsnorm=(lambda x, w: rmsnorm(x, w), [_rand(5, 14, 64), _rand(64, seed=2)]),
        norm_linear=(lambda x, l, w: fused_mlp.norm_linear(x, l, w, 1e-6, False),
                     [_rand(2, 35, 64), _rand(64, seed=2), _rand(96, 64, seed=3)]),
        glu_linear=(lambda h, w: fused_mlp.glu_linear(h, w, 0, 0.0, 0.0), [_rand(2, 35, 128), _rand(96, 64, seed=2)]),
        qkv=(lambda x, a, b: torch.cat([t.reshape(70, -1) for t in qkv_split_norm_rope(x, a, b, None, None, 2, 2, 64)[:3]], -1),
             [_rand(70, 512), _rand(64, seed=2), _rand(64, seed=3)]),
        attention=(lambda q, k, v: attention(q, k, v, cu, 40), [_rand(70, 4, 64), _rand(70, 2, 64, seed=2), _rand(70, 2, 64, seed=3)]),
        sinks=(lambda q, k, v, s: attention(q, k, v, cu, 40, sinks=s),
               [_rand(70, 4, 64), _rand(70, 2, 64, seed=2), _rand(70, 2, 64, seed=3), _rand(4, seed=4)]))


NAMES = ['linear', 'linear3', 'rmsnorm', 'norm_linear', 'glu_linear', 'qkv', 'attention', 'sinks']


@pytest.mark.parametrize('name', NAMES)
def test_a_node_behaves_as_one_of_torch(name):
    fn, inputs = _ops()[name]
    leaves = [t.clone().requires_grad_() for t in inputs]
    y = fn(*leaves)
    dy = torch.randn_like(y)
    want = torch.autograd.grad(y, leaves, dy, retain_graph=True)
    for g, t in zip(want, leaves):
        assert g.shape == t.shape and g.dtype == t.dtype and g.isfinite().all()
    for a, b in zip(torch.autograd.grad(y, leaves, dy), want):          # the same bits again, then the graph is gone
        assert torch.equal(a, b)
    with pytest.raises(RuntimeError, match='second time'):
        torch.autograd.grad(y, leaves, dy)
    with torch.no_grad():
        assert torch.equal(fn(*leaves), y) and not fn(*leaves).requires_grad
    # one input at a time wants a gradient: the others' come out as before where they are wanted
    for i in range(len(inputs)):
        some = [t.clone().requires_grad_(j == i) for j, t in enumerate(inputs)]
        assert torch.equal(torch.autograd.grad(fn(*some), [some[i]], dy)[0], want[i])
    # an expanded gradient, and hooks that replace what is saved
    packed = []

    def pack(t):
        packed.append(t)
        return t.cpu() if t.is_cuda else t

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.to(DEV)):
        z = fn(*leaves)
    assert packed
    for a, b in zip(torch.autograd.grad(z, leaves, dy), want):
        assert torch.equal(a, b)
    ones = torch.autograd.grad(fn(*leaves).sum(), leaves)
    for a, b in zip(ones, torch.autograd.grad(fn(*leaves), leaves, torch.ones_like(dy))):
        assert torch.equal(a, b)
    # a saved input that changes in place is noticed
    last = [t.clone().requires_grad_() for t in inputs]
    moved = [t * 1 for t in last]
    z = fn(*moved)
    with torch.no_grad():
        for t in moved:
            t.add_(1)
    with pytest.raises(RuntimeError, match='inplace'):
        torch.autograd.grad(z, last, dy)


@pytest.mark.parametrize('name', NAMES)
def test_transforms_are_refused(name):
    fn, inputs = _ops()[name]
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.vmap(lambda t: fn(t, *inputs[1:]))(torch.stack([inputs[0]] * 2))
    import torch.autograd.forward_ad as fw
    with fw.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        fn(fw.make_dual(inputs[0], torch.ones_like(inputs[0])), *inputs[1:])


@pytest.mark.parametrize('name,at', [('linear', 1), ('linear3', 1), ('norm_linear', 2), ('glu_linear', 1)])
def test_weight_gradients_go_where_the_optimizer_wants_them(name, at):
    fn, inputs = _ops()[name]
    leaves = [torch.nn.Parameter(t.clone()) for t in inputs]
    dy = torch.randn_like(fn(*leaves))
    want = torch.autograd.grad(fn(*leaves), leaves, dy)
    w, calls = leaves[at], []
    w.main_grad = torch.ones(w.shape, device=DEV)
    w.grad_ready_hook = lambda: calls.append(w.main_grad.clone())
    fn(*leaves).backward(dy)
    assert w.grad is None and len(calls) == 1 and torch.equal(calls[0], w.main_grad)
    # fp32 sum of the product that was rounded to bf16 before: half a unit in the last place of 8 bits
    assert ((w.main_grad - 1) - want[at].float()).abs().max() <= 2 ** -8 * want[at].float().abs().max() + 1e-5
    for i, t in enumerate(leaves):
        assert i == at or torch.equal(t.grad, want[i])

    def broken():
        raise ValueError('not now')

    w.grad_ready_hook = broken
    with pytest.raises(ValueError, match='not now'):
        fn(*leaves).backward(dy)


def test_outputs_nobody_uses():
    from mcore_bridge_b200.ops.rope import qkv_split_norm_rope
    x = _rand(70, 512).requires_grad_()
    q, k, v, gate = qkv_split_norm_rope(x, None, None, None, None, 2, 2, 64)
    assert gate is None
    dx = torch.autograd.grad(k, x, torch.ones_like(k))[0].view(70, 2, 4, 64)
    assert (dx[:, :, 2] == 1).all() and (dx[:, :, :2] == 0).all() and (dx[:, :, 3] == 0).all()


@pytest.mark.parametrize('shape,n,k', [((70,), 96, 64), ((2, 35), 104, 64), ((300,), 512, 128), ((1, 129), 264, 72)])
def test_residuals_are_added_as_by_an_addition(shape, n, k):
    """The same bits as a sum of its own, in the product's epilogue (also where the kernel does not take the residual: 104 columns,
    off their boundary) and in the norm's backward pass."""
    from mcore_bridge_b200.ops import fused_mlp
    from mcore_bridge_b200.ops.linear import linear
    x, h, w, v, ln = (_rand(*s, seed=i) for i, s in enumerate([(*shape, k), (*shape, 2 * k), (n, k), (k, k), (k,)]))
    bias, res = _rand(n, seed=7), _rand(*shape, n, seed=8) if n != 104 else _rand(*shape, n + 1, seed=8)[..., 1:]
    dy = _rand(*shape, n, seed=9)
    for first, fused, apart in [
            (x, lambda x, w, b, r: linear(x, w, b, residual=r), lambda x, w, b, r: r + linear(x, w, b)),
            (h, lambda h, w, b, r: fused_mlp.glu_linear(h, w, 0, 0.0, 0.0, r),
             lambda h, w, b, r: r + fused_mlp.glu_linear(h, w, 0, 0.0, 0.0))]:
        leaves = [t.detach().requires_grad_() for t in (first, w, bias, res)]
        a, b = fused(*leaves), apart(*leaves)
        assert torch.equal(a, b)
        for g, e in zip(torch.autograd.grad(a, leaves, dy, allow_unused=True), torch.autograd.grad(b, leaves, dy, allow_unused=True)):
            assert (g is None and e is None) or torch.equal(g, e)
        with torch.no_grad():
            assert torch.equal(fused(*leaves), a)

    leaves = [t.clone().requires_grad_() for t in (x, ln, v)]
    dk = _rand(*shape, k, seed=10)

    def block(keep):
        if keep:
            y, kept = fused_mlp.norm_linear(*leaves, 1e-6, False, True)
        else:
            y, kept = fused_mlp.norm_linear(*leaves, 1e-6, False), leaves[0]
        return y, kept

    y, kept = block(True)
    assert torch.equal(kept, x) and torch.equal(y, block(False)[0])
    got = torch.autograd.grad(block(True), leaves, [dk, dk])
    want = torch.autograd.grad(block(False), leaves, [dk, dk])
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert torch.equal(torch.autograd.grad(block(True)[1], leaves[0], dk)[0], dk)     # the residual alone
    assert torch.equal(torch.autograd.grad(block(True)[0], leaves[0], dk)[0], torch.autograd.grad(block(False)[0], leaves[0], dk)[0])


def test_residual_of_a_wide_row():
    """More columns than the norm's backward kernel has registers for: the gradients are added behind it."""
    from mcore_bridge_b200.ops import fused_mlp
    x, ln, v = _rand(5, 8200, seed=1), _rand(8200, seed=2), _rand(64, 8200, seed=3, scale=0.01)
    leaves = [t.requires_grad_() for t in (x, ln, v)]
    dy, dk = _rand(5, 64, seed=4), _rand(5, 8200, seed=5)
    got = torch.autograd.grad(fused_mlp.norm_linear(*leaves, 1e-6, False, True), leaves, [dy, dk])
    want = torch.autograd.grad(fused_mlp.norm_linear(*leaves, 1e-6, False), leaves, dy)
    assert torch.equal(got[0], want[0] + dk) and torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])


@pytest.mark.parametrize('name', ['linear', 'glu_linear'])
@pytest.mark.parametrize('shape', [(70,), (2, 35)])
def test_a_residual_of_another_type(name, shape):
    """An fp32 residual under bf16 operands: fp32 results, and gradients as of an addition."""
    from mcore_bridge_b200.ops import _lib, fused_mlp
    x, w, res = _rand(*shape, 128), _rand(96, 128 if name == 'linear' else 64, seed=2), _rand(*shape, 96, seed=3).float()
    nat = _lib.native()

    def op(x, w, r):
        return nat.linear(x, w, None, False, r) if name == 'linear' else fused_mlp.glu_linear(x, w, 0, 0.0, 0.0, r)

    leaves = [t.requires_grad_() for t in (x, w, res)]
    a, b = op(*leaves), res + op(x, w, None)
    assert a.dtype == torch.float32 and torch.equal(a, b)
    dy = torch.randn_like(a)
    for g, e in zip(torch.autograd.grad(a, leaves, dy), torch.autograd.grad(b, leaves, dy)):
        assert g.dtype == e.dtype and torch.equal(g, e)


def test_a_feed_forward_block_under_an_fp32_residual_stream():
    from mcore_bridge_b200.layers.mlp import MLP
    from mcore_bridge_b200.train.presets import model_config
    with torch.device(DEV):
        mlp = MLP(model_config('qwen3_tiny', bf16=True), fuse_input_norm=True)
    for i, p in enumerate(mlp.parameters()):
        with torch.no_grad():
            p.copy_(_rand(*p.shape, seed=i, scale=0.02))
    x = _rand(50, mlp.config.hidden_size).float().requires_grad_()
    leaves, dy = [x, *mlp.parameters()], torch.randn(50, mlp.config.hidden_size, device=DEV)
    a, b = mlp(x, True), x + mlp(x)
    assert a.dtype == torch.float32 and torch.equal(a, b)
    for g, e in zip(torch.autograd.grad(a, leaves, dy), torch.autograd.grad(b, leaves, dy)):
        assert g.dtype == e.dtype and torch.equal(g, e)
