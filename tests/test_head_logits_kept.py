"""When the head keeps its logits for the backward pass."""
import pytest
import torch

from mcore_bridge_b200.ops import cross_entropy as ce


@pytest.fixture
def asked(monkeypatch):
    """The head's kernels replaced by torch; records what the forward pass wants to keep."""
    seen = []

    def keep(T, vl, H, device):
        seen.append(torch.empty(T, vl))
        return seen[-1]

    def stats(h2, weight, lab, vocab_start, logits=None):
        full = h2.float() @ weight.float().t()
        if logits is not None:
            logits.copy_(full)
        return ce._stats_torch(full, lab, vocab_start)

    monkeypatch.setattr(ce, '_head_kernel_ok', lambda h2, weight: True)
    monkeypatch.setattr(ce, '_logits_to_keep', keep)
    monkeypatch.setattr(ce, '_head_stats', stats)
    monkeypatch.setattr(ce, '_kept_dlogits', lambda *a: ce._dlogits(*a, torch.float32))
    return seen


def _operands(grad=True):
    gen = torch.Generator().manual_seed(3)
    h, w = torch.randn(6, 16, generator=gen), torch.randn(24, 16, generator=gen)
    return h.requires_grad_(grad), w.requires_grad_(grad), torch.randint(0, 24, (6,), generator=gen)


def test_a_loss_without_a_graph_keeps_nothing(asked):
    h, w, lab = _operands()
    want = torch.nn.functional.cross_entropy(h @ w.t(), lab, reduction='none')
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            assert torch.allclose(ce.fused_linear_cross_entropy(h, w, lab), want, atol=1e-5)
    frozen = _operands(grad=False)
    ce.fused_linear_cross_entropy(*frozen)
    assert not asked
    ce.fused_linear_cross_entropy(h, w, lab)
    assert len(asked) == 1
    ce.fused_linear_cross_entropy(h.detach(), w, lab)      # one of the two operands is enough
    assert len(asked) == 2


def test_the_first_pass_of_a_checkpointed_head_keeps_nothing(asked):
    from torch.utils.checkpoint import checkpoint
    h, w, lab = _operands()
    loss = checkpoint(lambda a: ce.fused_linear_cross_entropy(a, w, lab).sum(), h, use_reentrant=True)
    assert not asked
    loss.backward()
    assert len(asked) == 1                                 # the pass it is repeated in
    want = torch.autograd.grad(torch.nn.functional.cross_entropy(h @ w.t(), lab, reduction='sum'), (h, w))
    assert torch.allclose(h.grad, want[0], atol=1e-4) and torch.allclose(w.grad, want[1], atol=1e-4)


@pytest.mark.gpu
def test_a_loss_without_gradients_allocates_no_logits():
    T, V, H = 512, 32000, 1024
    h = torch.randn(T, H, device='cuda').bfloat16()
    w = (torch.randn(V, H, device='cuda') * 0.05).bfloat16().requires_grad_()
    lab = torch.randint(0, V, (T,), device='cuda')
    ce.fused_linear_cross_entropy(h, w, lab)
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            torch.cuda.reset_peak_memory_stats()
            base = torch.cuda.memory_allocated()
            ce.fused_linear_cross_entropy(h, w, lab)
            assert torch.cuda.max_memory_allocated() - base < 4 * T * V // 4


@pytest.mark.gpu
@pytest.mark.parametrize('T,V,H,chunk', [(515, 4104, 1024, 4096),      # a last column tile with 8 columns
                                         (1, 264, 1032, 4096),
                                         (1030, 2056, 1024, 600),      # two chunks
                                         (1100, 8200, 1024, 4096)])    # the gradient epilogue on CTA pairs
def test_kept_and_repeated_logits_give_the_same_bits(T, V, H, chunk):
    gen = torch.Generator(device='cuda').manual_seed(4)
    h = torch.randn(T, H, generator=gen, device='cuda').bfloat16().requires_grad_()
    w = (torch.randn(V, H, generator=gen, device='cuda') * 0.05).bfloat16().requires_grad_()
    lab = torch.randint(0, V, (T,), generator=gen, device='cuda')
    g = torch.rand(T, generator=gen, device='cuda')
    loss = ce.fused_linear_cross_entropy(h, w, lab, chunk=chunk)
    kept = torch.autograd.grad(loss, (h, w), g, retain_graph=True)
    again = torch.autograd.grad(loss, (h, w), g)
    assert torch.equal(kept[0], again[0]) and torch.equal(kept[1], again[1])
