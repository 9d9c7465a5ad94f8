"""When the head keeps its logits for the backward pass."""
import pytest
import torch

from mcore_bridge_b200.ops import cross_entropy as ce


@pytest.fixture
def asked(monkeypatch):
    """The head's kernels replaced by torch; records what the forward pass wants to keep."""
    seen = []

    def keep(T, vl, H, device, backward):
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


def test_hooks_on_saved_tensors_keep_nothing(asked):
    from torch.utils.checkpoint import checkpoint
    h, w, lab = _operands()
    want = torch.autograd.grad(torch.nn.functional.cross_entropy(h @ w.t(), lab, reduction='sum'), (h, w))
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t):
        loss = ce.fused_linear_cross_entropy(h, w, lab).sum()
    again = checkpoint(lambda a: ce.fused_linear_cross_entropy(a, w, lab).sum(), h, use_reentrant=False)
    with pytest.MonkeyPatch.context() as m:
        m.setattr(ce, '_head_kernel_ok', lambda h2, weight: False)        # the form without the head's kernels
        for x in (loss, again):
            got = torch.autograd.grad(x, (h, w))
            assert all(torch.allclose(a, b, atol=1e-4) for a, b in zip(got, want))
    assert not asked


def test_logits_are_given_back(asked, monkeypatch):
    h, w, lab = _operands()
    want = torch.autograd.grad(torch.nn.functional.cross_entropy(h @ w.t(), lab, reduction='sum'), (h, w))
    cpu = torch.device('cpu')
    loss = ce.fused_linear_cross_entropy(h, w, lab).sum()
    other = ce.fused_linear_cross_entropy(h, w, lab).sum()
    assert len(ce._kept_on(cpu)) == 2 and not ce._kept_on(torch.device('meta'))
    ce.release_kept_logits(torch.device('meta'))
    assert len(ce._kept_on(cpu)) == 2
    ce.release_kept_logits(cpu)
    assert not ce._kept_on(cpu)
    monkeypatch.setattr(ce, '_head_kernel_ok', lambda h2, weight: False)
    got = torch.autograd.grad(loss, (h, w))
    assert all(torch.allclose(a, b, atol=1e-4) for a, b in zip(got, want))
    del other
    monkeypatch.setattr(ce, '_head_kernel_ok', lambda h2, weight: True)
    loss = ce.fused_linear_cross_entropy(h, w, lab).sum()
    assert len(ce._kept_on(cpu)) == 1
    del loss                                               # a graph that is dropped gives its logits back too
    assert not ce._kept_on(cpu)


MB = 1 << 20


@pytest.fixture
def device(monkeypatch):
    """A device of 64 GB as the rule sees it; its free memory is set by the test."""
    state = dict(free=0, reserved=0, allocated=0, asked=0, capturing=False, fraction=1.0)

    def mem_get_info(dev):
        state['asked'] += 1
        return state['free'], 64 << 30

    class Native:
        memory = staticmethod(lambda index: (state['reserved'], state['allocated']))

    class Properties:
        total_memory = 64 << 30

    empty = torch.empty
    monkeypatch.setattr(torch.cuda, 'mem_get_info', mem_get_info)
    monkeypatch.setattr(torch.cuda, 'get_per_process_memory_fraction', lambda dev: state['fraction'])
    monkeypatch.setattr(torch.cuda, 'get_device_properties', lambda dev: Properties)
    monkeypatch.setattr(torch.cuda, 'is_current_stream_capturing', lambda: state['capturing'])
    monkeypatch.setattr(ce._lib, 'native', lambda: Native)
    monkeypatch.setattr(torch, 'empty', lambda *a, **k: empty(*a, **{**k, 'device': 'meta'}))
    monkeypatch.setattr(ce, '_driver_free', {})
    monkeypatch.setattr(ce, '_device_bytes', {})
    return state


def _keeps(T, vl=4096, backward=0, H=1024):
    return ce._logits_to_keep(T, vl, H, torch.device('meta'), backward) is not None


def test_logits_are_kept_only_where_memory_is_left(device):
    need, T = 16 * MB, 1024                                # T x 4096 fp32
    for free, backward, kept in [(4 * need, 0, True), (4 * need - 1, 0, False), (4 * need, 1, False),
                                 (4 * need + 100 * MB, 100 * MB, True)]:
        ce._driver_free.clear()
        device.update(free=free)
        assert _keeps(T, backward=backward) == kept
    ce._driver_free.clear()
    device.update(free=2 * need, reserved=10 * need, allocated=8 * need)     # half of it unused in the allocator
    assert _keeps(T)
    device.update(capturing=True)
    assert not _keeps(T)
    device.update(capturing=False)
    assert not _keeps(0) and not _keeps(T, vl=4100) and not _keeps(T, H=512)
    # a process that may take half of the 64 GB and has taken all but 3 buffers of that
    ce._driver_free.clear()
    device.update(fraction=0.5, free=32 << 30, reserved=(32 << 30) - 3 * need, allocated=(32 << 30) - 3 * need)
    assert not _keeps(T)


def test_large_buffers_ask_the_driver_each_time(device):
    device.update(free=8 << 30)
    for T in (1024, 1024, 1024):                            # 16 MB: one question while the allocator holds the same
        assert _keeps(T)
    assert device['asked'] == 1
    device.update(reserved=MB)
    assert _keeps(1024) and device['asked'] == 2
    assert _keeps(32768) and _keeps(32768) and device['asked'] == 4          # 512 MB


def test_all_kept_logits_together_are_bounded(device):
    device.update(free=60 << 30)
    held = []
    for _ in range(4):                                      # 512 MB each, a 32nd of the device is 2 GB
        held.append(ce._Kept(ce._logits_to_keep(32768, 4096, 1024, torch.device('meta'))))
    assert not _keeps(32768) and not _keeps(1024)
    held[0].take()
    assert _keeps(32768)


def test_backward_bytes():
    w = torch.empty(64, 8, dtype=torch.bfloat16)
    assert ce._backward_bytes(10, 16, w, True, True) == 2 * 10 * 64 + 2 * 10 * 8 + 2 * 64 * 8
    assert ce._backward_bytes(40, 16, w, False, True) == 2 * 16 * 64 + 6 * 64 * 8       # fp32 sum of the chunks, then bf16
    w.main_grad = torch.empty(64, 8)
    assert ce._backward_bytes(40, 16, w, True, True) == 2 * 16 * 64 + 2 * 40 * 8


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


@pytest.mark.gpu
def test_a_head_that_may_not_keep_its_logits(monkeypatch):
    T, V, H = 300, 4104, 1024
    gen = torch.Generator(device='cuda').manual_seed(5)
    h = torch.randn(T, H, generator=gen, device='cuda').bfloat16().requires_grad_()
    w = (torch.randn(V, H, generator=gen, device='cuda') * 0.05).bfloat16().requires_grad_()
    lab = torch.randint(0, V, (T,), generator=gen, device='cuda')

    def grads():
        loss = ce.fused_linear_cross_entropy(h, w, lab)
        return len(ce._kept_on(h.device)), torch.autograd.grad(loss.sum(), (h, w))

    n, want = grads()
    assert n == 1
    reserved, allocated = ce._lib.native().memory(h.device.index)
    assert reserved >= allocated >= h.numel() * 2 + w.numel() * 2
    monkeypatch.setattr(ce, '_memory_left', lambda device, need: 3 * need)
    n, got = grads()
    assert n == 0 and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
def test_a_model_gives_back_the_logits_of_earlier_graphs():
    from mcore_bridge_b200 import get_mcore_model
    from mcore_bridge_b200.train.presets import model_config
    cfg = model_config('qwen3_tiny', dict(num_hidden_layers=1, hidden_size=1024, intermediate_size=256,
                                          num_attention_heads=4, num_key_value_heads=2, head_dim=64, vocab_size=1024),
                       bf16=True)
    with torch.device('cuda'):
        model = get_mcore_model(cfg)[0]
    model = model.to('cuda').train()
    dev = next(model.parameters()).device
    gen = torch.Generator(device=dev).manual_seed(6)
    with torch.no_grad():
        for p in model.parameters():
            p.copy_(torch.randn(p.shape, generator=gen, device=dev) * 0.05 + (p.dim() == 1))
    ids = torch.randint(0, 1024, (1, 128), generator=gen, device=dev)
    pos = torch.arange(128, device=dev)[None]
    first = model(ids, position_ids=pos, labels=ids)
    assert len(ce._kept_on(dev)) == 1
    second = model(ids, position_ids=pos, labels=ids)
    assert len(ce._kept_on(dev)) == 1
    params = list(model.parameters())
    got, want = (torch.autograd.grad(x.sum(), params, allow_unused=True) for x in (first, second))
    assert not ce._kept_on(dev)
    assert all(torch.equal(a, b) for a, b in zip(got, want) if a is not None)
