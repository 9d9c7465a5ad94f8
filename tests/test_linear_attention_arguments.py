"""What the chunked linear-attention operators hand to their kernels, checked on the host: boundaries inside the batch,
tensors on 16-byte boundaries."""
import ctypes

import pytest
import torch

from mcore_bridge_b200.ops import _lib, gdn
from mcore_bridge_b200.utils.torch_utils import attach_host_list

T, H, D = 20, 2, 64


def _call(op, tensors, cu):
    q, k, v, g, beta = tensors
    if op == 'gla':
        return gdn.simple_gla(q, k, v, -torch.rand(H), cu)
    return gdn.chunk_gated_delta_rule(q, k, v, g, beta, cu)


def _tensors():
    gen = torch.Generator().manual_seed(0)
    return [torch.randn(T, H, D, generator=gen).bfloat16() for _ in range(3)] + [torch.rand(T, H, generator=gen)] * 2


@pytest.mark.parametrize('op', ['gla', 'rule'])
@pytest.mark.parametrize('bounds', [[0, T + 1], [0, 5, 3 * T], [-1, T]])
def test_boundaries_outside_the_batch_are_refused(monkeypatch, op, bounds):
    monkeypatch.setattr(gdn, '_cuda_ok', lambda *ts: True)       # the kernels' side of the dispatch
    with pytest.raises(ValueError, match='outside of the batch'):
        _call(op, _tensors(), torch.tensor(bounds, dtype=torch.int32))


@pytest.mark.parametrize('bounds,covered', [([0, T], True), ([0, 3, T], True), ([0, 7], False), ([2, T], False)])
def test_boundaries_become_contiguous_int32(bounds, covered):
    strided = torch.tensor([[b, -5] for b in bounds])[:, 0]
    cu, known = gdn._kernel_bounds(strided, T, torch.device('cpu'))
    assert cu.tolist() == bounds and cu.is_contiguous() and cu.dtype == torch.int32 and known is covered
    cu, known = gdn._kernel_bounds(attach_host_list(strided, strided), T, torch.device('cpu'))
    assert cu.tolist() == bounds and known is covered


class _Recorder:
    """Stands in for the CUDA library: every pointer that reaches it, by entry point."""

    def __init__(self):
        self.pointers = {}

    def __getattr__(self, name):
        def call(*args):
            self.pointers[name] = [a.value for a in args if isinstance(a, ctypes.c_void_p) and a.value]
            return 4 if name.endswith(('chunks', 'boundaries', 'partials')) else 0
        return call


def _shifted(t):
    """The same values, contiguous, one element behind a 16-byte boundary."""
    view = torch.empty(t.numel() + 8, dtype=t.dtype)[1:t.numel() + 1].view(t.shape).copy_(t)
    assert view.is_contiguous() and view.data_ptr() % 16
    return view


@pytest.mark.parametrize('op', ['gla', 'rule', 'inputs'])
def test_kernels_only_see_aligned_tensors(monkeypatch, op):
    """Contiguous views with an odd storage offset, among them the cotangents, are copied before a kernel reads them."""
    rec = _Recorder()
    monkeypatch.setattr(gdn, '_cuda_ok', lambda *ts: True)
    monkeypatch.setattr(_lib, 'lib', lambda: rec)
    monkeypatch.setattr(_lib, 'stream_ptr', lambda: ctypes.c_void_p(0))
    monkeypatch.setattr(_lib, 'status_word', lambda device=None: torch.zeros(16, dtype=torch.int32))
    q, k, v, g, beta = (_shifted(t).requires_grad_() for t in _tensors())
    if op == 'inputs':
        proj = _shifted(torch.randn(T, 2 * (3 * D + D + 2)).bfloat16()).requires_grad_()
        w, head = torch.randn(2 * 3 * D, 4).bfloat16(), torch.randn(2).bfloat16()
        out = gdn.gdn_inputs(proj, w, head, head, torch.zeros(T, dtype=torch.int32), 2, 1, D)
        torch.autograd.grad(out, proj, [_shifted(torch.ones_like(t)) for t in out])
    else:
        o = gdn.simple_gla(q, k, v, -torch.rand(H)) if op == 'gla' else gdn.chunk_gated_delta_rule(q, k, v, g, beta)
        torch.autograd.grad(o, (q, k, v), _shifted(torch.ones_like(o)))
    calls = {n: p for n, p in rec.pointers.items() if n.endswith(('_fwd', '_bwd'))}
    assert len(calls) == 2
    for pointers in calls.values():
        assert all(p % 16 == 0 for p in pointers)


@pytest.mark.parametrize('op', ['gla', 'rule'])
def test_kernels_that_wait_know_where_to_report(monkeypatch, op):
    """A wait that gives up is reported through the device's status word, in both directions."""
    rec, status = _Recorder(), torch.zeros(16, dtype=torch.int32)
    monkeypatch.setattr(gdn, '_cuda_ok', lambda *ts: True)
    monkeypatch.setattr(_lib, 'lib', lambda: rec)
    monkeypatch.setattr(_lib, 'stream_ptr', lambda: ctypes.c_void_p(0))
    monkeypatch.setattr(_lib, 'status_word', lambda device=None: status)
    q, k, v, g, beta = (t.requires_grad_() for t in _tensors())
    o = gdn.simple_gla(q, k, v, -torch.rand(H)) if op == 'gla' else gdn.chunk_gated_delta_rule(q, k, v, g, beta)
    torch.autograd.grad(o, (q, k, v), torch.ones_like(o))
    calls = {n: p for n, p in rec.pointers.items() if n.endswith(('_fwd', '_bwd'))}
    assert len(calls) == 2 and all(status.data_ptr() in p for p in calls.values())


def test_what_the_delta_rule_keeps(monkeypatch):
    """Of a chunk's two triangular 64 x 64 matrices, in three terms, the ten 16 x 16 blocks on and below the diagonal."""
    monkeypatch.setattr(gdn, '_cuda_ok', lambda *ts: True)
    monkeypatch.setattr(_lib, 'lib', lambda: _Recorder())
    monkeypatch.setattr(_lib, 'stream_ptr', lambda: ctypes.c_void_p(0))
    monkeypatch.setattr(_lib, 'status_word', lambda device=None: torch.zeros(16, dtype=torch.int32))
    inputs = [t.requires_grad_() for t in _tensors()]
    kept = {}
    with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.setdefault(t.data_ptr(), t), lambda t: t):
        gdn.chunk_gated_delta_rule(*inputs)
    own = sum(t.numel() * t.element_size() for p, t in kept.items() if p not in {x.data_ptr() for x in inputs})
    chunks = 4 * H                               # _Recorder's, of every head
    assert own <= chunks * (6 * 10 * 256 * 2 + 6 * 64 * 4) + 64
