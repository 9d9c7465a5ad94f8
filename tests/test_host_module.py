"""The module behind the most frequent calls: what it refuses, and the switch it reads."""
import pytest
import torch

from mcore_bridge_b200.ops import _lib

pytestmark = pytest.mark.skipif(not (_lib._LIB_PATH.exists() and _lib._HOST_PATH.exists()),
                                reason='the CUDA library and its host module are not built')


def test_arguments_are_checked_before_anything_runs():
    nat = _lib.native()
    x = torch.zeros(8, 8)
    before = _lib.LAUNCHES
    with pytest.raises(TypeError):
        nat.mm(0, x, x)
    with pytest.raises(TypeError):
        nat.mm(0, None, x, None, None, False, False, 1.0, 0, 0)
    with pytest.raises(AssertionError):
        nat.mm(0, x, torch.zeros(8, 7), None, None, False, False, 1.0, 0, 0)     # contraction sizes differ
    with pytest.raises(AssertionError):
        nat.mm(0, x, x, None, torch.zeros(8, 7), False, False, 1.0, 0, 0)        # output of another shape
    assert _lib.LAUNCHES == before


BF16, META = torch.bfloat16, torch.device('meta')


def _bf(*shape):
    return torch.zeros(shape, dtype=BF16)


@pytest.mark.parametrize('call', [
    lambda n: n.mm(0, _bf(8, 8), torch.zeros(8, 8), None, None, False, False, 1.0, 0, 0),                 # an fp32 weight
    lambda n: n.mm(0, _bf(8, 8).half(), _bf(8, 8), None, None, False, False, 1.0, 0, 0),
    lambda n: n.mm(1, _bf(8, 8), _bf(8, 8), None, torch.zeros(8, 8, dtype=torch.float16), False, False, 1.0, 0, 0),
    lambda n: n.mm(0, _bf(8, 8), _bf(8, 8), None, torch.zeros(8, 8, device=META), False, False, 1.0, 0, 0),
    lambda n: n.mm(0, _bf(8, 8), _bf(8, 8), torch.zeros(7), None, False, False, 1.0, 0, 0),               # a bias too short
    lambda n: n.mm(2, _bf(8, 8), _bf(8, 8), None, _bf(2, 4, 8), False, False, 1.0, 0, 0),                  # a gradient of 3 axes
    lambda n: n.rmsnorm(_bf(4, 16), torch.zeros(16), 1e-6, False),
    lambda n: n.rmsnorm(_bf(4, 16), _bf(8), 1e-6, False),
    lambda n: n.rmsnorm(torch.zeros(4, 16), _bf(16), 1e-6, False),
    lambda n: n.linear(_bf(4, 16), torch.zeros(8, 16), None, False, None),
    lambda n: n.linear(_bf(4, 16), _bf(8, 8), None, False, None),
    lambda n: n.linear(_bf(4, 16), _bf(8, 16), torch.zeros(7), False, None),
    lambda n: n.linear(_bf(4, 16), _bf(8, 16), None, False, _bf(4, 16)),                                   # a residual of another shape
    lambda n: n.linear(_bf(4, 16), _bf(8, 16), None, False, _bf(4, 8).to(META)),
    lambda n: n.norm_linear(_bf(4, 16), _bf(16).to(META), _bf(8, 16), 1e-6, False, False),
    lambda n: n.glu_fwd(torch.zeros(4, 16), None, 0, 0.0, 0.0),
    lambda n: n.glu_fwd(_bf(4, 16), torch.zeros(3), 0, 0.0, 0.0),
    lambda n: n.glu_bwd(_bf(4, 8), _bf(4, 16), torch.zeros(3), 0, 0.0, 0.0),
    lambda n: n.glu_linear(torch.zeros(4, 16), _bf(8, 8), 0, 0.0, 0.0, None),
    lambda n: n.qkv(_bf(4, 31), None, None, None, None, 1, 2, 8, False, False, 1e-6, False),               # 4 heads of 8
    lambda n: n.qkv(_bf(4, 32), _bf(8), _bf(4), None, None, 1, 2, 8, False, False, 1e-6, False),
    lambda n: n.qkv(_bf(4, 32), None, None, torch.zeros(4, 4), torch.zeros(3, 4), 1, 2, 8, False, False, 1e-6, False),
    lambda n: n.attention(_bf(4, 2, 64), _bf(4, 2, 64), torch.zeros(4, 2, 64), torch.zeros(4, dtype=torch.int32), None, None, None,
                          None, 1.0),
])
def test_operands_the_kernels_would_misread_are_refused(call):
    before = _lib.LAUNCHES
    with pytest.raises(AssertionError):
        call(_lib.native())
    assert _lib.LAUNCHES == before


def test_kernels_are_switched_off_by_the_environment(monkeypatch):
    nat = _lib.native()
    monkeypatch.delenv('MCB200_DISABLE_CUDA_KERNELS', raising=False)
    assert nat.enabled()
    monkeypatch.setenv('MCB200_DISABLE_CUDA_KERNELS', '1')
    assert not nat.enabled()
    monkeypatch.setenv('MCB200_DISABLE_CUDA_KERNELS', '0')
    assert nat.enabled()


def test_a_module_for_another_torch_is_not_loaded(monkeypatch, tmp_path):
    from mcore_bridge_b200 import build_ext
    mine = build_ext.host_name()
    assert _lib._HOST_PATH.name == mine
    monkeypatch.setattr(torch, '__version__', '99.0+other')
    assert build_ext.host_name() != mine
    monkeypatch.setattr(_lib, '_native', None)
    monkeypatch.setattr(_lib, '_HOST_PATH', tmp_path / build_ext.host_name())
    monkeypatch.setattr(torch.cuda, 'is_available', lambda: False)
    with pytest.raises(_lib.KernelError, match='build_ext'):
        _lib.native()


def test_kernels_of_the_library_alone_do_without_the_module(monkeypatch):
    def missing():
        raise _lib.KernelError('no module')

    monkeypatch.setattr(_lib, 'cuda_enabled', lambda: True)
    monkeypatch.setattr(_lib, 'native', missing)
    assert _lib.available()


def test_split_of_the_key_gradient_kernel(monkeypatch):
    nat = _lib.native()
    for text, splits in [('1', 1), ('2', 2), ('4', 4), ('3', 1), ('0', 1), ('-2', 1)]:     # 4 query heads share a kv head
        monkeypatch.setenv('MCB200_ATTN_DKV_SPLITS', text)
        assert nat.attn_dkv_splits(1000, 8, 2) == splits
    monkeypatch.setenv('MCB200_ATTN_DKV_SPLITS', 'many')
    with pytest.raises(ValueError):
        nat.attn_dkv_splits(1000, 8, 2)
    monkeypatch.delenv('MCB200_ATTN_DKV_SPLITS')
    with pytest.raises(AssertionError):
        nat.attn_dkv_splits(1000, 8, 0)
    for tokens, heads, kv_heads, want in [(3000, 9, 3, 3), (777, 5, 1, 5), (2048, 32, 8, 4), (8192, 32, 8, 1), (100, 12, 2, 6),
                                          (100, 7, 7, 1), (12800, 12, 2, 3), (4096, 24, 8, 1)]:
        assert nat.attn_dkv_splits(tokens, heads, kv_heads) == want
