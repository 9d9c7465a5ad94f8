"""The first token of every token's sequence, as a caller passes it: forms that are read as they are meant, and refusals
before anything is launched."""
import pytest
import torch

from mcore_bridge_b200.ops import _lib, attention_cuda

T, META = 5, torch.device('meta')
REFUSED = [torch.zeros(T - 1, dtype=torch.int32), torch.zeros(0, dtype=torch.int32), torch.zeros(T),
           torch.zeros(T, dtype=torch.int32, device=META)]


@pytest.mark.parametrize('one_each', [False, True])
@pytest.mark.parametrize('start', [
    torch.arange(T, dtype=torch.int32), torch.arange(T), torch.arange(T, dtype=torch.int16),
    torch.arange(T, dtype=torch.int32)[None], torch.arange(2 * T, dtype=torch.int32).view(T, 2)[:, 0] // 2])
def test_forms_of_the_same_starts(start, one_each):
    got = attention_cuda._row_starts(start, T, torch.device('cpu'), one_each)
    assert got.dtype == torch.int32 and got.is_contiguous() and got.tolist() == list(range(T))


def test_one_start_for_every_token():
    for start in (torch.tensor(3), torch.tensor([3], dtype=torch.int32)):
        got = attention_cuda._row_starts(start, T, torch.device('cpu'), True)
        assert got.dtype == torch.int32 and got.is_contiguous() and got.tolist() == [3] * T


def test_more_starts_than_tokens():
    start = torch.arange(T + 2, dtype=torch.int32)
    assert attention_cuda._row_starts(start, T, torch.device('cpu'), False).tolist() == list(range(T))
    with pytest.raises(RuntimeError):
        attention_cuda._row_starts(start, T, torch.device('cpu'), True)


@pytest.mark.parametrize('window', [None, (2, 0)])
@pytest.mark.parametrize('start', REFUSED)
def test_attention_refuses_other_starts(start, window):
    q = torch.zeros(T, 2, 64, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match='seq_start'):
        attention_cuda.attention(q, q, q, None, None, 1.0, seq_start=start, window=window)


@pytest.mark.skipif(not (_lib._LIB_PATH.exists() and _lib._HOST_PATH.exists()),
                    reason='the CUDA library and its host module are not built')
@pytest.mark.parametrize('bad', REFUSED)
def test_ranges_are_checked_before_the_launch(bad):
    nat, q, good = _lib.native(), torch.zeros(T, 2, 64, dtype=torch.bfloat16), torch.zeros(T, dtype=torch.int32)
    before = _lib.LAUNCHES
    for ranges in [(bad, None), (good, bad)]:
        with pytest.raises(AssertionError):
            nat.attention(q, q, q, *ranges, None, None, None, 1.0)
    with pytest.raises(AssertionError):
        nat.attention(q, q, q, good, None, None, None, torch.zeros(1), 1.0)  # two heads
    leaf = q.clone().requires_grad_()
    for ranges in [(bad, None, None, None), (good, bad, good, good), (good, good, bad, good), (good, good, good, bad)]:
        with pytest.raises(AssertionError):
            nat.attention(leaf, q, q, *ranges, None, 1.0)
    assert _lib.LAUNCHES == before


@pytest.mark.gpu
@pytest.mark.parametrize('window', [None, (40, 0)])
def test_forms_of_starts_on_the_device(window):
    from mcore_bridge_b200.ops.attention import attention
    n = 300
    q, k, v = (torch.randn(n, 2, 64, device='cuda').bfloat16() for _ in range(3))
    start = torch.tensor([0] * 100 + [100] * 200, dtype=torch.int32, device='cuda')
    want = attention(q, k, v, torch.tensor([0, 100, n], dtype=torch.int32, device='cuda'), window=window)
    for form in (start, start.long(), torch.stack([start, start], dim=1)[:, 0]):
        assert torch.equal(attention(q, k, v, seq_start=form, window=window), want)
    want = attention(q, k, v, window=window)
    assert torch.equal(attention(q, k, v, seq_start=start[:1], window=window), want)
