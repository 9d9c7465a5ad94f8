"""Tables and statistics that were tensor operations: the same bits as these where nothing is summed."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = 'cuda'


@pytest.mark.parametrize('dtype', [torch.int32, torch.int64])
@pytest.mark.parametrize('cu,T', [([0, 1], 1), ([0, 5, 5, 9], 9), ([0, 300], 300), ([0, 100, 257], 300), ([3, 10], 12),
                                  (list(range(0, 2001, 2)), 2000), ([0, 0, 0, 7], 7)])
def test_sequence_starts(cu, T, dtype):
    from mcore_bridge_b200.ops import _lib
    from mcore_bridge_b200.ops.attention_cuda import seq_start_from_cu
    host = torch.tensor(cu)
    seg = torch.searchsorted(host[1:].contiguous(), torch.arange(T), right=True)
    want = host[:-1][seg.clamp(max=len(cu) - 2)].int()
    before = _lib.LAUNCHES
    got = seq_start_from_cu(host.to(DEV, dtype), T, DEV)
    assert _lib.LAUNCHES == before + 1
    assert got.dtype == torch.int32 and torch.equal(got.cpu(), want)
    wide = torch.stack([host, host], 1).to(DEV, dtype)[:, 0]             # strided
    assert torch.equal(seq_start_from_cu(wide, T, DEV).cpu(), want)


@pytest.mark.parametrize('dtype', [torch.int32, torch.int64])
@pytest.mark.parametrize('T,R,scale', [(1, 1, 1.0), (7, 32, 1.0), (1000, 64, 1.2079441541679836), (4097, 3, 1.0)])
def test_rope_tables(T, R, scale, dtype):
    from mcore_bridge_b200.ops import _lib
    gen = torch.Generator(device=DEV).manual_seed(1)
    pos = torch.randint(0, 131072, (T,), generator=gen, device=DEV).to(dtype)
    inv = 1.0 / 1e6 ** (torch.arange(R, device=DEV) / R)
    freqs = pos.float()[:, None] * inv[None]
    cos, sin = _lib.native().rope_tables(pos, inv, scale)
    assert torch.equal(cos, freqs.cos() * scale) and torch.equal(sin, freqs.sin() * scale)


@pytest.mark.parametrize('rows,tiles', [(1, 1), (9, 31), (300, 33), (64, 594)])
def test_head_statistics(rows, tiles):
    from mcore_bridge_b200.ops import _lib
    gen = torch.Generator(device=DEV).manual_seed(2)
    part = torch.rand(rows, tiles, 2, generator=gen, device=DEV) * 10
    part[0, 0, 0] = -float('inf')                                       # a tile whose logits are all -inf
    part[0, 0, 1] = float(tiles == 1)
    tgt = torch.randn(rows, generator=gen, device=DEV)
    m, s = _lib.native().ce_combine(part)
    lse, loss = _lib.native().ce_loss(m, s, tgt)
    wide = part.double()
    want = torch.logsumexp(wide[..., 0] + wide[..., 1].log(), 1)
    assert torch.equal(m, part[..., 0].amax(1))
    ok = torch.isfinite(want)
    assert ok.sum() >= rows - 1
    # fp32 sums of up to 594 positive terms in 32 chains: a few units in the last place
    assert ((lse.double() - want).abs()[ok] <= 2 ** -21 * want.abs().clamp(min=1)[ok]).all()
    assert torch.equal(loss[ok], (lse - tgt)[ok])


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason='needs 2 GPUs')
def test_tables_of_another_device_than_the_current():
    from mcore_bridge_b200.ops import _lib
    from mcore_bridge_b200.ops.attention_cuda import seq_start_from_cu
    cu = torch.tensor([0, 100, 257], dtype=torch.int32, device='cuda:1')
    got = seq_start_from_cu(cu, 300, 'cuda:1')
    assert got.device == cu.device and got.tolist() == [0] * 100 + [100] * 200
    assert seq_start_from_cu(cu, 300, 'cuda').device == torch.device('cuda', torch.cuda.current_device())
    pos, inv = torch.arange(50, device='cuda:1'), torch.rand(8, device='cuda:1')
    cos, sin = _lib.native().rope_tables(pos, inv, 1.0)
    freqs = pos.float()[:, None] * inv[None]
    assert torch.equal(cos, freqs.cos()) and torch.equal(sin, freqs.sin())
