"""The router's load-balancing loss and two-term gradients: the tensor operations' bits where nothing is summed."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = 'cuda'


@pytest.mark.parametrize('T,E', [(1, 8), (3, 128), (1000, 64), (4097, 512)])
def test_split_terms_and_halves(T, E):
    from mcore_bridge_b200.ops.moe import add_halves, split_terms
    gen = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(T, E, generator=gen, device=DEV) * 10 ** torch.randint(-20, 20, (T, 1), generator=gen, device=DEV).float()
    hi = x.bfloat16()
    assert torch.equal(split_terms(x), torch.cat([hi, (x - hi.float()).bfloat16()], 1))
    odd = torch.cat([x.new_zeros(1), x.reshape(-1)])[1:].view(T, E)                      # four bytes from a wider boundary
    assert torch.equal(split_terms(odd), split_terms(x)) and torch.equal(split_terms(x.t().contiguous().t()), split_terms(x))
    y = torch.randn(2 * E, 8 * T, generator=gen, device=DEV)
    assert torch.equal(add_halves(y), (y[:E] + y[E:]).bfloat16())


@pytest.mark.parametrize('T,E,k', [(1, 32, 1), (777, 128, 8), (16384, 512, 4)])
def test_load_balancing_loss(T, E, k):
    from mcore_bridge_b200.ops.moe import RouterAuxLoss
    gen = torch.Generator(device=DEV).manual_seed(2)
    counts = torch.randint(0, T * k + 1, (E,), generator=gen, device=DEV, dtype=torch.int32)
    sums = (torch.rand(E, generator=gen, device=DEV) * T).requires_grad_()
    ref_sums, coeff = sums.detach().clone().requires_grad_(), 1.7e-3
    tokens = torch.full((), float(T), device=DEV)
    ref = coeff * E * ((counts.float() / (tokens * k)) * (ref_sums / tokens)).sum()
    aux, value = RouterAuxLoss.apply(sums, counts, T, k, coeff)
    for a, b in ((aux, ref), (value, ref / coeff)):                                      # sums of E positive terms
        assert (a - b).abs() <= b.abs() * E * 2 ** -24
    scale = torch.tensor(3.7, device=DEV)
    assert torch.equal(torch.autograd.grad(aux, sums, scale)[0], torch.autograd.grad(ref, ref_sums, scale)[0])
