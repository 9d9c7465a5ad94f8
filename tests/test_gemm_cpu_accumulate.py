"""Products without the kernels that are added to a given tensor."""
import pytest
import torch

from mcore_bridge_b200.ops import gemm


@pytest.mark.parametrize('op', ['nt', 'nn'])
def test_a_sum_is_rounded_once(op):
    """An fp32 product added to a bf16 tensor: the sum is formed in fp32 and rounded, the product by itself is not."""
    x, w = torch.tensor([[1 + 2.0 ** -8 - 2.0 ** -12]]), torch.ones(1, 1)          # by itself it rounds to 1
    out = torch.full((1, 1), 2.0 ** -9, dtype=torch.bfloat16)
    (gemm.mm_nt if op == 'nt' else gemm.mm_nn)(x, w, out=out, accumulate=True)
    assert out.item() == 1 + 2.0 ** -7                      # 1 + 2^-8 + 2^-9 - 2^-12 lies above the middle of 1 and 1 + 2^-7


def test_a_weight_gradient_keeps_its_shape():
    dy, x = torch.ones(3, 2), torch.ones(3, 4)
    out = torch.zeros(2, 2, 4)
    assert gemm.mm_tn(dy, x, out=out, accumulate=True) is out and torch.equal(out, torch.full((2, 2, 4), 3.0))
    with pytest.raises(RuntimeError):
        gemm.mm_tn(dy, x, out=torch.zeros(8))
