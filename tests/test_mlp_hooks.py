"""Hooks on the second projection of a gated feed-forward block see its input and output."""
import pytest
import torch

from mcore_bridge_b200.layers.mlp import MLP
from mcore_bridge_b200.ops import fused_mlp
from mcore_bridge_b200.train.presets import model_config


@pytest.mark.parametrize('grad', [False, True])
def test_forward_hooks_are_called(monkeypatch, grad):
    torch.manual_seed(0)
    mlp = MLP(model_config('qwen3_tiny')).eval()
    x = torch.randn(3, mlp.config.hidden_size).to(next(mlp.parameters()).dtype)
    for p in mlp.parameters():
        torch.nn.init.normal_(p, std=0.02)
    with torch.no_grad():
        want = mlp(x)
    fused = []
    # where the fused block covers the operands (as on a GPU)
    monkeypatch.setattr(fused_mlp, 'usable', lambda x, w: w is mlp.linear_fc2.weight)
    monkeypatch.setattr(fused_mlp, 'glu_linear', lambda *a: fused.append(a) or want)
    seen = []
    with torch.set_grad_enabled(grad):
        mlp(x)
        assert len(fused) == 1
        for register in (mlp.linear_fc2.register_forward_hook, mlp.linear_fc2.register_forward_pre_hook):
            handle = register(lambda module, *a: seen.append(len(a)))
            y = mlp(x)
            handle.remove()
            assert torch.equal(y, want) and len(fused) == 1
        assert seen == [2, 1]
        mlp(x)
        assert len(fused) == 2
