"""A layer calls its projections as modules wherever somebody could be listening, or has put something else in their place."""
import pytest
import torch
from torch.nn.modules import module as torch_module

from mcore_bridge_b200.layers.attention import SelfAttention
from mcore_bridge_b200.layers.context import ForwardContext
from mcore_bridge_b200.layers.linear import LayerNormColumnParallelLinear, RowParallelLinear, is_plain
from mcore_bridge_b200.layers.mlp import MLP
from mcore_bridge_b200.models.transformer_layer import TransformerLayer
from mcore_bridge_b200.train.presets import model_config

SEEN_BY = ['linear_qkv', 'linear_proj', 'linear_fc1', 'linear_fc2']


def _layer():
    torch.manual_seed(0)
    layer = TransformerLayer(model_config('qwen3_tiny'), 1)
    for p in layer.parameters():
        torch.nn.init.normal_(p, std=0.02)
    d = layer.self_attention.head_dim if hasattr(layer.self_attention, 'head_dim') else layer.config.kv_channels
    x = torch.randn(6, layer.config.hidden_size, dtype=layer.config.params_dtype)
    ang = torch.rand(6, d // 2)
    ctx = ForwardContext(cu_seqlens=torch.tensor([0, 6], dtype=torch.int32), max_seqlen=6,
                         seq_start=torch.zeros(6, dtype=torch.int32))
    ctx.cos, ctx.sin = ang.cos(), ang.sin()
    return layer, x, ctx


def _names(layer):
    return {m: n.rsplit('.', 1)[-1] for n, m in layer.named_modules()}


@pytest.mark.parametrize('register', [torch_module.register_module_forward_hook, torch_module.register_module_forward_pre_hook])
def test_global_hooks_see_every_module(register):
    layer, x, ctx = _layer()
    want, names, seen, outputs = layer(x, ctx), _names(layer), [], {}

    def hook(module, args, *out):
        seen.append(names.get(module))
        if out:
            outputs[names.get(module)] = out[0]

    handle = register(hook)
    try:
        got = layer(x, ctx)
    finally:
        handle.remove()
    assert torch.equal(got, want)
    assert [n for n in seen if n in SEEN_BY] == SEEN_BY
    if outputs:                                  # a block's result is its own, without the residual
        assert torch.equal(x + outputs['self_attention'] + outputs['mlp'], got)
    assert is_plain(layer.mlp, MLP)


def test_global_backward_hooks_see_every_module():
    layer, x, ctx = _layer()
    names, seen = _names(layer), []
    handle = torch_module.register_module_full_backward_hook(lambda module, *grads: seen.append(names.get(module)))
    try:
        layer(x.requires_grad_(), ctx).float().sum().backward()
    finally:
        handle.remove()
    assert sorted(n for n in seen if n in SEEN_BY) == sorted(SEEN_BY)


@pytest.mark.parametrize('cls,name', [(SelfAttention, 'self_attention'), (MLP, 'mlp'), (RowParallelLinear, 'linear_proj'),
                                      (LayerNormColumnParallelLinear, 'linear_qkv')])
def test_a_forward_put_in_the_class_is_called(monkeypatch, cls, name):
    layer, x, ctx = _layer()
    want, names, seen, own = layer(x, ctx), _names(layer), [], cls.forward

    def forward(self, x, *ctx):                  # as the class's own before it took a residual
        assert len(ctx) <= (cls is SelfAttention)
        seen.append(names[self])
        return own(self, x, *ctx)

    monkeypatch.setattr(cls, 'forward', forward)
    assert torch.equal(layer(x, ctx), want)
    assert name in seen
