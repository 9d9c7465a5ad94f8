"""The work this framework spends a training run's time on, as measurable cases.

Every case is one forward + backward pass (or a forward pass alone) through a public entry point: the attention and
linear-attention operators, the dense and mixture-of-experts blocks, a whole decoder layer, the language-model head
with its loss, and a small model end to end.  Sizes are those of the presets (``train/presets.py``), of the benchmark
and of the tests, with ragged token counts among them.  ``exact`` restates each case in plain torch in 64 bits.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from mcore_bridge_b200 import ModelConfig, get_mcore_model, hf_to_mcore_config
from mcore_bridge_b200.layers.context import ForwardContext, PackedSeqParams
from mcore_bridge_b200.layers.gated_delta_net import GatedDeltaNet
from mcore_bridge_b200.layers.mlp import MLP
from mcore_bridge_b200.layers.moe import MoELayer
from mcore_bridge_b200.models.transformer_layer import TransformerLayer
from mcore_bridge_b200.ops.attention import attention
from mcore_bridge_b200.ops.attention_cuda import seq_start_from_cu
from mcore_bridge_b200.ops.cross_entropy import fused_linear_cross_entropy
from mcore_bridge_b200.ops.gdn import simple_gla
from mcore_bridge_b200.train.presets import model_config
from mcore_bridge_b200.utils.torch_utils import attach_host_list

DEV, BF16, F64 = 'cuda', torch.bfloat16, torch.float64


# ---------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one short packed row of a small model: latency and launch count decide
        dict(name='attn_short', kind='attention', tokens=333, heads=4, kv_heads=2, dim=64, segments=3, window=0),
        # the training benchmark's micro-batch: 8192 packed tokens, 32 query / 8 kv heads
        dict(name='attn_packed', kind='attention', tokens=8192, heads=32, kv_heads=8, dim=128, segments=5, window=0),
        # long-context training: a single long sequence
        dict(name='attn_long', kind='attention', tokens=16384, heads=32, kv_heads=8, dim=128, segments=1, window=0),
        # sliding-window layer with learnable softmax sinks (the GPT-OSS family)
        dict(name='attn_window', kind='attention', tokens=4095, heads=64, kv_heads=8, dim=64, segments=2, window=128),
        # feed-forward block of a small model on a ragged micro-batch
        dict(name='mlp_ragged', kind='mlp', tokens=773, hidden=2048, ffn=6144),
        # one decoder layer of the training benchmark (8B shape, 8192 packed tokens)
        dict(name='layer_dense', kind='layer', tokens=8192, hidden=4096, ffn=12288, heads=32, kv_heads=8, dim=128,
             segments=5),
        # language-model head + loss over the full vocabulary
        dict(name='head_loss', kind='head', tokens=4096, hidden=4096, vocab=151936),
        # mixture-of-experts layer of the 30B-A3B shape, all 128 experts on one GPU
        dict(name='moe_layer', kind='moe', tokens=4096, hidden=2048, ffn=768, experts=128, topk=8),
        # linear-attention block of the Qwen3-Next family
        dict(name='gdn_layer', kind='gdn', tokens=4096, hidden=2048, k_heads=16, v_heads=32, dim=128, segments=3),
        # lightning attention (Ling / Ring hybrid family): linear attention with a constant decay per head
        dict(name='lightning', kind='gla', tokens=4096, heads=16, dim=128, segments=2),
        # evaluation of a small model on a short ragged prompt: logits
        dict(name='model_eval', kind='model', tokens=201, layers=4, hidden=256, ffn=768, heads=4, kv_heads=2, dim=64,
             vocab=1024, train=False),
        # training pass of a small model: per-token losses and every gradient
        dict(name='model_train', kind='model', tokens=1024, layers=4, hidden=256, ffn=768, heads=4, kv_heads=2, dim=64,
             vocab=1024, train=True),
    ]


def _log(rng, lo, hi, multiple=1):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(multiple, min(hi, n // multiple * multiple))


def draw(rng):
    kind = rng.choice(['attention', 'attention', 'attention', 'mlp', 'mlp', 'layer', 'head', 'moe', 'gdn', 'gla',
                       'model'])
    if kind == 'attention':
        dim = rng.choice([64, 128])
        kv = rng.choice([1, 2, 4, 8])
        heads = kv * rng.choice([1, 2, 3, 4, 8])
        tokens = _log(rng, 64, 16384 if heads <= 32 else 8192)
        return dict(kind=kind, tokens=tokens, heads=heads, kv_heads=kv, dim=dim, segments=rng.choice([1, 1, 2, 3, 7]),
                    window=rng.choice([0, 0, 0, 128, 1000]))
    if kind == 'mlp':
        return dict(kind=kind, tokens=_log(rng, 32, 8192), hidden=_log(rng, 256, 4096, 64),
                    ffn=_log(rng, 512, 12288, 64))
    if kind == 'layer':
        kv = rng.choice([2, 4, 8])
        return dict(kind=kind, tokens=_log(rng, 128, 8192), hidden=_log(rng, 256, 4096, 128),
                    ffn=_log(rng, 512, 12288, 128), heads=kv * rng.choice([2, 4]), kv_heads=kv,
                    dim=rng.choice([64, 128]), segments=rng.choice([1, 2, 5]))
    if kind == 'head':
        return dict(kind=kind, tokens=_log(rng, 64, 4096), hidden=_log(rng, 256, 4096, 64),
                    vocab=_log(rng, 1024, 151936, 8))
    if kind == 'moe':
        experts = rng.choice([8, 32, 64, 128])
        return dict(kind=kind, tokens=_log(rng, 64, 8192), hidden=_log(rng, 256, 2048, 128),
                    ffn=_log(rng, 128, 1024, 64), experts=experts, topk=rng.choice([2, 4, 8]))
    if kind == 'gdn':
        kh = rng.choice([2, 4, 8, 16])
        return dict(kind=kind, tokens=_log(rng, 64, 8192), hidden=_log(rng, 256, 2048, 128), k_heads=kh,
                    v_heads=kh * rng.choice([1, 2]), dim=rng.choice([64, 128]), segments=rng.choice([1, 3, 6]))
    if kind == 'gla':
        return dict(kind=kind, tokens=_log(rng, 64, 8192), heads=rng.choice([4, 8, 16, 32]), dim=rng.choice([64, 128]),
                    segments=rng.choice([1, 2, 5]))
    return dict(kind=kind, tokens=_log(rng, 32, 4096), layers=rng.choice([2, 4]), hidden=256, ffn=768, heads=4,
                kv_heads=2, dim=64, vocab=1024, train=rng.random() < 0.5)


# ---------------------------------------------------------------------------------------------------- inputs
def _bounds(case):
    """Packed segment boundaries: ragged lengths in a fixed pattern, the same for every seed."""
    n, total = case.get('segments', 1), case['tokens']
    weights = [(5, 2, 7, 3, 1, 6, 4)[i % 7] for i in range(n)]
    cu, acc = [0], 0
    for w in weights[:-1]:
        acc += w
        cu.append(max(cu[-1] + 1, total * acc // sum(weights)))
    return cu + [total]


def _packing(case):
    host = torch.tensor(_bounds(case), dtype=torch.int32)
    cu = host.to(DEV)
    attach_host_list(cu, host)
    return cu, int((host[1:] - host[:-1]).max())


class _Gen:

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(1000 + seed)

    def normal(self, *shape, std=1.0, dtype=BF16, grad=False):
        return (torch.randn(*shape, generator=self.g, device=DEV) * std).to(dtype).requires_grad_(grad)

    def ints(self, high, *shape):
        return torch.randint(0, high, shape, generator=self.g, device=DEV)


def _fill(module, gen, zero_centered=False):
    """Random weights of a module: N(0, 0.02) matrices, norm weights around their identity, decays of trained size."""
    with torch.no_grad():
        for name, p in sorted(module.named_parameters()):
            if name.endswith('A_log'):
                p.copy_(torch.log(1 + 15 * torch.rand(p.shape, generator=gen.g, device=DEV)))
            elif name.endswith('dt_bias'):
                p.copy_(1 + gen.normal(*p.shape, std=0.1))
            elif 'conv1d' in name:
                p.copy_(gen.normal(*p.shape, std=0.3))
            elif p.dim() == 1:
                identity = 0.0 if zero_centered and 'out_norm' not in name else 1.0
                p.copy_(identity + gen.normal(*p.shape, std=0.1))
            else:
                p.copy_(gen.normal(*p.shape, std=0.02))


def _dense_config(case):
    return model_config('qwen3_tiny', dict(
        num_hidden_layers=case.get('layers', 1), hidden_size=case['hidden'], intermediate_size=case['ffn'],
        num_attention_heads=case.get('heads', 4), num_key_value_heads=case.get('kv_heads', 2),
        head_dim=case.get('dim', 64), vocab_size=case.get('vocab', 1024)), bf16=True)


def _moe_config(case):
    return model_config('qwen3_moe_tiny', dict(
        hidden_size=case['hidden'], moe_intermediate_size=case['ffn'], num_experts=case['experts'],
        num_experts_per_tok=case['topk']), bf16=True, moe_aux_loss_coeff=1e-3,
        moe_router_load_balancing_type='aux_loss')


def _gdn_config(case):
    from transformers import Qwen3NextConfig
    hf = Qwen3NextConfig(
        num_hidden_layers=4, hidden_size=case['hidden'], num_attention_heads=4, num_key_value_heads=2, head_dim=64,
        intermediate_size=256, moe_intermediate_size=64, shared_expert_intermediate_size=64, num_experts=8,
        num_experts_per_tok=2, linear_num_key_heads=case['k_heads'], linear_num_value_heads=case['v_heads'],
        linear_key_head_dim=case['dim'], linear_value_head_dim=case['dim'], linear_conv_kernel_dim=4, vocab_size=256,
        max_position_embeddings=512, full_attention_interval=4, partial_rotary_factor=0.25, tie_word_embeddings=False,
        decoder_sparse_step=1, mlp_only_layers=[], norm_topk_prob=True)
    return ModelConfig(**hf_to_mcore_config(hf), params_dtype=BF16)


def _positions(bounds):
    return torch.cat([torch.arange(e - s) for s, e in zip(bounds[:-1], bounds[1:])]).to(DEV)


def _rope_tables(bounds, dim, base=1e6):
    inv = 1.0 / base ** (torch.arange(0, dim, 2, dtype=F64, device=DEV) / dim)
    ang = _positions(bounds).to(F64)[:, None] * inv
    return ang.cos().float(), ang.sin().float()


def prepare(case, seed):
    gen, kind, T = _Gen(seed), case['kind'], case['tokens']
    s = dict(case=case)
    if kind == 'attention':
        nq, nkv, d = case['heads'], case['kv_heads'], case['dim']
        cu, longest = _packing(case)
        s.update(q=gen.normal(T, nq, d, grad=True), k=gen.normal(T, nkv, d, grad=True),
                 v=gen.normal(T, nkv, d, grad=True), dy=gen.normal(T, nq, d), cu=cu, longest=longest,
                 start=seq_start_from_cu(cu, T, DEV), sinks=None)
        if case['window']:
            s['sinks'] = gen.normal(nq, grad=True)
    elif kind in ('mlp', 'layer', 'moe', 'gdn'):
        with torch.device(DEV):
            if kind == 'mlp':
                module = MLP(_dense_config(case))
            elif kind == 'layer':
                module = TransformerLayer(_dense_config(case), 1)
            elif kind == 'moe':
                module = MoELayer(_moe_config(case))
            else:
                module = GatedDeltaNet(_gdn_config(case), 1)
        _fill(module, gen, zero_centered=kind == 'gdn')
        module.train()
        s.update(module=module, x=gen.normal(T, case['hidden'], grad=True), dy=gen.normal(T, case['hidden']),
                 params=[p for _, p in sorted(module.named_parameters())])
        if kind in ('layer', 'gdn'):
            cu, longest = _packing(case)
            s['ctx'] = ForwardContext(cu_seqlens=cu, max_seqlen=longest, seq_start=seq_start_from_cu(cu, T, DEV))
            if kind == 'layer':
                s['ctx'].cos, s['ctx'].sin = _rope_tables(_bounds(case), case['dim'])
    elif kind == 'head':
        s.update(h=gen.normal(T, case['hidden'], grad=True),
                 w=gen.normal(case['vocab'], case['hidden'], std=0.02, grad=True), labels=gen.ints(case['vocab'], T),
                 dy=torch.full((T,), 1.0 / T, device=DEV))
    elif kind == 'gla':
        h, d = case['heads'], case['dim']
        cu, _ = _packing(case)
        s.update(q=gen.normal(T, h, d, grad=True), k=gen.normal(T, h, d, grad=True), v=gen.normal(T, h, d, grad=True),
                 dy=gen.normal(T, h, d), cu=cu,
                 decay=-(2.0 ** (-8.0 * torch.arange(1, h + 1, device=DEV, dtype=torch.float32) / h)))
    else:
        with torch.device(DEV):
            module = get_mcore_model(_dense_config(case))[0]
        module = module.to(DEV)
        _fill(module, gen)
        module.train(case['train'])
        cu, longest = _packing(case)
        s.update(module=module, ids=gen.ints(case['vocab'], 1, T), labels=gen.ints(case['vocab'], 1, T),
                 pos=_positions(_bounds(case))[None], dy=torch.full((1, T), 1.0 / T, device=DEV),
                 packed=PackedSeqParams(cu_seqlens_q=cu, cu_seqlens_kv=cu, max_seqlen_q=longest, max_seqlen_kv=longest),
                 params=[p for _, p in sorted(module.named_parameters())])
    return s


# ---------------------------------------------------------------------------------------------------- one pass
def run(s):
    case = s['case']
    kind = case['kind']
    if kind == 'attention':
        window = (case['window'], 0) if case['window'] else None
        o = attention(s['q'], s['k'], s['v'], s['cu'], s['longest'], window=window, sinks=s['sinks'],
                      seq_start=s['start'])
        inputs = [s['q'], s['k'], s['v']] + ([s['sinks']] if s['sinks'] is not None else [])
        return [o.detach(), *torch.autograd.grad(o, inputs, s['dy'])]
    if kind in ('mlp', 'moe'):
        y = s['module'](s['x'])
        return [y.detach(), *torch.autograd.grad(y, [s['x'], *s['params']], s['dy'])]
    if kind in ('layer', 'gdn'):
        y = s['module'](s['x'], s['ctx'])
        return [y.detach(), *torch.autograd.grad(y, [s['x'], *s['params']], s['dy'])]
    if kind == 'head':
        loss = fused_linear_cross_entropy(s['h'], s['w'], s['labels'])
        return [loss.detach(), *torch.autograd.grad(loss, [s['h'], s['w']], s['dy'])]
    if kind == 'gla':
        o = simple_gla(s['q'], s['k'], s['v'], s['decay'], s['cu'])
        return [o.detach(), *torch.autograd.grad(o, [s['q'], s['k'], s['v']], s['dy'])]
    if not case['train']:
        with torch.no_grad():
            return s['module'](s['ids'], position_ids=s['pos'], packed_seq_params=s['packed'])
    loss = s['module'](s['ids'], position_ids=s['pos'], labels=s['labels'], packed_seq_params=s['packed'])
    return [loss.detach(), *torch.autograd.grad(loss, s['params'], s['dy'])]


# ---------------------------------------------------------------------------------------------------- its work
def _pairs(case):
    """(query, key) pairs that attend to each other: causal inside each packed segment, within the window."""
    w, total = case.get('window', 0), 0
    b = _bounds(case)
    for s, e in zip(b[:-1], b[1:]):
        n = e - s
        total += n * (n + 1) // 2
        if w and n > w + 1:
            total -= (n - w - 1) * (n - w) // 2
    return total


def _dense_params(case):
    qkv = case['hidden'] * (case['heads'] + 2 * case['kv_heads']) * case['dim']
    return qkv + case['heads'] * case['dim'] * case['hidden'] + 3 * case['hidden'] * case['ffn']


def work(case):
    kind, T = case['kind'], case['tokens']
    if kind == 'attention':
        nq, nkv, d = case['heads'], case['kv_heads'], case['dim']
        # two products forward, five backward; q, o, dy, dq and k, v, dk, dv once each
        return dict(bytes=2 * T * d * (4 * nq + 4 * nkv), flops=14 * _pairs(case) * nq * d)
    if kind == 'mlp':
        p = 3 * case['hidden'] * case['ffn']
        return dict(bytes=2 * (2 * p + 4 * T * case['hidden']), flops=6 * T * p)
    if kind == 'layer':
        p = _dense_params(case)
        return dict(bytes=2 * (2 * p + 4 * T * case['hidden']),
                    flops=6 * T * p + 14 * _pairs(case) * case['heads'] * case['dim'])
    if kind == 'head':
        p = case['hidden'] * case['vocab']
        return dict(bytes=2 * (2 * p + 2 * T * case['hidden']) + 12 * T, flops=6 * T * p)
    if kind == 'moe':
        p = 3 * case['hidden'] * case['ffn']
        return dict(bytes=2 * (2 * p * case['experts'] + 4 * T * case['hidden']),
                    flops=6 * T * (p * case['topk'] + case['hidden'] * case['experts']))
    if kind == 'gdn':
        d, kh, vh = case['dim'], case['k_heads'], case['v_heads']
        p = case['hidden'] * (kh * 2 * d + vh * (3 * d + 2))
        # the recurrence per token and value head: decay-free state read, write and query, forward and twice backward
        return dict(bytes=2 * (2 * p + 4 * T * case['hidden']), flops=6 * T * p + 3 * 6 * T * vh * d * d)
    if kind == 'gla':
        h, d = case['heads'], case['dim']
        return dict(bytes=2 * 8 * T * h * d, flops=3 * 4 * T * h * d * d)
    p = case['layers'] * _dense_params(case) + case['hidden'] * case['vocab']
    att = case['layers'] * _pairs(case) * case['heads'] * case['dim']
    if case['train']:
        return dict(bytes=2 * 2 * (p + case['hidden'] * case['vocab']) + 12 * T, flops=6 * T * p + 14 * att)
    return dict(bytes=2 * (p + T * (case['hidden'] + case['vocab'])) + 8 * T, flops=2 * T * p + 4 * att)


def tolerance(case):
    """About four times the measured distance of bf16 results from the 64-bit ones (in brackets): the products of one
    operator, then the chains of a block, a layer and a model."""
    return {'rel': dict(attention=0.011,    # 0.0019 .. 0.0028
                        gla=0.007,          # 0.0017
                        head=0.007,         # 0.0017
                        mlp=0.017,          # 0.0042
                        moe=0.017,          # 0.0034 .. 0.0041
                        layer=0.03,         # 0.0049 .. 0.0079
                        gdn=0.03,           # 0.007 .. 0.014
                        model=0.03)[case['kind']]}   # 0.0055 .. 0.014


# ---------------------------------------------------------------------------------------------------- 64 bits
def _exact_norm(x, w, eps=1e-6):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _exact_rope(x, cos, sin):
    c, s = cos.to(F64)[:, None], sin.to(F64)[:, None]
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _exact_attention(q, k, v, bounds, window=0, sinks=None):
    """Head by head and, for long sequences, block of queries by block; each block is recomputed in backward."""
    from torch.utils.checkpoint import checkpoint
    nq, nkv, d = q.shape[1], k.shape[1], q.shape[2]

    def block(qb, kb, vb, first, key0, sink):
        sc = qb @ kb.t() / math.sqrt(d)
        i = torch.arange(qb.shape[0], device=DEV)[:, None] + first
        j = torch.arange(kb.shape[0], device=DEV)[None] + key0
        hide = j > i
        if window:
            hide = hide | (j < i - window)
        sc = sc.masked_fill(hide, float('-inf'))
        if sink is not None:
            p = torch.softmax(torch.cat([sc, sink.expand(sc.shape[0], 1)], dim=1), dim=1)[:, :-1]
        else:
            p = torch.softmax(sc, dim=1)
        return p @ vb

    heads = []
    for h in range(nq):
        g, rows = h // (nq // nkv), []
        for s, e in zip(bounds[:-1], bounds[1:]):
            for b in range(s, e, 4096):
                t = min(e, b + 4096)
                key0 = max(s, b - window) if window else s
                rows.append(checkpoint(block, q[b:t, h], k[key0:t, g], v[key0:t, g], b, key0,
                                       None if sinks is None else sinks[h:h + 1], use_reentrant=False))
        heads.append(torch.cat(rows))
    return torch.stack(heads, dim=1)


def _exact_swiglu(h):
    g, u = h.chunk(2, dim=-1)
    return F.silu(g) * u


def _exact_mlp(x, p):
    h = _exact_norm(x, p['linear_fc1.layer_norm_weight']) @ p['linear_fc1.weight'].t()
    return _exact_swiglu(h) @ p['linear_fc2.weight'].t()


def _exact_dense_layer(x, p, case, cos, sin):
    nkv, d = case['kv_heads'], case['dim']
    a = {n[len('self_attention.'):]: v for n, v in p.items() if n.startswith('self_attention.')}
    qkv = _exact_norm(x, a['linear_qkv.layer_norm_weight']) @ a['linear_qkv.weight'].t()
    qkv = qkv.view(x.shape[0], nkv, -1, d)
    q, k, v = qkv[:, :, :-2].reshape(x.shape[0], -1, d), qkv[:, :, -2], qkv[:, :, -1]
    q = _exact_rope(_exact_norm(q, a['q_layernorm.weight']), cos, sin)
    k = _exact_rope(_exact_norm(k, a['k_layernorm.weight']), cos, sin)
    o = _exact_attention(q, k, v, _bounds(case))
    x = x + o.reshape(x.shape[0], -1) @ a['linear_proj.weight'].t()
    return x + _exact_mlp(x, {n[len('mlp.'):]: v for n, v in p.items() if n.startswith('mlp.')})


def _exact_moe(x, p, case):
    T, E, k = case['tokens'], case['experts'], case['topk']
    logits = x @ p['router.weight'].t()
    idx = logits.topk(k, dim=-1).indices
    probs = torch.softmax(logits.gather(1, idx), dim=-1)
    share = torch.bincount(idx.reshape(-1), minlength=E).to(F64) / (T * k)
    aux = 1e-3 * E * (share * torch.softmax(logits, dim=-1).mean(0)).sum()
    y = torch.zeros_like(x)
    for e in range(E):
        t, c = (idx == e).nonzero(as_tuple=True)
        if t.numel():
            h = _exact_swiglu(x[t] @ p['experts.linear_fc1.weight'][e].t()) * probs[t, c][:, None]
            y = y.index_add(0, t, h @ p['experts.linear_fc2.weight'][e].t())
    return y, aux


def _exact_delta_rule(q, k, v, g, beta, chunk=64):
    """The gated delta rule of one sequence ``[h, L, d]``: inside a chunk the writes are one triangular solve."""
    h, L, d = q.shape
    S = torch.zeros(h, d, v.shape[-1], dtype=F64, device=DEV)
    out = []
    for s in range(0, L, chunk):
        qc, kc, vc, bc = q[:, s:s + chunk], k[:, s:s + chunk], v[:, s:s + chunk], beta[:, s:s + chunk, None]
        gc = g[:, s:s + chunk].cumsum(-1)
        n = qc.shape[1]
        decay = (gc[:, :, None] - gc[:, None, :]).tril().exp().tril()
        A = torch.eye(n, dtype=F64, device=DEV) + (bc * (kc @ kc.transpose(1, 2)) * decay).tril(-1)
        rhs = bc * (vc - gc.exp()[..., None] * (kc @ S))
        u = torch.linalg.solve_triangular(A, rhs, upper=False, unitriangular=True)
        out.append((qc * gc.exp()[..., None]) @ S + ((qc @ kc.transpose(1, 2)) * decay) @ u)
        last = gc[:, -1]
        S = S * last.exp()[:, None, None] + (kc * (last[:, None] - gc).exp()[..., None]).transpose(1, 2) @ u
    return torch.cat(out, dim=1)


def _exact_gdn(x, p, case, bounds):
    T, kh, vh, d = case['tokens'], case['k_heads'], case['v_heads'], case['dim']
    r = vh // kh
    proj = (_exact_norm(x, 1 + p['in_proj.layer_norm_weight']) @ p['in_proj.weight'].t()).view(T, kh, -1)
    qkv, z, b, a = proj.split([(2 + r) * d, r * d, r, r], dim=-1)
    w = p['conv1d.weight'].squeeze(1)
    qkv, taps = qkv.reshape(T, -1), w.shape[1]
    pieces = []
    for s, e in zip(bounds[:-1], bounds[1:]):
        xs = F.pad(qkv[s:e], (0, 0, taps - 1, 0))
        pieces.append(sum(xs[j:j + e - s] * w[:, j] for j in range(taps)))
    qkv = F.silu(torch.cat(pieces)).view(T, kh, -1)
    q, k, v = qkv.split([d, d, r * d], dim=-1)
    q, k = (t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (t.repeat_interleave(r, dim=1) for t in (q * d ** -0.5, k))
    v, z, b, a = v.reshape(T, vh, d), z.reshape(T, vh, d), b.reshape(T, vh), a.reshape(T, vh)
    g = -p['A_log'].exp() * F.softplus(a + p['dt_bias'])
    q, k, v, g, beta = (t.transpose(0, 1) for t in (q, k, v, g, torch.sigmoid(b)))
    o = torch.cat([_exact_delta_rule(q[:, s:e], k[:, s:e], v[:, s:e], g[:, s:e], beta[:, s:e])
                   for s, e in zip(bounds[:-1], bounds[1:])], dim=1).transpose(0, 1)
    o = _exact_norm(o, p['out_norm.weight']) * F.silu(z)
    return o.reshape(T, vh * d) @ p['out_proj.weight'].t()


def _exact_gla(q, k, v, decay, bounds):
    out = []
    for s, e in zip(bounds[:-1], bounds[1:]):
        n = torch.arange(e - s, device=DEV, dtype=F64)
        gap = n[:, None] - n[None]
        heads = []
        for h in range(q.shape[1]):
            mix = (decay[h].to(F64) * gap.clamp(min=0)).exp() * (gap >= 0) * q.shape[2] ** -0.5
            heads.append(((q[s:e, h] @ k[s:e, h].t()) * mix) @ v[s:e, h])
        out.append(torch.stack(heads, dim=1))
    return torch.cat(out)


def exact(case, seed):
    s = prepare(case, seed)
    kind, bounds = case['kind'], _bounds(case)

    def wide(t):
        return t.detach().to(F64).requires_grad_(t.requires_grad)

    if 'module' in s:
        p = {n: wide(v) for n, v in sorted(s['module'].named_parameters())}
        s['module'] = None
    if kind == 'attention':
        leaves = [wide(s[n]) for n in 'qkv'] + ([wide(s['sinks'])] if s['sinks'] is not None else [])
        y = _exact_attention(*leaves[:3], bounds, case['window'], leaves[3] if len(leaves) > 3 else None)
    elif kind in ('mlp', 'layer', 'moe', 'gdn'):
        x = wide(s['x'])
        leaves = [x, *p.values()]
        if kind == 'mlp':
            y = _exact_mlp(x, p)
        elif kind == 'layer':
            y = _exact_dense_layer(x, p, case, s['ctx'].cos, s['ctx'].sin)
        elif kind == 'gdn':
            y = _exact_gdn(x, p, case, bounds)
        else:
            y, aux = _exact_moe(x, p, case)
            return [y.detach(), *torch.autograd.grad([y, aux], leaves, [s['dy'].to(F64), torch.ones_like(aux)])]
    elif kind == 'head':
        leaves = [wide(s['h']), wide(s['w'])]
        y = F.cross_entropy(leaves[0] @ leaves[1].t(), s['labels'], reduction='none')
    elif kind == 'gla':
        leaves = [wide(s[n]) for n in 'qkv']
        y = _exact_gla(*leaves, s['decay'], bounds)
    else:
        leaves = list(p.values())
        cos, sin = _rope_tables(bounds, case['dim'])
        h = p['embedding.word_embeddings.weight'][s['ids'].reshape(-1)]
        for i in range(case['layers']):
            pre = f'decoder.layers.{i}.'
            h = _exact_dense_layer(h, {n[len(pre):]: v for n, v in p.items() if n.startswith(pre)}, case, cos, sin)
        logits = _exact_norm(h, p['decoder.final_layernorm.weight']) @ p['output_layer.weight'].t()
        if not case['train']:
            return logits.detach()[None]
        y = F.cross_entropy(logits, s['labels'].reshape(-1), reduction='none')[None]
    return [y.detach(), *torch.autograd.grad(y, leaves, s['dy'].to(F64))]
