"""Results that a backward pass forms again or finds kept, tile widths of the GEMM, growing maxima in attention: at the sizes
where they can go wrong, against 64-bit references."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = 'cuda'


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-30)).item()


@pytest.mark.parametrize('T,V,H,chunk', [(515, 4104, 1024, 4096),      # ragged rows, a last column tile with 8 columns
                                         (1, 264, 1032, 4096),
                                         (1030, 2056, 1024, 600)])     # two chunks of kept logits
def test_head_loss_with_kept_logits(T, V, H, chunk):
    from mcore_bridge_b200.ops import cross_entropy as ce
    gen = torch.Generator(device=DEV).manual_seed(1)
    h = torch.randn(T, H, generator=gen, device=DEV).bfloat16().requires_grad_()
    w = (torch.randn(V, H, generator=gen, device=DEV) * 0.05).bfloat16().requires_grad_()
    lab = torch.randint(0, V, (T,), generator=gen, device=DEV)
    lab[0] = V - 1
    g = torch.rand(T, generator=gen, device=DEV)
    assert ce._logits_to_keep(T, V, H, h.device) is not None
    loss = ce.fused_linear_cross_entropy(h, w, lab, chunk=chunk)
    kept = torch.autograd.grad(loss, (h, w), g, retain_graph=True)
    again = torch.autograd.grad(loss, (h, w), g)                        # the logits are gone: formed a second time
    hw, ww = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    ref = torch.nn.functional.cross_entropy(hw @ ww.t(), lab, reduction='none')
    want = torch.autograd.grad(ref, (hw, ww), g.double())
    # logits and their sums are fp32; dlogits and the results are rounded to bf16, 2^-9 each
    assert (loss.double() - ref).abs().max() < 1e-4
    for got in (kept, again):
        assert _rel(got[0], want[0]) < 2 ** -8 and _rel(got[1], want[1]) < 2 ** -8


@pytest.mark.parametrize('rows', [1, 7, 130])
@pytest.mark.parametrize('H', [264, 1032, 4104])       # one, one and several vectors a thread, the last ones partly idle
def test_norm_linear_recomputes_the_normalised_input(rows, H):
    from mcore_bridge_b200.ops import fused_mlp
    gen = torch.Generator(device=DEV).manual_seed(2)
    x = torch.randn(rows, H, generator=gen, device=DEV).bfloat16().requires_grad_()
    lw = (1 + 0.1 * torch.randn(H, generator=gen, device=DEV)).bfloat16().requires_grad_()
    w = (torch.randn(72, H, generator=gen, device=DEV) * 0.05).bfloat16().requires_grad_()
    dy = torch.randn(rows, 72, generator=gen, device=DEV).bfloat16()
    y = fused_mlp.norm_linear(x, lw, w, 1e-6, False)
    got = [y, *torch.autograd.grad(y, (x, lw, w), dy)]
    xd, ld, wd = (t.detach().double().requires_grad_() for t in (x, lw, w))
    ref = (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * ld) @ wd.t()
    want = [ref, *torch.autograd.grad(ref, (xd, ld, wd), dy.double())]
    # at most the normalised input, its gradient and the result are rounded to bf16: 3 x 2^-9
    for a, b in zip(got, want):
        assert _rel(a, b) < 2 ** -7


@pytest.mark.parametrize('rows', [1, 7, 130])
@pytest.mark.parametrize('F', [264, 1536])
def test_glu_linear_recomputes_the_activation(rows, F):
    from mcore_bridge_b200.ops import fused_mlp
    gen = torch.Generator(device=DEV).manual_seed(3)
    h = torch.randn(rows, 2 * F, generator=gen, device=DEV).bfloat16().requires_grad_()
    w = (torch.randn(72, F, generator=gen, device=DEV) * 0.05).bfloat16().requires_grad_()
    dy = torch.randn(rows, 72, generator=gen, device=DEV).bfloat16()
    y = fused_mlp.glu_linear(h, w, 0, 0.0, 0.0)
    got = [y, *torch.autograd.grad(y, (h, w), dy)]
    hd, wd = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    gate, up = hd.chunk(2, dim=-1)
    ref = (torch.nn.functional.silu(gate) * up) @ wd.t()
    want = [ref, *torch.autograd.grad(ref, (hd, wd), dy.double())]
    for a, b in zip(got, want):
        assert _rel(a, b) < 2 ** -7


@pytest.mark.parametrize('M,N,K', [(1, 8, 8), (129, 264, 72), (300, 1000, 64), (520, 2056, 200)])
def test_gemm_tile_widths_agree(M, N, K):
    """Every width adds the same products in the same order; operands of both layouts, remainders in all three extents."""
    from mcore_bridge_b200.ops import gemm
    gen = torch.Generator(device=DEV).manual_seed(4)
    x = torch.randn(M, K, generator=gen, device=DEV).bfloat16()
    w = torch.randn(N, K, generator=gen, device=DEV).bfloat16()
    dy = torch.randn(M, N, generator=gen, device=DEV).bfloat16()
    ref = {'nt': x.double() @ w.double().t(), 'nn': dy.double() @ w.double(), 'tn': dy.double().t() @ x.double()}
    for bn in (0, 64, 128, 256, 512):
        got = {'nt': gemm.mm_nt(x, w, force_bn=bn), 'nn': gemm.mm_nn(dy, w, force_bn=bn),
               'tn': gemm.mm_tn(dy, x, force_bn=bn)}
        for k, r in ref.items():
            # fp32 sums of at most 2056 products (1e-5 of their size), rounded to bf16
            assert ((got[k].double() - r).abs() <= 2 ** -8 * r.abs() + 1e-3).all(), (k, bn)


@pytest.mark.parametrize('T,nq,nkv,d', [(300, 2, 1, 64), (2500, 3, 1, 128), (3000, 32, 8, 128)])
def test_attention_maxima_that_grow_with_every_block(T, nq, nkv, d):
    """Every block raises the maxima of its rows, which rescales every accumulator every time; split tiles, pairs of heads."""
    from mcore_bridge_b200.ops.attention import attention
    gen = torch.Generator(device=DEV).manual_seed(5)
    q = torch.rand(T, nq, d, generator=gen, device=DEV).bfloat16() + 0.5
    ramp = torch.linspace(0.1, 2.0, T, device=DEV)[:, None, None]
    k = (torch.rand(T, nkv, d, generator=gen, device=DEV) * ramp).bfloat16()
    v = torch.randn(T, nkv, d, generator=gen, device=DEV).bfloat16()
    o = attention(q, k, v)
    kk, vv = (t.double().repeat_interleave(nq // nkv, dim=1).transpose(0, 1) for t in (k, v))
    mask = torch.ones(T, T, dtype=torch.bool, device=DEV).triu(1)
    for h in range(nq):
        s = (q[:, h].double() @ kk[h].t() * d ** -0.5).masked_fill(mask, float('-inf'))
        # probabilities and the result are rounded to bf16, 2^-9 each
        assert _rel(o[:, h], torch.softmax(s, dim=-1) @ vv[h]) < 2 ** -8


@pytest.mark.parametrize('hidden,ffn', [(192, 320), (128, 64)])         # 2.5 and half a column tile
def test_expert_widths_that_end_inside_a_tile(monkeypatch, hidden, ffn):
    """Results of the gather + expert GEMM leave through shared memory."""
    from mcore_bridge_b200.layers.moe import MoELayer
    from mcore_bridge_b200.ops import _lib
    from mcore_bridge_b200.train.presets import model_config
    cfg = model_config('qwen3_moe_tiny', dict(hidden_size=hidden, moe_intermediate_size=ffn, num_experts=8,
                                              num_experts_per_tok=2), bf16=True)
    gen = torch.Generator(device=DEV).manual_seed(6)
    with torch.device(DEV):
        layer = MoELayer(cfg).train()
    with torch.no_grad():
        for p in layer.parameters():
            p.copy_(torch.randn(p.shape, generator=gen, device=DEV) * 0.1)
    x = torch.randn(333, hidden, generator=gen, device=DEV).bfloat16()
    dy = torch.randn(333, hidden, generator=gen, device=DEV).bfloat16()
    res = {}
    for fused in ('1', '0'):
        monkeypatch.setenv('MCB200_FUSED_MOE', fused)
        xx = x.clone().requires_grad_()
        y = layer(xx)
        res[fused] = [y, *torch.autograd.grad(y, [xx, *layer.parameters()], dy)]
    _lib.check_status()
    # either path rounds the hidden rows, their activation, the expert outputs and the result to bf16: 4 x 2^-9 each
    for a, b in zip(res['1'], res['0']):
        assert _rel(a, b) < 2 ** -6


@pytest.mark.parametrize('T', [1, 511, 2050])                            # fewer tokens than threads, a remainder, many a thread
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('d', [64, 128])                                  # delta in the dQ kernel; 128: in it for few rows
def test_sink_and_window_gradients(T, dtype, d):
    from mcore_bridge_b200.ops.attention import attention, attention_ref
    gen = torch.Generator(device=DEV).manual_seed(8)
    nq, nkv = 20, 4
    q, k, v = (torch.randn(T, n, d, generator=gen, device=DEV).bfloat16().requires_grad_() for n in (nq, nkv, nkv))
    sinks = torch.randn(nq, generator=gen, device=DEV).to(dtype).requires_grad_()
    dy = torch.randn(T, nq, d, generator=gen, device=DEV).bfloat16()
    o = attention(q, k, v, window=(100, 0), sinks=sinks)
    got = [o, *torch.autograd.grad(o, (q, k, v, sinks), dy)]
    leaves = [t.detach().float().requires_grad_() for t in (q, k, v, sinks)]
    ref = attention_ref(*leaves[:3], window=(100, 0), sinks=leaves[3])
    want = [ref, *torch.autograd.grad(ref, leaves, dy.float())]
    # probabilities, dS and the results are rounded to bf16, 2^-9 each; a sink's gradient sums T products of such results
    for a, b, bound in zip(got, want, [2 ** -8] + 3 * [2 ** -6] + [2 ** -6]):
        if T > 1 or b.abs().max() > 1e-3:          # one token: P = 1 - p_sink, no gradient reaches beyond rounding in places
            assert _rel(a, b) < bound


@pytest.mark.parametrize('T,k,H', [(1, 4, 8), (37, 8, 520), (130, 5, 2048), (9, 8, 1032), (37, 3, 520), (37, 9, 520)])
def test_expert_rows_are_summed_in_order(T, k, H):
    """Rows that were not sent count as zero; pieces of 256 columns, the last one ragged; fewer than 4 or more than 8 rows
    take the other kernel."""
    import ctypes

    from mcore_bridge_b200.ops import _lib
    gen = torch.Generator(device=DEV).manual_seed(4)
    rows, experts = T * k + 3, 4
    y = torch.randn(rows, H, generator=gen, device=DEV).bfloat16()
    scalar = torch.rand(rows, generator=gen, device=DEV)
    idx = torch.randint(0, experts, (T, k), generator=gen, device=DEV, dtype=torch.int32)
    sent = torch.randperm(rows, generator=gen, device=DEV)[:T * k].view(T, k).int()
    sent[0, 0] = -1
    out = torch.empty(T, H, dtype=torch.bfloat16, device=DEV)
    got = torch.empty(T, k, device=DEV)
    table, scalars = ((ctypes.c_void_p * 1)(t.data_ptr()) for t in (y, scalar))
    rc = _lib.lib().mcb_moe_combine(table, scalars, *map(ctypes.c_int, (1, T, k, experts, H)), _lib.ptr(idx), _lib.ptr(sent),
                                    _lib.ptr(out), _lib.ptr(got), _lib.stream_ptr())
    _lib.check_rc(rc, 'mcb_moe_combine')
    hit = (sent >= 0)
    want = torch.zeros(T, H, device=DEV)
    for j in range(k):                                  # the kernels' order, in 32 bits: equal bits
        want += torch.where(hit[:, j, None], y[sent[:, j].clamp(min=0).long()].float(), 0.)
    assert torch.equal(out, want.bfloat16())
    assert torch.equal(got, torch.where(hit, scalar[sent.clamp(min=0).long()], 0.))


@pytest.mark.parametrize('T,nq,d', [(1, 1, 64), (200, 4, 64), (130, 3, 128),      # delta formed in the dQ kernel
                                    (3641, 9, 128)])                               # by the kernel of its own: 32769 rows
def test_attention_delta_has_one_order_of_sums(T, nq, d):
    """delta of a row has the same bits whichever kernel forms it: eight products of bf16 values, which are exact in fp32, added in
    pairs, then a tree over the D / 8 sums."""
    import ctypes

    from mcore_bridge_b200.ops import _lib
    gen = torch.Generator(device=DEV).manual_seed(9)
    q, o, do = (torch.randn(T, nq, d, generator=gen, device=DEV).bfloat16() for _ in range(3))
    k, v = (torch.randn(T, 1, d, generator=gen, device=DEV).bfloat16() for _ in range(2))
    lse = torch.full((nq, T), 10.0, device=DEV)
    start = torch.zeros(T, dtype=torch.int32, device=DEV)
    delta = torch.full((nq, T), float('nan'), device=DEV)
    dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
    rc = _lib.lib().mcb_attn_bwd_ranges(*map(_lib.ptr, (q, k, v, o, do, lse, delta)), ctypes.c_int(0), _lib.ptr(start), None, None,
                                        None, _lib.ptr(dq), _lib.ptr(dk), _lib.ptr(dv), *map(ctypes.c_int, (T, T, nq, 1, d)),
                                        ctypes.c_float(0.1), None, ctypes.c_int(1), _lib.ptr(_lib.status_word(q.device)),
                                        _lib.stream_ptr())
    _lib.check_rc(rc, 'mcb_attn_bwd_ranges')
    pairs = (o.float() * do.float()).view(T, nq, d // 8, 4, 2)
    pairs = pairs[..., 0] + pairs[..., 1]
    term = ((pairs[..., 0] + pairs[..., 1]) + pairs[..., 2]) + pairs[..., 3]
    while term.shape[-1] > 1:
        half = term.shape[-1] // 2
        term = term[..., :half] + term[..., half:]
    assert torch.equal(delta, term[..., 0].t())


@pytest.mark.parametrize('nq,T', [(4096, 1), (3, 2050), (2, 70001)])    # one term; a few and many terms a thread
def test_sink_gradient_in_full_fp32_precision(nq, T):
    import ctypes

    from mcore_bridge_b200.ops import _lib
    gen = torch.Generator(device=DEV).manual_seed(10)
    # differences of multiples of 2^-12 below 64 are exact in fp32
    sinks = torch.randint(-4096 * 8, 4096 * 8, (nq,), generator=gen, device=DEV) / 4096
    lse = sinks[:, None] + torch.randint(0, 4096 * 16, (nq, T), generator=gen, device=DEV) / 4096
    delta = torch.randn(nq, T, generator=gen, device=DEV)
    out = torch.empty(nq, device=DEV)
    rc = _lib.lib().mcb_attn_sink_grad(*map(_lib.ptr, (sinks, lse, delta, out)), *map(ctypes.c_int, (0, T, nq)),
                                       _lib.stream_ptr())
    _lib.check_rc(rc, 'mcb_attn_sink_grad')
    terms = torch.exp(sinks.double()[:, None] - lse.double()) * delta.double()
    # expf is within one unit in the last place (2^-23), a product rounds by half of one; then a thread's sums, its warp's
    # five and the block's sixteen round by half of one of a partial sum each
    adds = (T + 511) // 512 - 1 + 5 + 16 if T > 1 else 0
    bound = (1.5 + 0.5 * adds) * 2.0 ** -23 * terms.abs().sum(1)
    assert ((out.double() + terms.sum(1)).abs() <= bound).all()
