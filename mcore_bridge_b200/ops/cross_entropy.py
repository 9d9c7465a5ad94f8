"""Vocab-parallel cross entropy and the fused linear + cross-entropy head.

* :func:`vocab_parallel_cross_entropy` — logits sharded on the vocab dim; max / sum-exp / target-logit
  reduced over the tensor-parallel group (parity: the ``compute_language_model_loss`` call at reference
  ``src/mcore_bridge/model/gpt_model.py:577``).
* :func:`fused_linear_cross_entropy` — the head and the loss in one.  On a GPU the head GEMM's epilogue reduces
  every 128 x 256 accumulator tile to per-row (max, sum-exp) partials and picks out the label's logit
  (``csrc/gemm``, ``EPI_CE_STATS``); the partials of a row are combined, the tensor-parallel ranks exchange their
  ``[T]`` statistics through peer memory (``parallel/dp_comm.py`` all-gather kernel; ``torch.distributed`` elsewhere)
  and the loss follows.  Backward turns the logits, which the forward pass keeps in fp32 while memory is plentiful, into
  their gradient per token chunk and feeds it to the two gradient GEMMs; otherwise only ``[T]`` statistics are kept and
  the head GEMM runs again with an epilogue that writes that gradient directly in bf16 (``EPI_CE_GRAD``).  On CPU the
  same chunked algorithm runs on torch ops.

Both return the per-token loss ``[T]`` in fp32 (the caller masks and averages).
"""
from __future__ import annotations

import ctypes
import threading
import weakref

import torch
import torch.distributed as dist

from ..parallel import state as ps
from . import _lib, gemm

_ll, _int, _f = ctypes.c_longlong, ctypes.c_int, ctypes.c_float


def _tp_info(group: str):
    n = ps.get_world_size(group)
    r = ps.get_rank_in(group) if n > 1 else 0
    return n, r, (ps.get_group(group) if n > 1 else None)


def _stats_torch(logits: torch.Tensor, labels: torch.Tensor, vocab_start: int):
    """Per-row (max, sum exp(l - max), target logit or 0) over the local vocab shard."""
    lf = logits.float()
    vl = lf.shape[-1]
    m = lf.max(dim=-1).values
    s = torch.exp(lf - m[:, None]).sum(-1)
    local = labels - vocab_start
    ok = (local >= 0) & (local < vl)
    tgt = lf.gather(1, local.clamp(0, vl - 1)[:, None]).squeeze(1)
    tgt = torch.where(ok, tgt, torch.zeros_like(tgt))
    return m, s, tgt


def _stats(logits, labels, vocab_start):
    if logits.is_cuda and logits.dtype in (torch.float32, torch.bfloat16) and _lib.available():
        rows, vl = logits.shape
        m = torch.empty(rows, dtype=torch.float32, device=logits.device)
        s = torch.empty_like(m)
        t = torch.empty_like(m)
        rc = _lib.lib().mcb_ce_stats(_lib.ptr(logits), _int(int(logits.dtype == torch.float32)), _ll(logits.stride(0)),
                                     _lib.ptr(labels), _ll(rows), _int(vl), _int(vocab_start), _lib.ptr(m),
                                     _lib.ptr(s), _lib.ptr(t), _lib.stream_ptr())
        _lib.check_rc(rc, 'mcb_ce_stats')
        return m, s, t
    return _stats_torch(logits, labels, vocab_start)


def _reduce_stats(m, s, tgt, group):
    """Combine per-shard softmax statistics across the tensor-parallel group -> (lse, target logit)."""
    if group is not None:
        gm = m.clone()
        dist.all_reduce(gm, op=dist.ReduceOp.MAX, group=group)
        packed = torch.stack([s * torch.exp(m - gm), tgt])
        dist.all_reduce(packed, group=group)
        s, tgt, m = packed[0], packed[1], gm
    return m + torch.log(s), tgt


def _dlogits(logits, labels, vocab_start, lse, g, out_dtype):
    """``(softmax - onehot) * g`` for the local shard."""
    if logits.is_cuda and _lib.available() and logits.dtype in (torch.float32, torch.bfloat16):
        rows, vl = logits.shape
        out = torch.empty((rows, vl), dtype=torch.bfloat16, device=logits.device) if out_dtype == torch.bfloat16 \
            else torch.empty((rows, vl), dtype=torch.float32, device=logits.device)
        rc = _lib.lib().mcb_ce_dlogits(_lib.ptr(logits), _int(int(logits.dtype == torch.float32)),
                                       _ll(logits.stride(0)), _lib.ptr(labels), _lib.ptr(lse), _lib.ptr(g), _ll(rows),
                                       _int(vl), _int(vocab_start), _lib.ptr(out),
                                       _int(int(out.dtype == torch.float32)), _lib.stream_ptr())
        _lib.check_rc(rc, 'mcb_ce_dlogits')
        return out
    lf = logits.float()
    vl = lf.shape[-1]
    p = torch.exp(lf - lse[:, None])
    local = labels - vocab_start
    ok = (local >= 0) & (local < vl)
    p[torch.arange(p.shape[0], device=p.device)[ok], local[ok]] -= 1.0
    return (p * g[:, None]).to(out_dtype)


_STATS_WS = {}


def _reduce_stats_peer(m, s, tgt, group_name):
    """Same combination as :func:`_reduce_stats`, with the ranks' ``[3, T]`` statistics exchanged by the in-tree
    peer-memory all-gather kernel instead of two NCCL all-reduces."""
    from ..parallel import dp_comm
    n, r = ps.get_world_size(group_name), ps.get_rank_in(group_name)
    T = m.numel()
    per = 3 * T
    per_al = (per + 3) // 4 * 4                     # 16-byte multiples per rank
    cur = _STATS_WS.get(group_name)
    if cur is None or cur[1].numel() < n * per_al:
        if cur is not None:
            torch.cuda.synchronize()
        cur = _STATS_WS[group_name] = dp_comm.allocate(group_name, n * max(per_al, 1 << 16), torch.float32)
    ws, flat = cur
    mine = flat[r * per_al:r * per_al + per].view(3, T)
    mine[0].copy_(m)
    mine[1].copy_(s)
    mine[2].copy_(tgt)
    dp_comm.all_gather_(ws, flat, 0, n * per_al)
    allr = flat[:n * per_al].view(n, per_al)[:, :per].view(n, 3, T)
    gm = allr[:, 0].max(dim=0).values
    ssum = (allr[:, 1] * torch.exp(allr[:, 0] - gm)).sum(0)
    return gm + torch.log(ssum), allr[:, 2].sum(0)


def _combine(m, s, tgt, group_name, group):
    if group is not None and m.is_cuda:
        from ..parallel import dp_comm
        if dp_comm.usable(group_name, m.device):
            return _reduce_stats_peer(m, s, tgt, group_name)
    return _reduce_stats(m, s, tgt, group)


def _head_kernel_ok(h2, weight) -> bool:
    return (h2.is_cuda and h2.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and _lib.available()
            and h2.shape[1] % 8 == 0 and weight.is_contiguous())


_KEEP_MIN_HIDDEN = 1024
_KEEP_SHARE = 32                 # of a device's memory, all kept logits together
_KEEP_ASK = 1 << 28              # buffers from here on ask the driver what is free each time


class _Kept:
    """Logits that a graph holds for its backward pass, until that or :func:`release_kept_logits` takes them."""

    def __init__(self, logits):
        self.logits = logits
        with _kept_lock:
            _kept.add(self)

    def take(self):
        return self.__dict__.pop('logits', None)       # one of several threads gets them


_kept: 'weakref.WeakSet[_Kept]' = weakref.WeakSet()
_kept_lock = threading.Lock()
_device_bytes: dict = {}         # device -> its memory
_driver_free: dict = {}          # device -> (bytes the allocator held, bytes the driver had left), when last asked


def _kept_on(device) -> list:
    """``(holder, logits)`` of the graphs on ``device`` that hold some."""
    if not len(_kept):
        return []
    with _kept_lock:
        pairs = [(k, k.__dict__.get('logits')) for k in _kept]
    return [(k, t) for k, t in pairs if t is not None and t.device == device]


def release_kept_logits(device) -> None:
    """Gives back the logits that graphs still hold: their backward passes form them again, with the same bits.  A model
    calls this before a forward pass, whose activations had that memory to themselves when no logits were kept."""
    for holder, _ in _kept_on(device):
        holder.take()


def _memory_left(device, need: int) -> int:
    """Bytes this process can still allocate: unused ones of its allocator and what the driver has for it.  The driver
    takes 60 to 130 us; a small buffer makes do with its answer of the last time the allocator grew or shrank."""
    reserved, allocated = _lib.native().memory(device.index)
    seen = _driver_free.get(device.index)
    if need > _KEEP_ASK or seen is None or seen[0] != reserved:
        free, total = torch.cuda.mem_get_info(device)
        own = int(torch.cuda.get_per_process_memory_fraction(device) * total) - reserved
        seen = _driver_free[device.index] = (reserved, max(0, min(free, own)))
    return reserved - allocated + seen[1]


def _logits_to_keep(T, vl, H, device, backward: int = 0):
    """A ``[T, vl]`` fp32 buffer that saves the backward pass the second head product, or ``None``.

    A kept logit costs 8 bytes of traffic and 4 of memory until the backward pass, a recomputed one ``2 H`` operations: at
    6.5 TB/s and 1.4 PFLOP/s the two are even near ``H`` = 860.  Forward + backward, us, recomputed and kept: 4096 x 151936
    at ``H`` 4096 14808 / 12990, 2048 7173 / 6743, 1024 4420 / 3941; 64 x 151936 at 4096 1347 / 1165.

    Memory comes first: a buffer is kept where the device has four times as much to spare beyond the ``backward`` bytes
    the head's own backward pass allocates, and where all that are kept stay within a 32nd of the device.  In a captured
    graph a buffer would last as long as the graph, so none is kept there."""
    if T == 0 or vl % 8 or H < _KEEP_MIN_HIDDEN or torch.cuda.is_current_stream_capturing():
        return None
    need = 4 * T * vl
    held = sum(4 * t.numel() for _, t in _kept_on(device))
    if device not in _device_bytes:
        _device_bytes[device] = torch.cuda.get_device_properties(device).total_memory
    if (held + need) * _KEEP_SHARE > _device_bytes[device]:
        return None
    if _memory_left(device, need) < 4 * need + backward:
        return None
    try:
        return torch.empty((T, vl), dtype=torch.float32, device=device)
    except torch.OutOfMemoryError:       # free, but in pieces
        return None


def _backward_bytes(T, chunk, weight, need_dh, need_dw) -> int:
    """What the head's backward pass allocates beside kept logits: a chunk's gradient of the logits and the results."""
    vl, H = weight.shape
    one = T <= chunk
    dw = 0 if not need_dw or getattr(weight, 'main_grad', None) is not None else (2 if one else 6) * vl * H
    return 2 * min(T, chunk) * vl + 2 * T * H * need_dh + dw


def _head_stats(h2, weight, lab, vocab_start, logits=None):
    """(max, sum exp, label logit) of every row over the local vocabulary shard, from the GEMM epilogue; the logits go
    to ``logits`` when that is given."""
    T, H = h2.shape
    vl = weight.shape[0]
    tiles_n = (vl + 255) // 256
    part = torch.empty((T, tiles_n, 2), dtype=torch.float32, device=h2.device)
    tgt = torch.zeros(T, dtype=torch.float32, device=h2.device)
    rc = _lib.lib().mcb_gemm_ce_bf16(_lib.ptr(h2), _ll(h2.stride(0)), _lib.ptr(weight), _ll(weight.stride(0)), _int(T),
                                     _int(vl), _int(H), _lib.ptr(lab), _int(vocab_start), _lib.ptr(part), _lib.ptr(tgt),
                                     None, None, _lib.ptr(logits), _ll(vl), _int(0),
                                     _lib.ptr(_lib.status_word(h2.device)), _lib.stream_ptr())
    _lib.check_rc(rc, 'mcb_gemm_ce_bf16')
    return *_lib.native().ce_combine(part), tgt


def _head_dlogits(h2, weight, lab, vocab_start, lse, g):
    T, H = h2.shape
    vl = weight.shape[0]
    d = torch.empty((T, vl), dtype=torch.bfloat16, device=h2.device)
    rc = _lib.lib().mcb_gemm_ce_bf16(_lib.ptr(h2), _ll(h2.stride(0)), _lib.ptr(weight), _ll(weight.stride(0)), _int(T),
                                     _int(vl), _int(H), _lib.ptr(lab), _int(vocab_start), None, None, _lib.ptr(lse),
                                     _lib.ptr(g), _lib.ptr(d), _ll(d.stride(0)), _int(1),
                                     _lib.ptr(_lib.status_word(h2.device)), _lib.stream_ptr())
    _lib.check_rc(rc, 'mcb_gemm_ce_bf16')
    return d


def _kept_dlogits(logits, lab, vocab_start, lse, g):
    """What :func:`_head_dlogits` forms, from logits that the forward pass kept: the same bits."""
    rows, vl = logits.shape
    d = torch.empty((rows, vl), dtype=torch.bfloat16, device=logits.device)
    rc = _lib.lib().mcb_ce_dlogits_head(_lib.ptr(logits), _lib.ptr(lab), _lib.ptr(lse), _lib.ptr(g), _ll(rows),
                                        _int(vl), _int(vocab_start), _lib.ptr(d), _lib.stream_ptr())
    _lib.check_rc(rc, 'mcb_ce_dlogits_head')
    return d


class _VocabParallelCE(torch.autograd.Function):

    @staticmethod
    def forward(ctx, logits, labels, group_name):
        n, r, group = _tp_info(group_name)
        vl = logits.shape[-1]
        l2 = logits.reshape(-1, vl)
        lab = labels.reshape(-1).to(torch.int64)
        m, s, tgt = _stats(l2, lab, r * vl)
        lse, tgt = _reduce_stats(m, s, tgt, group)
        ctx.save_for_backward(l2, lab, lse)
        ctx.vocab_start, ctx.shape = r * vl, logits.shape
        return (lse - tgt).view(labels.shape)

    @staticmethod
    def backward(ctx, g):
        l2, lab, lse = ctx.saved_tensors
        d = _dlogits(l2, lab, ctx.vocab_start, lse, g.reshape(-1).float().contiguous(), l2.dtype)
        return d.view(ctx.shape), None, None


def vocab_parallel_cross_entropy(logits: torch.Tensor, labels: torch.Tensor, group: str = 'tp') -> torch.Tensor:
    """``logits [..., V/tp]``, ``labels [...]`` (global ids) -> per-token loss (fp32)."""
    return _VocabParallelCE.apply(logits, labels, group)


class _FusedLinearCE(torch.autograd.Function):

    @staticmethod
    def forward(ctx, h, weight, labels, group_name, chunk, graph):
        n, r, group = _tp_info(group_name)
        vl, H = weight.shape
        h2 = h.reshape(-1, H)
        lab = labels.reshape(-1).to(torch.int64)
        T = h2.shape[0]
        if h2.stride(1) != 1 or h2.stride(0) % 8:
            h2 = h2.contiguous()
        if _head_kernel_ok(h2, weight):
            logits = None
            if graph:
                need = _backward_bytes(T, chunk, weight, *ctx.needs_input_grad[:2])
                logits = _logits_to_keep(T, vl, H, h2.device, need)
            if logits is not None:
                ctx.kept = _Kept(logits)
            m, s, tgt = _head_stats(h2, weight, lab, r * vl, logits)
            if group is None and m.is_cuda:
                lse_all, loss = _lib.native().ce_loss(m, s, tgt)
            else:
                lse_all, tgt = _combine(m, s, tgt, group_name, group)
                loss = lse_all - tgt
            ctx.save_for_backward(h2, weight, lab, lse_all)
            ctx.meta = (group_name, chunk, r * vl, h.shape, labels.shape)
            return loss.view(labels.shape)
        loss = torch.empty(T, dtype=torch.float32, device=h.device)
        lse_all = torch.empty(T, dtype=torch.float32, device=h.device)
        ldt = torch.float32
        for s0 in range(0, T, chunk):
            s1 = min(T, s0 + chunk)
            logits = gemm.mm_nt(h2[s0:s1], weight, out_dtype=ldt)
            m, s, tgt = _stats(logits, lab[s0:s1], r * vl)
            lse, tgt = _reduce_stats(m, s, tgt, group)
            loss[s0:s1] = lse - tgt
            lse_all[s0:s1] = lse
            del logits
        ctx.save_for_backward(h2, weight, lab, lse_all)
        ctx.meta = (group_name, chunk, r * vl, h.shape, labels.shape)
        return loss.view(labels.shape)

    @staticmethod
    def backward(ctx, g):
        h2, weight, lab, lse = ctx.saved_tensors
        group_name, chunk, vstart, hshape, _ = ctx.meta
        n, r, group = _tp_info(group_name)
        T, H = h2.shape
        g = g.reshape(-1).float().contiguous()
        dh = torch.empty_like(h2)
        mg = getattr(weight, 'main_grad', None)
        dw = None
        need_dw = ctx.needs_input_grad[1]
        ddt = h2.dtype if h2.dtype == torch.bfloat16 else torch.float32
        fused = _head_kernel_ok(h2, weight)
        kept = getattr(ctx, 'kept', None)
        kept = None if kept is None else kept.take()            # a second pass over the graph forms them again
        # without `main_grad` the chunks' products are summed in fp32 and rounded once; a single chunk needs no such
        # buffer (at 151936 x 4096 it costs 2.5 GB of zero fill, accumulation and conversion), its GEMM rounds itself
        one_chunk = 0 < T <= chunk and mg is None and weight.dtype in (torch.bfloat16, torch.float32)
        if need_dw and mg is None and not one_chunk:
            alloc = torch.empty if T > 0 else torch.zeros
            dw = alloc(weight.shape, dtype=torch.float32, device=weight.device)
        for s0 in range(0, T, chunk):
            s1 = min(T, s0 + chunk)
            if kept is not None:
                d = _kept_dlogits(kept[s0:s1], lab[s0:s1], vstart, lse[s0:s1], g[s0:s1])
            elif fused:
                d = _head_dlogits(h2[s0:s1], weight, lab[s0:s1], vstart, lse[s0:s1], g[s0:s1])
            else:
                logits = gemm.mm_nt(h2[s0:s1], weight, out_dtype=torch.float32)
                d = _dlogits(logits, lab[s0:s1], vstart, lse[s0:s1], g[s0:s1], ddt)
                del logits
            gemm.mm_nn(d, weight, out=dh[s0:s1])
            if need_dw and one_chunk:
                dw = gemm.mm_tn(d, h2, out_dtype=weight.dtype)
            elif need_dw:
                gemm.mm_tn(d, h2[s0:s1], out=mg if mg is not None else dw, accumulate=mg is not None or s0 > 0)
            del d
        del kept
        # dh is this vocab shard's partial gradient: the caller's input mapping (copy-to-region or
        # sequence-parallel gather) sums it over the tensor-parallel group in its own backward.
        if need_dw and mg is not None:
            hook = getattr(weight, 'grad_ready_hook', None)
            if hook is not None:
                hook()
        return dh.view(hshape), (dw.to(weight.dtype) if dw is not None else None), None, None, None, None


def fused_linear_cross_entropy(h: torch.Tensor, weight: torch.Tensor, labels: torch.Tensor, group: str = 'tp',
                               chunk: int = 4096) -> torch.Tensor:
    """``h [T, H]`` (full sequence on every TP rank), ``weight [V/tp, H]``, ``labels [T]`` -> loss ``[T]`` fp32."""
    # asked here: inside the function grad mode is off, and ``needs_input_grad`` does not depend on it.  Hooks on saved
    # tensors (checkpointing, offload) spare device memory: logits beside them would undo that.
    graph = (torch.is_grad_enabled() and (h.requires_grad or weight.requires_grad)
             and torch._C._autograd._top_saved_tensors_default_hooks(True) is None)
    return _FusedLinearCE.apply(h, weight, labels, group, chunk, graph)
