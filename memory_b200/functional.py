"""Autograd bindings of the CUDA operators.

Three differentiable pieces mirror the reference's sequence-level memory layer
(memory_transformer/model.py:624-692 followed by memory_block.py:549-558):

``route``             router forward/backward (router.py:94-156, 197-260; model.py:356-391)
``gather_chapters``   chapter gather + optional row norm + weight scaling (memory_bank.py:244-293,
                      model.py:393-432, 689-692), backward scatters only into touched chapters
``cross_attention``   Q/K/V/O projections and joint-softmax attention over already gathered rows
                      (memory_attention.py:209-261, 298-316, 452-478)

``memory_layer`` chains them without materialising anything on the host.
"""
from __future__ import annotations

import os
from typing import Dict, Optional, Tuple

import torch

from . import _lib as L
from . import ops

LOSS_KEYS = ("load_balance", "auxiliary", "z_loss", "entropy")


_KERNEL_DTYPES = (torch.float32, torch.bfloat16)


def _cast(v, dtype):
    return v if v is None or v.dtype == dtype else v.to(dtype)


# A pass that is one native call takes raw pointers and the sizes of its descriptor; what a tensor's shape says against
# those sizes is refused here, before the descriptor is filled.
def _check_width(name: str, t: torch.Tensor, width: int) -> None:
    if t.dim() != 2 or t.shape[1] != width:
        raise ValueError(f"inner dimensions differ: {name} {tuple(t.shape)} vs {width}")


def _check_numel(name: str, t: Optional[torch.Tensor], n: int) -> None:
    if t is not None and t.numel() != n:
        raise ValueError(f"{name} must have {n} elements, got shape {tuple(t.shape)}")


def _check_projections(d: int, mem_dim: int, wq, wk, wv, wo, num_heads: int, num_kv_heads: int) -> None:
    q, k, v, o = wq.shape, wk.shape, wv.shape, wo.shape
    if num_heads > 0 and d % num_heads == 0 and q == o == (d, d) and k == v == (num_kv_heads * (d // num_heads), mem_dim):
        return
    for name, shape, width in (("wq", q, d), ("wk", k, mem_dim), ("wv", v, mem_dim), ("wo", o, q[0])):
        if len(shape) != 2 or shape[1] != width:
            raise ValueError(f"inner dimensions differ: {name} {tuple(shape)} vs {width}")
    if num_heads <= 0 or num_kv_heads <= 0 or q[0] % num_heads != 0:
        raise ValueError(f"wq {tuple(q)} does not hold {num_heads} heads")
    dkv = num_kv_heads * (q[0] // num_heads)
    if k[0] != dkv or v[0] != dkv:
        raise ValueError(f"wk {tuple(k)} and wv {tuple(v)} must have num_kv_heads * head_dim = {dkv} rows")


class _LossDict(dict):
    """Router loss dict (same keys as the reference) that also carries the raw 4-vector as ``.vector`` (order of
    LOSS_KEYS), for a single backward seed and a single-kernel weighted sum.  A dict somebody has changed no longer
    says what the vector does and drops it."""

    def __init__(self, vector: torch.Tensor):
        super().__init__(zip(LOSS_KEYS, vector.unbind()))
        self.vector = vector

    def _changed(name):
        method = getattr(dict, name)

        def change(self, *args, **kwargs):
            self.vector = None
            return method(self, *args, **kwargs)
        return change

    __setitem__, __delitem__, __ior__ = _changed("__setitem__"), _changed("__delitem__"), _changed("__ior__")
    update, pop, popitem = _changed("update"), _changed("pop"), _changed("popitem")
    clear, setdefault = _changed("clear"), _changed("setdefault")
    del _changed


class _WeightedLosses(torch.autograd.Function):
    @staticmethod
    def forward(ctx, vector, coefs):
        ctx.coefs = coefs
        ctx.save_for_backward(vector)
        return ops.loss_total(vector, coefs)

    @staticmethod
    def backward(ctx, g):
        return ops.loss_total(ctx.saved_tensors[0], ctx.coefs, g.float()), None


def weighted_losses(losses: _LossDict, **coefs: float) -> torch.Tensor:
    """sum of coefficient * loss over the coefficients that are positive (router.py:490-527), one kernel each way."""
    return _WeightedLosses.apply(losses.vector, tuple(max(0.0, float(coefs.get(k, 0.0))) for k in LOSS_KEYS))


class SparseBankGrad:
    """Receives bank gradients as (chapter ids, [U*T, d] rows) instead of a dense tensor.

    Attach one to a bank parameter with ``param.moc_sparse_grad = SparseBankGrad()``; backward
    passes then append here and return no dense gradient for the bank.
    """

    def __init__(self, wire_dtype: Optional[torch.dtype] = None, wire_only: bool = False):
        self.entries = []   # list of (uniq int32 [n_pairs], num_unique int32 [1], rows fp32 [n_pairs*T, d], T)
        self.wire = []      # per entry: the same rows in ``wire_dtype`` (what a gradient exchange sends), or None
        self.wire_dtype = wire_dtype   # torch.bfloat16: backward passes also produce the bf16 copy
        # the fused layer then writes ONLY the bf16 rows (they become the entry's rows): for data-parallel steps whose
        # mean gradient is formed from the ranks' bf16 rows anyway, the local fp32 rows would be written for nobody
        self.wire_only = bool(wire_only and wire_dtype == torch.bfloat16)
        self.scale = 1.0    # factor the consumer applies to the summed rows (1 / world after a zero-copy reduction)

    def add(self, uniq, num_unique, rows, tokens_per_chapter, wire=None):
        self.entries.append((uniq, num_unique, rows, int(tokens_per_chapter)))
        self.wire.append(wire)

    def clear(self):
        self.entries.clear()
        self.wire.clear()

    def to_dense(self, like: torch.Tensor) -> torch.Tensor:
        dense = torch.zeros(like.shape, dtype=torch.float32, device=like.device)
        for uniq, num_unique, rows, t in self.entries:
            ops.scatter_bank_grad(rows if rows.dtype == torch.float32 else rows.float(),
                                  {"uniq": uniq, "num_unique": num_unique}, t, dense)
        if self.scale != 1.0:
            dense.mul_(self.scale)
        return dense


_side_streams: Dict[tuple, "torch.cuda.Stream"] = {}
_side_handles: Dict[tuple, int] = {}


def _side_stream(dev_index: int, main_handle: int) -> int:
    """Second stream of the layer, with the priority of the stream it runs beside (a step captured on a
    high-priority stream keeps both of its streams ahead of background work such as a gradient exchange).
    ``main_handle`` is the raw handle of the current stream; so is the result."""
    handle = _side_handles.get((dev_index, main_handle))
    if handle is None:
        device = torch.device("cuda", dev_index)
        key = (dev_index, torch.cuda.current_stream(device).priority)
        if key not in _side_streams:
            _side_streams[key] = torch.cuda.Stream(device=device, priority=key[1])
        handle = _side_handles[(dev_index, main_handle)] = _side_streams[key].cuda_stream
    return handle


# --------------------------------------------------------------------------------------------
# router
# --------------------------------------------------------------------------------------------
class _Route(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h, weight, bias, top_k, num_shared, routed_scale, with_losses, pos_weight):
        ctx.set_materialize_grads(False)
        if h.dim() != 3:
            raise ValueError(f"hidden_states must be 3D (B, T, D), got shape {tuple(h.shape)}")
        _check_width("router weight", weight, h.shape[2])
        _check_numel("router bias", bias, weight.shape[0])
        _check_numel("pos_weight", pos_weight, h.shape[1])
        L.require_cuda(h, weight, bias, pos_weight)
        dev, f32 = h.device, torch.float32
        hc, w = ops._contig(h), ops._contig(weight.float())
        bc = None if bias is None else ops._contig(bias.float())
        pw = None if pos_weight is None else ops._contig(pos_weight.float())
        b, l, d = h.shape
        c = w.shape[0]
        k = ops.router_selected_k(c, top_k, num_shared)
        idx = torch.empty(b, k, dtype=torch.int64, device=dev)
        weights = torch.empty(b, k, dtype=f32, device=dev)
        comb_idx = torch.empty(b, num_shared + k, dtype=torch.int32, device=dev)
        comb_w = torch.empty(b, num_shared + k, dtype=f32, device=dev)
        losses = torch.empty(4, dtype=f32, device=dev) if with_losses else None
        p = L.ptr
        s = L.RouteDesc(L.RouterShape(b, l, d, c, top_k, num_shared, routed_scale, L.dtype_code(h.dtype)), p(hc), p(w), p(bc),
                        p(pw), p(idx), p(weights), p(comb_idx), p(comb_w), p(losses), None, p(L.status_word(dev)),
                        L.stream_ptr(dev))
        arena = torch.empty(ops.route_arena_bytes(s), dtype=torch.uint8, device=dev)
        s.arena = p(arena)
        ops.route_fwd(s)
        if any(ctx.needs_input_grad[:3]):
            ctx.desc = s
            ctx.meta = (tuple(h.shape), h.dtype, weight.dtype, None if bias is None else bias.dtype)
            # Output tensors go through save_for_backward (autograd handles a node's own outputs there without a
            # reference cycle), so the node and its buffers are released by reference counting as soon as the graph is.
            ctx.save_for_backward(w, arena, idx, weights, comb_w, pw)
        ctx.mark_non_differentiable(idx, comb_idx)
        return idx, weights, comb_idx, comb_w, losses if with_losses else torch.zeros(4, dtype=f32, device=dev)

    @staticmethod
    def backward(ctx, _g_idx, g_w, _g_cidx, g_cw, g_losses):
        w, arena, idx, weights, comb_w, pw = ctx.saved_tensors
        s, p = ctx.desc, L.ptr
        h_shape, h_dtype, w_dtype, b_dtype = ctx.meta
        need, dev, f32 = ctx.needs_input_grad, w.device, torch.float32
        s.w, s.arena, s.idx, s.weights, s.comb_w, s.pos_weight = p(w), p(arena), p(idx), p(weights), p(comb_w), p(pw)
        s.stream = L.stream_ptr(dev)
        g_w, g_cw, g_losses = (None if g is None else ops._contig(g.float()) for g in (g_w, g_cw, g_losses))
        d_h = torch.empty(h_shape, dtype=h_dtype, device=dev) if need[0] else None
        want_b = b_dtype is not None and need[2]
        d_w = torch.empty(w.shape, dtype=f32, device=dev) if (need[1] or want_b) else None
        d_b = torch.empty(w.shape[0], dtype=f32, device=dev) if want_b else None
        scratch = torch.empty(ops.route_bwd_scratch_bytes(s), dtype=torch.uint8, device=dev)
        ops.route_bwd(s, g_w, g_cw, g_losses, d_h, d_w, d_b, scratch)
        return d_h, _cast(d_w, w_dtype) if need[1] else None, d_b, None, None, None, None, None


def route(h: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], top_k: int, num_shared: int,
          routed_scale: float = 1.0, with_losses: bool = True, pos_weight: Optional[torch.Tensor] = None):
    """Returns (idx int64 [B,k'], weights [B,k'], comb_idx int32 [B,S+k'], comb_w [B,S+k'], losses dict).
    ``pos_weight`` [L]: pool with these per-position coefficients instead of the plain mean (the
    sequence-rolling rule, see :func:`ops.rolling_pool_coefficients`)."""
    idx, w, cidx, cw, lv = _Route.apply(h, weight, bias, int(top_k), int(num_shared), float(routed_scale),
                                        bool(with_losses), pos_weight)
    return idx, w, cidx, cw, _LossDict(lv) if with_losses else {}


# --------------------------------------------------------------------------------------------
# gather
# --------------------------------------------------------------------------------------------
class _GatherChapters(torch.autograd.Function):
    @staticmethod
    def forward(ctx, bank, comb_idx, comb_w, tokens_per_chapter, norm_type, eps, out_dtype, sink):
        out, stats = ops.gather_rows_fwd(bank, tokens_per_chapter, comb_idx, comb_w, norm_type, eps, out_dtype)
        ctx.cfg = (int(tokens_per_chapter), norm_type, float(eps))
        ctx.sink = sink
        ctx.save_for_backward(bank, comb_idx, comb_w, stats)
        return out

    @staticmethod
    def backward(ctx, g):
        bank, comb_idx, comb_w, stats = ctx.saved_tensors
        t, norm, eps = ctx.cfg
        want_dw = comb_w is not None and ctx.needs_input_grad[2]
        want_bank = ctx.needs_input_grad[0]
        d_cw, rows, wire, dense, uniq, count = ops.gather_rows_bwd_lists(
            g, bank, t, comb_idx, comb_w, norm, eps, stats, want_dw, want_bank,
            dense=ctx.sink is None, wire=ctx.sink is not None and ctx.sink.wire_dtype == torch.bfloat16)
        if want_bank and ctx.sink is not None:
            ctx.sink.add(uniq, count, rows, t, wire=wire)
        d_bank = _cast(dense, bank.dtype)
        return d_bank, None, d_cw, None, None, None, None, None


def gather_chapters(bank: torch.Tensor, comb_idx: torch.Tensor, comb_w: Optional[torch.Tensor],
                    tokens_per_chapter: int, norm_type: Optional[str] = None, eps: float = 1e-5,
                    out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """[B, K*T, d] rows of the selected chapters, normalised and scaled by ``comb_w``."""
    sink = getattr(bank, "moc_sparse_grad", None)
    return _GatherChapters.apply(bank, comb_idx.to(torch.int32), comb_w, int(tokens_per_chapter), norm_type,
                                 float(eps), out_dtype or bank.dtype, sink)


# --------------------------------------------------------------------------------------------
# cross attention over gathered rows
# --------------------------------------------------------------------------------------------
class _CrossAttention(torch.autograd.Function):
    """One native call per pass (``moc_xattn_fwd`` / ``moc_xattn_bwd``)."""

    @staticmethod
    def forward(ctx, h, memory, wq, wk, wv, wo, norm_w, norm_b, num_heads, num_kv_heads, compute_dtype,
                norm_kind, norm_eps, add_residual, grad_on):
        b, l, d = h.shape
        cd = compute_dtype
        dev = h.device
        mem_shared = memory.dim() == 2
        in_dtype, mem_dtype, mem_shape = h.dtype, memory.dtype, memory.shape
        if not mem_shared and (memory.dim() < 3 or mem_shape[:-2].numel() != b):
            raise ValueError("memory must be (N, d) or (B, N, d) with the batch size of the hidden states")
        _check_projections(d, mem_shape[-1], wq, wk, wv, wo, num_heads, num_kv_heads)
        attn_dim, out_dim = wq.shape[0], wo.shape[0]
        if add_residual and out_dim != d:
            raise ValueError(f"the residual has {d} columns, the result {out_dim}")
        _check_numel("norm_weight", norm_w, d)
        _check_numel("norm_bias", norm_b, d)
        L.require_cuda(h, memory, wq, wk, wv, wo, norm_w, norm_b)
        # the kernels take fp32 or bf16; anything else goes through the compute dtype
        hc = ops._contig(h if in_dtype in _KERNEL_DTYPES else h.to(cd))
        mc = ops._contig(memory if mem_dtype in _KERNEL_DTYPES else memory.to(cd))
        w_dtypes = (wq.dtype, wk.dtype, wv.dtype, wo.dtype)
        same = len(set(w_dtypes)) == 1 and wq.dtype in _KERNEL_DTYPES
        ws = [ops._contig(w if same else w.float()) for w in (wq, wk, wv, wo)]
        nw = None if norm_w is None else ops._contig(norm_w.float())
        nb = None if norm_b is None else ops._contig(norm_b.float())
        need_grad = grad_on and any(ctx.needs_input_grad[:8])
        out = torch.empty(b, l, out_dim, dtype=in_dtype if in_dtype in (torch.float32, cd) else cd, device=dev)
        if cd == torch.float32 and out.dtype != cd:
            out = torch.empty(b, l, out_dim, dtype=cd, device=dev)
        main = L.stream_ptr(dev)
        code, p = L.dtype_code, L.ptr
        s = L.XattnDesc(b, l, mc.shape[-2], d, mc.shape[-1], num_heads, num_kv_heads, int(mem_shared), code(hc.dtype),
                        code(mc.dtype), code(ws[0].dtype), code(cd), code(out.dtype),
                        ops.NORM_KINDS[norm_kind] if norm_kind is not None else 0, int(add_residual), int(need_grad),
                        norm_eps, p(hc), p(mc), p(ws[0]), p(ws[1]), p(ws[2]), p(ws[3]), p(nw), p(nb), p(out), None,
                        p(L.status_word(dev)), main, _side_stream(L.device_index(dev), main), attn_dim, out_dim)
        arena = torch.empty(ops.xattn_arena_bytes(s), dtype=torch.uint8, device=dev)
        s.arena = p(arena)
        ops.xattn_fwd(s)
        if need_grad:
            ctx.desc = s
            ctx.dtypes = (in_dtype, mem_dtype, w_dtypes, None if norm_w is None else norm_w.dtype,
                          None if norm_b is None else norm_b.dtype, wk.shape[0], mem_shape)
            # inputs the backward pass reads itself: as projection operands, or for the normalisation
            keep_h = hc if (norm_kind is not None or hc.dtype == cd) else None
            keep_m = mc if mc.dtype == cd else None
            keep_w = (ws[0], ws[3]) if (cd == torch.float32 and ws[0].dtype == cd) else (None, None)
            ctx.save_for_backward(arena, keep_h, keep_m, *keep_w, nw)
        return _cast(out, in_dtype)

    @staticmethod
    def backward(ctx, g):
        arena, hc, mc, wq, wo, nw = ctx.saved_tensors
        s = ctx.desc
        in_dtype, mem_dtype, wdt, nw_dtype, nb_dtype, dkv, mem_shape = ctx.dtypes
        dev, f32, p = arena.device, torch.float32, L.ptr
        need = ctx.needs_input_grad
        cd = f32 if s.compute_dtype == L.MOC_F32 else torch.bfloat16
        s.arena, s.h, s.memory, s.wq, s.wo, s.norm_w = p(arena), p(hc), p(mc), p(wq), p(wo), p(nw)
        s.stream = L.stream_ptr(dev)
        s.side_stream = _side_stream(L.device_index(dev), s.stream)
        g = ops._contig(g if g.dtype in _KERNEL_DTYPES else g.to(cd))
        b, l, d, md = s.batch, s.seq, s.hidden_dim, s.mem_dim
        dh_dtype = in_dtype if in_dtype in (f32, cd) else cd
        dm_dtype = mem_dtype if mem_dtype in (f32, cd) else cd
        if nw is not None and cd == torch.bfloat16 and in_dtype not in _KERNEL_DTYPES:
            dh_dtype = f32
        d_h = torch.empty(b, l, d, dtype=dh_dtype if cd != f32 else f32, device=dev) if (need[0] or nw is not None) else None
        d_mem = torch.empty(mem_shape, dtype=dm_dtype if cd != f32 else f32, device=dev) if need[1] else None
        d_wq = torch.empty(s.attn_dim, d, dtype=f32, device=dev)
        d_wkv = torch.empty(2 * dkv, md, dtype=f32, device=dev)
        d_wo = torch.empty(s.out_dim, s.attn_dim, dtype=f32, device=dev)
        d_nw = torch.empty(d, dtype=f32, device=dev) if nw is not None else None
        d_nb = torch.empty(d, dtype=f32, device=dev) if nb_dtype is not None else None
        q = L.XattnBwdDesc(p(g), L.dtype_code(g.dtype), L.dtype_code(d_h.dtype) if d_h is not None else 0,
                           L.dtype_code(d_mem.dtype) if d_mem is not None else 0, p(d_h), p(d_mem), p(d_wq), p(d_wkv),
                           p(d_wo), p(d_nw), p(d_nb), None)
        scratch = torch.empty(ops.xattn_bwd_scratch_bytes(s, q), dtype=torch.uint8, device=dev)
        q.scratch = p(scratch)
        ops.xattn_bwd(s, q)
        return (_cast(d_h, in_dtype) if need[0] else None, _cast(d_mem, mem_dtype), _cast(d_wq, wdt[0]),
                _cast(d_wkv[:dkv], wdt[1]), _cast(d_wkv[dkv:], wdt[2]), _cast(d_wo, wdt[3]), _cast(d_nw, nw_dtype),
                _cast(d_nb, nb_dtype), None, None, None, None, None, None, None)


def cross_attention(h: torch.Tensor, memory: torch.Tensor, wq, wk, wv, wo, num_heads: int,
                    num_kv_heads: Optional[int] = None, compute_dtype: Optional[torch.dtype] = None, *,
                    pre_norm: Optional[str] = None, norm_weight: Optional[torch.Tensor] = None,
                    norm_bias: Optional[torch.Tensor] = None, norm_eps: float = 1e-6,
                    add_residual: bool = False) -> torch.Tensor:
    """softmax(Q K^T / sqrt(D)) V over the given memory rows, with the four projections.

    ``pre_norm`` ("rms" or "layernorm") normalises ``h`` first and ``add_residual`` adds ``h`` to the result:
    together they are the memory sub-block of the reference's transformer block, h + attn(norm(h), memory)
    (memory_block.py:549-558), with the normalisation fused into the query projection's operand and the
    residual add into the output projection's epilogue.
    """
    if pre_norm is not None:
        if pre_norm not in ops.NORM_KINDS:
            raise ValueError(f"unknown pre_norm {pre_norm!r}")
        if norm_weight is None:
            raise ValueError("pre_norm needs norm_weight")
        if pre_norm in ("rms", "rmsnorm"):
            norm_bias = None
    return _CrossAttention.apply(h, memory, wq, wk, wv, wo, norm_weight if pre_norm else None,
                                 norm_bias if pre_norm else None, int(num_heads), int(num_kv_heads or num_heads),
                                 compute_dtype or h.dtype, pre_norm, float(norm_eps), bool(add_residual),
                                 torch.is_grad_enabled())


# --------------------------------------------------------------------------------------------
# the whole layer as one node with two streams (bf16 path)
# --------------------------------------------------------------------------------------------
# The dQ kernel runs on the side stream beside the dK/dV kernel (fused route): 768 CTAs over 296 slots leave the last
# of dQ's three rounds 59 % full, and the other kernel's CTAs take the free slots (measured 1.189 -> 1.177 ms per
# step).  MOC_DQ_ON_SIDE_STREAM=0 puts both back on the main stream.
_DQ_ON_SIDE_STREAM = os.environ.get("MOC_DQ_ON_SIDE_STREAM", "1") != "0"


class _MemoryLayerTwoStream(torch.autograd.Function):
    """Router, gather, projections and attention of one layer as a single autograd node of one native call per pass
    (``moc_layer_fwd`` / ``moc_layer_bwd``): the bandwidth- and latency-bound kernels (router, chapter bookkeeping,
    gather backward) run on a second stream beside the tensor-core kernels, and the host pays one call instead of one
    per kernel.

      forward   side: router, chapter segments      | main: weight pack, (norm,) query projection
                join, then gather, K/V projection, attention, output projection on main
      backward  main: dO projection, attention backward, memory-row gradient, bank / chapter-weight
                gradients, router backward           | side: the four weight-gradient and the hidden-state
                                                       projections, normalisation backward

    Both streams fork from and join the caller's stream with events, which a CUDA-graph capture records as
    ordinary dependencies.  Every buffer is allocated on the caller's stream, behind which the side stream is joined
    before the call returns.
    """

    @staticmethod
    def forward(ctx, h_router, h_attn, bank, router_w, router_b, wq, wk, wv, wo, norm_w, norm_b, cfg, sink,
                fused=None):
        ctx.set_materialize_grads(False)       # an output nobody used has no gradient: no zeros to fill and add
        (num_heads, num_kv_heads, t, top_k, num_shared, routed_scale, row_norm, row_eps, with_losses,
         pre_norm, pre_eps, add_residual, grad_on) = cfg
        if h_router.dim() != 3:
            raise ValueError(f"hidden_states must be 3D (B, T, D), got shape {tuple(h_router.shape)}")
        dev = h_attn.device
        b, l, d = h_attn.shape
        rows, c = bank.shape[0], router_w.shape[0]
        if h_router.shape[0] != b:
            raise ValueError(f"h_router and h_attn must share the batch: {h_router.shape[0]} vs {b}")
        # (the router may look at states of another width than the attention's)
        _check_width("router_weight", router_w, h_router.shape[2])
        _check_numel("router_bias", router_b, c)
        _check_numel("pre_norm_weight", norm_w, d)
        _check_numel("pre_norm_bias", norm_b, d)
        L.require_cuda(h_router, h_attn, bank, router_w, router_b, wq, wk, wv, wo, norm_w, norm_b)
        # the kernels take fp32 or bf16 activations; anything else computes in bf16 and is cast back
        in_dtype = h_attn.dtype
        ha = ops._contig(h_attn if in_dtype in (torch.float32, torch.bfloat16) else h_attn.to(torch.bfloat16))
        hr = ha if h_router is h_attn else ops._contig(h_router)
        k_sel = ops.router_selected_k(c, top_k, num_shared)
        # the reference only normalises when both a shared and a routed slice exist (model.py:413-418)
        norm = row_norm if (num_shared > 0 and k_sel > 0) else None
        if fused is not None and (norm not in (None, "rms") or (norm == "rms" and fused.get("inv_rms") is None)):
            fused = None                      # affine-free LayerNorm rows are not a row scale: two-pass route
        shadow = None if fused is None else ops._contig(fused["shadow"])
        if shadow is not None and (shadow.dtype != torch.bfloat16 or shadow.shape != bank.shape):
            raise TypeError("bank_shadow must be a bf16 tensor shaped like the bank")
        inv_rms = ops._contig(fused["inv_rms"].float()) if (fused is not None and norm == "rms") else None
        _check_numel("bank_inv_rms", inv_rms, rows)
        L.require_cuda(shadow, inv_rms)
        bank_c = ops._contig(bank)
        rw = ops._contig(router_w.float())
        rb = None if router_b is None else ops._contig(router_b.float())
        ws = [ops._contig(w) for w in (wq, wk, wv, wo)]
        nw = None if norm_w is None else ops._contig(norm_w.float())
        nb = None if norm_b is None else ops._contig(norm_b.float())
        # (a node's forward always runs with gradients off; needs_input_grad says nothing about the caller's mode)
        need_grad = grad_on and any(ctx.needs_input_grad[:11])
        n_pairs = b * (num_shared + k_sel)
        f32, i32 = torch.float32, torch.int32
        out = torch.empty(b, l, d, dtype=ha.dtype, device=dev)
        idx = torch.empty(b, k_sel, dtype=torch.int64, device=dev)
        weights = torch.empty(b, k_sel, dtype=f32, device=dev)
        comb_idx = torch.empty(b, num_shared + k_sel, dtype=i32, device=dev)
        comb_w = torch.empty(b, num_shared + k_sel, dtype=f32, device=dev)
        losses = torch.empty(4, dtype=f32, device=dev) if with_losses else torch.zeros(4, dtype=f32, device=dev)
        touched = torch.empty(n_pairs + 1, dtype=i32, device=dev) if need_grad else None    # ids, then their count
        index = L.device_index(dev)
        main = L.stream_ptr(dev)
        s = L.LayerDesc(
            b, l, hr.shape[1], d, num_heads, num_kv_heads, c, t, top_k, num_shared, L.dtype_code(hr.dtype),
            L.dtype_code(ha.dtype), L.dtype_code(bank.dtype), L.dtype_code(wq.dtype), L.NORM_CODES[norm],
            ops.NORM_KINDS[pre_norm] if pre_norm is not None else 0, int(add_residual), int(with_losses),
            int(fused is not None), int(need_grad), routed_scale, row_eps, pre_eps, rows, hr.data_ptr(), ha.data_ptr(),
            bank_c.data_ptr(), L.ptr(shadow), L.ptr(inv_rms), rw.data_ptr(), L.ptr(rb), ws[0].data_ptr(),
            ws[1].data_ptr(), ws[2].data_ptr(), ws[3].data_ptr(), L.ptr(nw), L.ptr(nb), out.data_ptr(), idx.data_ptr(),
            weights.data_ptr(), comb_idx.data_ptr(), comb_w.data_ptr(), losses.data_ptr(), L.ptr(touched),
            None if touched is None else touched.data_ptr() + 4 * n_pairs, None, L.status_word(dev).data_ptr(), main,
            _side_stream(index, main), hr.shape[2])
        arena = torch.empty(ops.layer_arena_bytes(s), dtype=torch.uint8, device=dev)
        s.arena = arena.data_ptr()
        ops.layer_fwd(s)

        ctx.desc, ctx.sink = s, sink
        ctx.same_h = h_router is h_attn
        ctx.wkv_in_place = bool(fused is not None and fused.get("wkv_grad_in_place"))
        ctx.shapes = (tuple(h_router.shape), h_router.dtype, in_dtype, router_b is not None,
                      (wq.dtype, wk.dtype, wv.dtype, wo.dtype), None if norm_w is None else norm_w.dtype,
                      None if norm_b is None else norm_b.dtype, wk.shape[0])
        if need_grad:
            # outputs of this node (weights, combined lists) go through save_for_backward: kept as attributes they
            # would tie the node to its own outputs in a reference cycle.  The attention input is saved where the
            # backward pass reads it itself: as the bf16 projection operand, or for the normalisation.
            keep_h = ha if (pre_norm is not None or ha.dtype == torch.bfloat16) else None
            ctx.save_for_backward(arena, touched, keep_h, bank_c, shadow, inv_rms, rw, nw, idx, weights, comb_idx, comb_w)
        ctx.mark_non_differentiable(idx, comb_idx)
        return out if in_dtype == out.dtype else out.to(in_dtype), idx, weights, comb_idx, comb_w, losses

    @staticmethod
    def backward(ctx, g, _g_idx, g_w, _g_cidx, g_cw, g_losses):
        arena, touched, ha, bank, shadow, inv_rms, rw, nw, idx, weights, comb_idx, comb_w = ctx.saved_tensors
        s, sink = ctx.desc, ctx.sink
        hr_shape, hr_dtype, in_dtype, has_rbias, wdt, nw_dtype, nb_dtype, dkv = ctx.shapes
        t = s.tokens_per_chapter
        need = ctx.needs_input_grad
        dev = arena.device
        f32 = torch.float32
        b, l, d = s.batch, s.seq, s.hidden_dim
        n_pairs = touched.numel() - 1
        attn_dtype = f32 if s.attn_dtype == L.MOC_F32 else torch.bfloat16
        # saved tensors may have been moved (hooks): take their addresses again
        p = L.ptr
        s.arena, s.uniq, s.num_unique = p(arena), p(touched), p(touched) + 4 * n_pairs
        s.h_attn, s.bank, s.bank_shadow, s.bank_inv_rms, s.router_w, s.norm_w = p(ha), p(bank), p(shadow), p(inv_rms), p(rw), p(nw)
        s.idx, s.weights, s.comb_idx, s.comb_w = p(idx), p(weights), p(comb_idx), p(comb_w)
        s.stream = L.stream_ptr(dev)
        s.side_stream = _side_stream(L.device_index(dev), s.stream)

        g = torch.zeros(b, l, d, dtype=attn_dtype, device=dev) if g is None else ops._contig(g.to(attn_dtype))
        as_f32 = lambda v: None if v is None else ops._contig(v.float())     # noqa: E731
        g_w, g_cw, g_losses = as_f32(g_w), as_f32(g_cw), as_f32(g_losses)
        fuse_dh = ctx.same_h and need[0] and hr_dtype == in_dtype and in_dtype == attn_dtype
        d_ha = torch.empty(b, l, d, dtype=attn_dtype, device=dev)
        r_dtype = f32 if s.router_dtype == L.MOC_F32 else torch.bfloat16      # what the router's kernels write
        d_hr = None if fuse_dh or not need[0] else torch.empty(hr_shape, dtype=r_dtype, device=dev)
        rows = wire = dense = None
        if need[2]:
            n_rows = n_pairs * t
            if sink is None:
                dense = torch.empty(bank.shape, dtype=f32, device=dev)
            else:
                wire_only = sink.wire_only and s.fused and d % 8 == 0 and d <= 1024
                if not wire_only:
                    rows = torch.empty(n_rows, d, dtype=f32, device=dev)
                if sink.wire_dtype == torch.bfloat16:
                    wire = torch.empty(n_rows, d, dtype=torch.bfloat16, device=dev)
        d_rw = torch.empty(rw.shape, dtype=f32, device=dev) if (need[3] or need[4]) else None
        d_rb = torch.empty(rw.shape[0], dtype=f32, device=dev) if (has_rbias and need[4]) else None
        d_wq = torch.empty(d, d, dtype=f32, device=dev)
        d_wkv = torch.empty(2 * dkv, d, dtype=f32, device=dev)
        d_wo = torch.empty(d, d, dtype=f32, device=dev)
        d_nw = torch.empty(d, dtype=f32, device=dev) if nw is not None else None
        d_nb = torch.empty(d, dtype=f32, device=dev) if nb_dtype is not None else None
        q = L.LayerBwdDesc(p(g), p(g_w), p(g_cw), p(g_losses), int(need[0]), int(_DQ_ON_SIDE_STREAM), int(ctx.wkv_in_place),
                           int(d_rw is not None), p(d_ha), p(d_hr), p(rows), p(wire), p(dense), p(d_rw), p(d_rb), p(d_wq),
                           p(d_wkv), p(d_wo), p(d_nw), p(d_nb), None)
        scratch = torch.empty(ops.layer_bwd_scratch_bytes(s, q), dtype=torch.uint8, device=dev)
        q.scratch = scratch.data_ptr()
        ops.layer_bwd(s, q)
        if rows is not None or wire is not None:
            sink.add(touched[:n_pairs], touched[n_pairs:], wire if rows is None else rows, t, wire=wire)

        d_ha, d_hr = _cast(d_ha, in_dtype), _cast(d_hr, hr_dtype)
        if fuse_dh:
            d_hr, d_ha = d_ha, None
        return (d_hr, d_ha, _cast(dense, bank.dtype), _cast(d_rw, rw.dtype) if need[3] else None, d_rb, _cast(d_wq, wdt[0]),
                _cast(d_wkv[:dkv], wdt[1]), _cast(d_wkv[dkv:], wdt[2]), _cast(d_wo, wdt[3]),
                _cast(d_nw, nw_dtype), _cast(d_nb, nb_dtype), None, None, None)


# --------------------------------------------------------------------------------------------
# the fused layer
# --------------------------------------------------------------------------------------------
def memory_layer(h_router: torch.Tensor, h_attn: torch.Tensor, bank: torch.Tensor,
                 router_weight: torch.Tensor, router_bias: Optional[torch.Tensor],
                 wq, wk, wv, wo, *, num_heads: int, num_kv_heads: Optional[int], tokens_per_chapter: int,
                 top_k: int, num_shared_chapters: int = 1, routed_scaling_factor: float = 2.5,
                 norm_type: Optional[str] = None, norm_eps: float = 1e-5, with_losses: bool = True,
                 compute_dtype: Optional[torch.dtype] = None, pre_norm: Optional[str] = None,
                 pre_norm_weight: Optional[torch.Tensor] = None, pre_norm_bias: Optional[torch.Tensor] = None,
                 pre_norm_eps: float = 1e-6, add_residual: bool = False,
                 two_stream: bool = True, bank_shadow: Optional[torch.Tensor] = None,
                 bank_inv_rms: Optional[torch.Tensor] = None,
                 wkv_grad_in_place: bool = False) -> Tuple[torch.Tensor, Dict[str, torch.Tensor], Dict]:
    """Sequence-level Mixture-of-Chapters memory layer on the GPU.

    Returns (out [B,L,d], router losses, info) with info = indices / weights of the routing.
    ``norm_type`` normalises the gathered bank rows; ``pre_norm`` / ``add_residual`` wrap the attention as
    h_attn + attn(pre_norm(h_attn), memory) (see :func:`cross_attention`).  With bf16 compute the layer runs as
    one autograd node that overlaps its small kernels with the tensor-core kernels on a second stream
    (``two_stream=False`` chains the three separate nodes instead; results are the same).

    ``bank_shadow`` (bf16 copy of ``bank``, e.g. ``ChapteredMemoryBank.bf16_shadow()`` or the copy
    ``SparseBankAdamW`` refreshes) switches the bf16 layer to the fused gather-and-project route: the K/V projection
    reads the selected chapters straight from that copy and no gathered rows are materialised, forward or
    backward.  With ``norm_type="rms"`` it also needs ``bank_inv_rms`` (``ops.row_inv_rms`` of the bank with
    ``norm_eps``); ``norm_type="layernorm"`` keeps the two-pass route.  ``wkv_grad_in_place`` lets the Wk / Wv
    gradient read the bank through a gather list as well instead of copying the raw selected rows out on the side
    stream first (no gathered copy at all, but slower at the paper shape).
    """
    cd, d = compute_dtype or h_attn.dtype, h_attn.shape[-1]
    _check_projections(d, bank.shape[1], wq, wk, wv, wo, int(num_heads), int(num_kv_heads or num_heads))
    if (cd == torch.bfloat16 and two_stream and wq.dtype == wk.dtype == wv.dtype == wo.dtype
            and bank.shape[1] == wq.shape[0] == wo.shape[0] == d):
        cfg = (int(num_heads), int(num_kv_heads or num_heads), int(tokens_per_chapter), int(top_k),
               int(num_shared_chapters), float(routed_scaling_factor), norm_type, float(norm_eps), bool(with_losses),
               pre_norm, float(pre_norm_eps), bool(add_residual), torch.is_grad_enabled())
        if pre_norm is not None and pre_norm not in ops.NORM_KINDS:
            raise ValueError(f"unknown pre_norm {pre_norm!r}")
        if pre_norm in ("rms", "rmsnorm"):
            pre_norm_bias = None
        out, idx, w, cidx, cw, lv = _MemoryLayerTwoStream.apply(
            h_router, h_attn, bank, router_weight, router_bias, wq, wk, wv, wo,
            pre_norm_weight if pre_norm else None, pre_norm_bias if pre_norm else None, cfg,
            getattr(bank, "moc_sparse_grad", None),
            None if bank_shadow is None else {"shadow": bank_shadow, "inv_rms": bank_inv_rms,
                                              "wkv_grad_in_place": wkv_grad_in_place})
        losses = _LossDict(lv) if with_losses else {}
        return out, losses, {"indices": idx, "weights": w, "combined_indices": cidx, "combined_weights": cw}
    idx, w, cidx, cw, losses = route(h_router, router_weight, router_bias, top_k, num_shared_chapters,
                                     routed_scaling_factor, with_losses)
    k_sel = idx.shape[1]
    # the reference only normalises when both a shared and a routed slice exist (model.py:413-418)
    norm = norm_type if (num_shared_chapters > 0 and k_sel > 0) else None
    memory = gather_chapters(bank, cidx, cw, tokens_per_chapter, norm, norm_eps, out_dtype=cd)
    out = cross_attention(h_attn, memory, wq, wk, wv, wo, num_heads, num_kv_heads, cd, pre_norm=pre_norm,
                          norm_weight=pre_norm_weight, norm_bias=pre_norm_bias, norm_eps=pre_norm_eps,
                          add_residual=add_residual)
    return out, losses, {"indices": idx, "weights": w, "combined_indices": cidx, "combined_weights": cw}


# --------------------------------------------------------------------------------------------
# token-level routing (every token selects its own chapters)
# --------------------------------------------------------------------------------------------
def _weight_grad_splits(cd, rows: int, out_rows: int, out_cols: int) -> int:
    """K-splits of a weight-gradient projection dW[out_rows, out_cols] = dY^T X over ``rows``: enough (tile, split)
    items to fill the SMs once (tensor-core kernel only; the splits add into a zeroed fp32 output)."""
    if cd != torch.bfloat16:
        return 1
    tiles = -(-out_rows // 128) * -(-out_cols // 256)
    return max(1, min(148 // max(tiles, 1), rows // 512))


# rows * chapters * hidden above which a bf16 model's token router projects on the tensor cores (split fp32 weight)
_SPLIT_ROUTER_MIN_WORK = 1 << 27


class _RouteTokens(torch.autograd.Function):
    """ChapterRouter.route_token_level (router.py:262-340): logits of every token by an fp32 projection, then the
    same softmax / prefix mask / top-k / renormalisation / loss kernels as the sequence router with one routing
    row per token."""

    @staticmethod
    def forward(ctx, h, weight, bias, top_k, num_shared, with_losses):
        ctx.set_materialize_grads(False)
        b, l, d = h.shape
        _check_width("router weight", weight, d)
        _check_numel("router bias", bias, weight.shape[0])
        L.require_cuda(h, weight, bias)
        rows = b * l
        h2 = h.reshape(rows, d).contiguous()
        w32 = weight.float().contiguous()
        c = w32.shape[0]
        ctx.cfg = ((b, l, d), h.dtype, int(top_k), int(num_shared), bias is not None)
        ctx.desc = None
        if h.dtype == torch.bfloat16 and d % 8 == 0 and rows * c * d >= _SPLIT_ROUTER_MIN_WORK:
            desc, idx, weights, losses, arena = ops.token_route_fwd(h2, w32, None if bias is None else bias.float(), top_k,
                                                                    num_shared, with_losses)
            if any(ctx.needs_input_grad[:3]):
                ctx.desc = desc
                ctx.save_for_backward(h2, arena, idx, weights)
            idx = idx.view(b, l, -1)
            ctx.mark_non_differentiable(idx)
            return (idx, weights.view(b, l, -1),
                    losses if with_losses else torch.zeros(4, dtype=torch.float32, device=h.device))
        h32 = ops.cast(h2, torch.float32)
        logits = ops.gemm(h32, w32, tag="token_router_logits")                 # [rows, C] fp32, no bias yet
        r = ops.router_fwd(h32.view(rows, 1, d), w32, bias, top_k, num_shared, 1.0, with_losses, pooled=h32, logits=logits)
        k = r["idx"].shape[1]
        ctx.internals = {n: r[n] for n in ("pooled", "probs", "idx", "row_stats", "chapter_stats", "_ws", "comb_w")}
        ctx.save_for_backward(w32, r["weights"])
        idx = r["idx"].view(b, l, k)
        ctx.mark_non_differentiable(idx)
        losses = r["losses"] if with_losses else torch.zeros(4, dtype=torch.float32, device=h.device)
        return idx, r["weights"].view(b, l, k), losses

    @staticmethod
    def backward(ctx, _g_idx, g_w, g_losses):
        (b, l, d), h_dtype, top_k, num_shared, has_bias = ctx.cfg
        rows = b * l
        if ctx.desc is not None:
            h2, arena, idx, weights = ctx.saved_tensors
            d_h, d_w, d_b = ops.token_route_bwd(ctx.desc, h2, arena, idx, weights,
                                                None if g_w is None else g_w.reshape(rows, -1).float().contiguous(),
                                                None if g_losses is None else g_losses.float().contiguous(),
                                                ctx.needs_input_grad[0], ctx.needs_input_grad[1],
                                                has_bias and ctx.needs_input_grad[2])
            return None if d_h is None else d_h.view(b, l, d), d_w, d_b, None, None, None
        w32, weights = ctx.saved_tensors
        saved = dict(ctx.internals, weights=weights)
        g_w = None if g_w is None else g_w.reshape(rows, -1).float().contiguous()
        g_losses = None if g_losses is None else g_losses.float()
        r = ops.router_bwd((rows, 1, d), torch.float32, w32, saved, top_k, num_shared, 1.0, g_w, None, g_losses,
                           want_dh=False, parts=1, logits_only=True)
        d_logits = r["d_logits"]
        h32 = saved["pooled"]
        d_h = d_w = d_b = None
        if ctx.needs_input_grad[0]:
            d_h = ops.gemm(d_logits, w32, b_kmajor=False, tag="token_router_dh").view(b, l, d).to(h_dtype)
        if ctx.needs_input_grad[1]:
            d_w = ops.gemm(d_logits, h32, a_kmajor=False, b_kmajor=False, tag="token_router_dw")
        if has_bias and ctx.needs_input_grad[2]:
            d_b = ops.col_sum(d_logits)
        return d_h, d_w, d_b, None, None, None


def route_tokens(h: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], top_k: int, num_shared: int,
                 with_losses: bool = True):
    """Returns (global chapter ids int64 [B,L,k'], weights [B,L,k'], losses dict); k' = min(k, C - num_shared)."""
    idx, w, lv = _RouteTokens.apply(h, weight, bias, int(top_k), int(num_shared), bool(with_losses))
    return idx, w, _LossDict(lv) if with_losses else {}


class _TokenRoutedAttention(torch.autograd.Function):
    """MemoryCrossAttention._forward_token_routed_attention + o_proj (memory_attention.py:480-716, 452-456) with
    per-token chapter weights:

        out = Wo [ attn(q, shared rows)  +  rho * sum_s w[t,s] softmax(q K_{c(t,s)}^T) V_{c(t,s)} ]

    The routed bank is projected once (the reference projects it once per batch item); the shared branch is the
    dense attention kernel over the S*T shared rows with all B*L tokens as one sequence."""

    @staticmethod
    def _native(h, shared_mem, routed_mem, idx_local, wq, wk, wv, wo, num_heads, num_kv_heads, t, cd) -> bool:
        """Whether ``moc_token_attn_fwd`` takes the call: bf16 arithmetic, head_dim 64, whole 64-row chapters."""
        ok = (torch.float32, torch.bfloat16)
        return (cd == torch.bfloat16 and t == 64 and h.shape[-1] == num_heads * 64 and wk.shape[0] == num_kv_heads * 64
                and wv.shape == wk.shape and num_heads % num_kv_heads == 0 and wq.shape == wo.shape == (h.shape[-1], h.shape[-1])
                and wk.dtype == wq.dtype == wv.dtype == wo.dtype and wq.dtype in ok and h.dtype in ok and h.numel() > 0
                and idx_local.shape[-1] > 0 and routed_mem is not None and routed_mem.numel() > 0
                and routed_mem.shape[0] % 64 == 0 and routed_mem.dtype in ok
                and (shared_mem is None or shared_mem.dtype in ok))

    @staticmethod
    def forward(ctx, h, shared_mem, routed_mem, idx_local, weights, wq, wk, wv, wo, cfg):
        num_heads, num_kv_heads, t, rho, cd = cfg
        b, l, d = h.shape
        rows = b * l
        ctx.desc = None
        if _TokenRoutedAttention._native(h, shared_mem, routed_mem, idx_local, wq, wk, wv, wo, num_heads, num_kv_heads, t, cd):
            need_grad = any(ctx.needs_input_grad)
            desc, out, keep = ops.token_attn_fwd(h.reshape(rows, d), shared_mem, routed_mem, idx_local, weights, wq, wk, wv, wo,
                                                 num_heads, num_kv_heads, rho, need_grad)
            if need_grad:
                ctx.desc = desc
                ctx.meta = (tuple(h.shape), weights.dtype, tuple(weights.shape))
                ctx.save_for_backward(*keep)
            return out.view(b, l, -1)
        dkv = wk.shape[0]
        head_dim = d // num_heads
        scale = head_dim ** -0.5
        h2 = ops.cast(h.reshape(rows, d).contiguous(), cd)
        wq_c, wo_c = ops.cast(wq, cd), ops.cast(wo, cd)
        wkv_c = ops.cast(torch.cat([wk, wv], dim=0), cd)
        q = ops.gemm(h2, wq_c, tag="q_proj")                                            # [rows, H*D]
        comb = None
        sh = None
        if shared_mem is not None and shared_mem.numel() > 0:
            sm2 = ops.cast(shared_mem.contiguous(), cd)
            kv_sh = ops.gemm(sm2, wkv_c, tag="kv_proj_shared")                          # [S*T, 2*dkv]
            # bf16 attention backward wants the query count in multiples of 64: pad with zero rows
            pad = (-rows) % 64 if cd == torch.bfloat16 else 0
            q_sh = q if pad == 0 else torch.cat([q, q.new_zeros(pad, q.shape[1])], dim=0)
            o_sh, lse_sh = ops.attn_fwd(q_sh.view(1, rows + pad, -1), kv_sh.view(1, kv_sh.shape[0], -1), num_heads,
                                        num_kv_heads, scale)
            sh = (sm2, kv_sh, q_sh, o_sh, lse_sh, pad)
            comb = o_sh.view(rows + pad, -1)[:rows]
        rt = None
        k_sel = idx_local.shape[-1]
        if routed_mem is not None and routed_mem.numel() > 0 and k_sel > 0:
            rm2 = ops.cast(routed_mem.contiguous(), cd)
            kv_rt = ops.gemm(rm2, wkv_c, tag="kv_proj_routed")                          # [(C-S)*T, 2*dkv]
            n_rt = kv_rt.shape[0]
            k4 = kv_rt[:, :dkv].unflatten(1, (num_kv_heads, head_dim)).unsqueeze(0)
            v4 = kv_rt[:, dkv:].unflatten(1, (num_kv_heads, head_dim)).unsqueeze(0)
            w2 = weights.reshape(1, rows, k_sel).float().contiguous()
            q4 = q.view(1, rows, num_heads, head_dim)
            base = None if comb is None else comb.contiguous().view(1, rows, num_heads, head_dim)
            bidx = idx_local.reshape(1, rows, 1, k_sel).expand(1, rows, num_kv_heads, k_sel).to(torch.int32).contiguous()
            comb4, lse_slots = ops.sparse_attn_weighted_fwd(q4, k4, v4, bidx, w2, t, scale, base=base, out_scale=rho)
            comb = comb4.view(rows, -1)
            rt = (rm2, kv_rt, bidx, w2, lse_slots, n_rt)
        if comb is None:
            comb = q.new_zeros(rows, d)
        out = ops.gemm(comb.contiguous(), wo_c, out_dtype=h.dtype if h.dtype in (torch.float32, cd) else cd, tag="o_proj")
        ctx.cfg = cfg
        ctx.meta = (b, l, d, dkv, scale, h.dtype, None if shared_mem is None else shared_mem.dtype,
                    None if routed_mem is None else routed_mem.dtype, weights.dtype,
                    (wq.dtype, wk.dtype, wv.dtype, wo.dtype))
        ctx.sh, ctx.rt = sh, rt
        ctx.save_for_backward(h2, q, comb, wq_c, wkv_c, wo_c)
        return out.view(b, l, -1).to(h.dtype)

    @staticmethod
    def backward(ctx, g):
        if ctx.desc is not None:
            h_shape, w_dtype, w_shape = ctx.meta
            d_h, d_sh, d_rt, d_w, d_wq, d_wkv, d_wo = ops.token_attn_bwd(ctx.desc, ctx.saved_tensors, g,
                                                                        ctx.needs_input_grad[1], ctx.needs_input_grad[2])
            dkv, wd = d_wkv.shape[0] // 2, ctx.saved_tensors[5].dtype
            return (d_h.view(h_shape), d_sh, d_rt, None, _cast(d_w, w_dtype).view(w_shape), _cast(d_wq, wd),
                    _cast(d_wkv[:dkv], wd), _cast(d_wkv[dkv:], wd), _cast(d_wo, wd), None)
        h2, q, comb, wq_c, wkv_c, wo_c = ctx.saved_tensors
        num_heads, num_kv_heads, t, rho, cd = ctx.cfg
        b, l, d, dkv, scale, h_dtype, sh_dtype, rt_dtype, w_dtype, wdt = ctx.meta
        rows = b * l
        head_dim = d // num_heads
        f32 = torch.float32
        g2 = ops.cast(g.reshape(rows, -1).contiguous(), cd)
        d_comb = ops.gemm(g2, wo_c, b_kmajor=False, tag="d_attn_out")                   # [rows, H*D]
        d_wo = ops.gemm(g2, comb, a_kmajor=False, b_kmajor=False, out_dtype=f32,
                        split_k=_weight_grad_splits(cd, rows, wo_c.shape[0], wo_c.shape[1]), tag="d_wo")
        d_q = None
        d_wkv = None
        d_shared = d_routed = d_weights = None
        if ctx.sh is not None:
            sm2, kv_sh, q_sh, o_sh, lse_sh, pad = ctx.sh
            dc = d_comb if pad == 0 else torch.cat([d_comb, d_comb.new_zeros(pad, d_comb.shape[1])], dim=0)
            d_q_sh, d_kv_sh = ops.attn_bwd(q_sh.view(1, rows + pad, -1), kv_sh.view(1, kv_sh.shape[0], -1), o_sh, lse_sh,
                                           dc.view(1, rows + pad, -1), num_heads, num_kv_heads, scale)
            d_q = d_q_sh.view(rows + pad, -1)[:rows].contiguous()
            d_kv_sh2 = d_kv_sh.view(kv_sh.shape[0], -1)
            d_shared = ops.gemm(d_kv_sh2, wkv_c, b_kmajor=False, out_dtype=sh_dtype if sh_dtype in (f32, cd) else cd,
                                tag="d_shared_mem").to(sh_dtype)
            d_wkv = ops.gemm(d_kv_sh2, sm2, a_kmajor=False, b_kmajor=False, out_dtype=f32,
                             split_k=_weight_grad_splits(cd, sm2.shape[0], 2 * dkv, d), tag="d_wkv_shared")
        if ctx.rt is not None:
            rm2, kv_rt, bidx, w2, lse_slots, n_rt = ctx.rt
            k4 = kv_rt[:, :dkv].unflatten(1, (num_kv_heads, head_dim)).unsqueeze(0)
            v4 = kv_rt[:, dkv:].unflatten(1, (num_kv_heads, head_dim)).unsqueeze(0)
            d_kv_rt = torch.zeros(n_rt, 2 * dkv, dtype=f32, device=q.device)
            dk4 = d_kv_rt[:, :dkv].unflatten(1, (num_kv_heads, head_dim)).unsqueeze(0)
            dv4 = d_kv_rt[:, dkv:].unflatten(1, (num_kv_heads, head_dim)).unsqueeze(0)
            q4, dc4 = q.view(1, rows, num_heads, head_dim), d_comb.view(1, rows, num_heads, head_dim)
            d_q4 = None if d_q is None else d_q.view(1, rows, num_heads, head_dim)
            d_q, d_w = ops.sparse_attn_weighted_bwd(q4, k4, v4, bidx, w2, lse_slots, dc4, t, scale, rho, dk4, dv4,
                                                    d_q_accum=d_q4)
            d_kv_c = ops.cast(d_kv_rt, cd)
            d_q = d_q.view(rows, -1)
            d_weights = d_w.view(b, l, -1).to(w_dtype)
            # written in the bank's dtype by the projection's epilogue (an fp32 master bank: no conversion pass
            # over 805 MB afterwards)
            d_routed = ops.gemm(d_kv_c, wkv_c, b_kmajor=False, out_dtype=rt_dtype if rt_dtype in (f32, cd) else cd,
                                tag="d_routed_mem").to(rt_dtype)
            g_wkv = ops.gemm(d_kv_c, rm2, a_kmajor=False, b_kmajor=False, out_dtype=f32,
                             split_k=_weight_grad_splits(cd, n_rt, 2 * dkv, d), tag="d_wkv_routed")
            d_wkv = g_wkv if d_wkv is None else d_wkv + g_wkv
        if d_q is None:
            d_q = q.new_zeros(rows, d)
        d_h = ops.gemm(d_q, wq_c, b_kmajor=False, tag="d_h").view(b, l, d).to(h_dtype)
        d_wq = ops.gemm(d_q, h2, a_kmajor=False, b_kmajor=False, out_dtype=f32,
                        split_k=_weight_grad_splits(cd, rows, d, d), tag="d_wq")
        if d_wkv is None:
            d_wkv = torch.zeros(2 * dkv, d, dtype=f32, device=q.device)
        return (d_h, d_shared, d_routed, None, d_weights, d_wq.to(wdt[0]), d_wkv[:dkv].to(wdt[1]),
                d_wkv[dkv:].to(wdt[2]), d_wo.to(wdt[3]), None)


def token_routed_attention(h: torch.Tensor, shared_memory: Optional[torch.Tensor],
                           routed_memory: Optional[torch.Tensor], token_chapter_indices: torch.Tensor,
                           chapter_weights: torch.Tensor, wq, wk, wv, wo, *, num_heads: int,
                           num_kv_heads: Optional[int], tokens_per_chapter: int, routed_scale: float = 1.0,
                           compute_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """Token-routed memory cross-attention with router-weighted chapters, output projection included.
    ``token_chapter_indices`` [B,L,k] are ids LOCAL to ``routed_memory`` (global id minus the shared prefix,
    model.py:583-595); ``chapter_weights`` [B,L,k] carry the router's gradient."""
    cfg = (int(num_heads), int(num_kv_heads or num_heads), int(tokens_per_chapter), float(routed_scale),
           compute_dtype or h.dtype)
    return _TokenRoutedAttention.apply(h, shared_memory, routed_memory, token_chapter_indices, chapter_weights,
                                       wq, wk, wv, wo, cfg)


class _Linear(torch.autograd.Function):
    """y = x W^T by the projection kernels (nn.Linear without bias), differentiable in x and W."""

    @staticmethod
    def forward(ctx, x, w, cd):
        x2 = ops.cast(x.reshape(-1, x.shape[-1]).contiguous(), cd)
        wc = ops.cast(w.contiguous(), cd)
        ctx.save_for_backward(x2, wc)
        ctx.meta = (x.shape, x.dtype, w.dtype, cd)
        return ops.gemm(x2, wc).view(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, g):
        x2, wc = ctx.saved_tensors
        shape, x_dtype, w_dtype, cd = ctx.meta
        g2 = ops.cast(g.reshape(-1, g.shape[-1]).contiguous(), cd)
        d_x = ops.gemm(g2, wc, b_kmajor=False).view(shape).to(x_dtype) if ctx.needs_input_grad[0] else None
        d_w = (ops.gemm(g2, x2, a_kmajor=False, b_kmajor=False, out_dtype=torch.float32).to(w_dtype)
               if ctx.needs_input_grad[1] else None)
        return d_x, d_w, None


def linear(x: torch.Tensor, w: torch.Tensor, compute_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    return _Linear.apply(x, w, compute_dtype or x.dtype)


class _DenseAttention(torch.autograd.Function):
    """softmax(q K^T scale) V for q [B, L, H*D] and kv [B, N, 2*HK*D] (K heads then V heads per row)."""

    @staticmethod
    def forward(ctx, q, kv, num_heads, num_kv_heads, scale):
        o, lse = ops.attn_fwd(q, kv, num_heads, num_kv_heads, scale)
        ctx.save_for_backward(q, kv, o, lse)
        ctx.cfg = (num_heads, num_kv_heads, scale)
        return o

    @staticmethod
    def backward(ctx, g):
        q, kv, o, lse = ctx.saved_tensors
        d_q, d_kv = ops.attn_bwd(q, kv, o, lse, g.contiguous(), *ctx.cfg)
        return d_q, d_kv, None, None, None


def token_routed_attention_joint(h, shared_memory, routed_memory, token_chapter_indices, wq, wk, wv, wo, *,
                                 num_heads: int, num_kv_heads: Optional[int], tokens_per_chapter: int,
                                 routed_scale: float = 1.0, compute_dtype: Optional[torch.dtype] = None):
    """Token-routed attention WITHOUT chapter weights (memory_attention.py:688-704): the selected chapters of a
    token share one softmax; out = Wo [ attn(q, shared) + rho * attn(q, selected chapters) ].  Composed from the
    differentiable projection, dense-attention and per-token sparse-attention operators."""
    from .memory_cross_attn import MemoryCrossAttnFunction
    cd = compute_dtype or h.dtype
    hk = int(num_kv_heads or num_heads)
    b, l, d = h.shape
    rows = b * l
    head_dim = d // num_heads
    scale = head_dim ** -0.5
    q = linear(h.reshape(1, rows, d), wq, cd)                                        # [1, rows, H*D]
    comb = None
    if shared_memory is not None and shared_memory.numel() > 0:
        kv_sh = torch.cat([linear(shared_memory, wk, cd), linear(shared_memory, wv, cd)], dim=-1).unsqueeze(0)
        pad = (-rows) % 64 if cd == torch.bfloat16 else 0
        q_sh = q if pad == 0 else torch.cat([q, q.new_zeros(1, pad, q.shape[-1])], dim=1)
        comb = _DenseAttention.apply(q_sh, kv_sh, num_heads, hk, scale)[:, :rows]
    k_sel = token_chapter_indices.shape[-1]
    if routed_memory is not None and routed_memory.numel() > 0 and k_sel > 0 and tokens_per_chapter > 0:
        k4 = linear(routed_memory, wk, cd).view(1, -1, hk, head_dim)
        v4 = linear(routed_memory, wv, cd).view(1, -1, hk, head_dim)
        bidx = token_chapter_indices.reshape(1, rows, 1, k_sel).expand(1, rows, hk, k_sel).to(torch.int32).contiguous()
        routed = MemoryCrossAttnFunction.apply(q.view(1, rows, num_heads, head_dim).contiguous(), k4.contiguous(),
                                               v4.contiguous(), bidx, int(tokens_per_chapter), scale)
        routed = routed.view(1, rows, -1) * float(routed_scale)
        comb = routed if comb is None else comb + routed
    if comb is None:
        comb = q.new_zeros(1, rows, d)
    return linear(comb, wo, cd).view(b, l, -1).to(h.dtype)
