"""The per-layer pack tuple of the reference's graph decode path and the in-place layer step that consumes it.

The reference flattens every layer into a 41-slot tuple (rwkv7_hf/native_jit_packing.py:13-146) that its
``_block_ip_batched`` (rwkv7_hf/native_jit_decode.py:481-901) unpacks:

    0 i, 1 H, 2 N, 3 eps (= N * 1e-5), 4 has_pre, 5-6 pre_norm w/b, 7-8 attn_norm w/b, 9-10 ffn_norm w/b,
    11-16 x_r x_w x_k x_v x_a x_g [D], 17 k_k [A], 18 k_a [A], 19 r_k [H,N],
    20-23 Rw Kw Vw Ow, 24-26 w1 w2 w0, 27-29 a1 a2 a0, 30-32 v1 v2 v0 (layer 0: zero dummies), 33-34 g1 g2,
    35-36 g_norm w/b [A], 37 fx_k [D], 38 fK, 39 fV, 40 RKVw ([3,D,A] stacked dense r/k/v, or empty)

A projection slot holds the dense ``[out,in]`` weight tensor of an ``nn.Linear`` or, for a quantised projection,
the module itself as a callable operand whose ``rwkv7_forward_*`` hooks carry the fused epilogues.  This file
builds that tuple from a model of this package (``extract_graph_packs``) and runs one layer from it
(``block_ip_batched``): the model's own decode step is a loop over these calls, so a host that already holds
reference packs drives the same kernels through the same structure.
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import _lib
from . import gemm as _gemm
from . import lora as _lora
from . import norm_mix as _nm
from . import quant as _q
from . import recurrent as _rec
from . import rows as _rowsk
from ._util import zero_lists

PACK_SLOTS = 41
_QUANT_TYPES = (_q.MM4Linear, _q.MM8Linear, _q.A8W8Linear)


def graph_linear_operand(mod):
    """What a projection contributes to the pack: a quantised module stays a callable operand, a dense
    ``nn.Linear`` without bias is its weight tensor (rwkv7_hf/native_jit_graph_dispatch.py graph_linear_operand)."""
    if isinstance(mod, _QUANT_TYPES):
        return mod
    if isinstance(mod, nn.Linear) and mod.bias is None:
        return mod.weight
    return mod


def graph_linear_is_dense(op) -> bool:
    return isinstance(op, torch.Tensor)


def extract_graph_packs(model, *, rkv_policy: str = "", unused_as_zeros: bool = True):
    """``(packs, H, N, eps)`` for ``model`` (rwkv7_hf/native_jit_packing.py:61-146).  ``rkv_policy="vkwr_auto"`` stacks
    dense r/k/v weights into slot 40; any other value leaves that slot empty.  ``unused_as_zeros=False`` leaves None in
    the slots a layer does not use (its pre-norm, layer 0's v LoRA) instead of the reference's zeros: a decode step builds
    its packs inside the captured region, where each of those 65 tensors was a fill to replay."""
    layers = model.model.layers
    H = int(layers[0].attn.num_heads)
    N = int(layers[0].attn.head_dim)
    eps = float(N * 1e-5)
    emb = model.model.embeddings.weight
    hidden = int(emb.shape[1])
    A = H * N
    packs = []
    for i, layer in enumerate(layers):
        a = layer.attn
        vl = getattr(a, "v_lora", None)
        if vl is not None:
            v1, v2, v0 = graph_linear_operand(vl.lora[0]), vl.lora[2].weight, vl.lora[2].bias
        elif i == 0 and not unused_as_zeros:
            v1 = v2 = v0 = None
        else:
            v1 = torch.zeros(1, hidden, device=emb.device, dtype=emb.dtype)
            v2 = torch.zeros(A, 1, device=emb.device, dtype=emb.dtype)
            v0 = torch.zeros(A, device=emb.device, dtype=emb.dtype)
        if hasattr(layer, "pre_norm"):
            pre_w, pre_b, has_pre = layer.pre_norm.weight, layer.pre_norm.bias, 1
        elif not unused_as_zeros:
            pre_w, pre_b, has_pre = None, None, 0
        else:
            pre_w = torch.zeros(hidden, device=emb.device, dtype=emb.dtype)
            pre_b = torch.zeros(hidden, device=emb.device, dtype=emb.dtype)
            has_pre = 0
        r_op, k_op, v_op = (graph_linear_operand(m) for m in (a.r_proj, a.k_proj, a.v_proj))
        if rkv_policy == "vkwr_auto" and all(graph_linear_is_dense(o) for o in (r_op, k_op, v_op)):
            stacked = torch.stack((r_op.t(), k_op.t(), v_op.t())).contiguous()
        else:
            stacked = emb.new_empty((0,))
        packs.append((
            i, H, N, eps, has_pre,
            pre_w, pre_b, layer.attn_norm.weight, layer.attn_norm.bias,
            layer.ffn_norm.weight, layer.ffn_norm.bias,
            a.x_r.reshape(-1), a.x_w.reshape(-1), a.x_k.reshape(-1),
            a.x_v.reshape(-1), a.x_a.reshape(-1), a.x_g.reshape(-1),
            a.k_k, a.k_a, a.r_k,
            r_op, k_op, v_op, graph_linear_operand(a.o_proj),
            graph_linear_operand(a.w_lora.lora[0]), a.w_lora.lora[2].weight, a.w_lora.lora[2].bias,
            graph_linear_operand(a.a_lora.lora[0]), a.a_lora.lora[2].weight, a.a_lora.lora[2].bias,
            v1, v2, v0,
            graph_linear_operand(a.g_lora.lora[0]), a.g_lora.lora[2].weight,
            a.g_norm.weight, a.g_norm.bias,
            layer.ffn.x_k,
            graph_linear_operand(layer.ffn.key), graph_linear_operand(layer.ffn.value),
            stacked,
        ))
    return packs, H, N, eps


def init_batched_from_packs(packs, batch_size: int, device, dtype, *, state_dtype=None):
    """Zero recurrent buffers for ``batch_size`` sequences (rwkv7_hf/native_jit_packing.py:163-182):
    ``(state, xpa, xpf)`` lists with one ``[B,H,N,N]`` / ``[B,D]`` / ``[B,D]`` tensor per layer."""
    n = len(packs)
    H, N = int(packs[0][1]), int(packs[0][2])
    hid = int(packs[0][7].numel())
    if state_dtype is None:
        state_dtype = torch.float32
    state = [torch.empty(batch_size, H, N, N, device=device, dtype=state_dtype) for _ in range(n)]
    xpa = [torch.empty(batch_size, hid, device=device, dtype=dtype) for _ in range(n)]
    xpf = [torch.empty(batch_size, hid, device=device, dtype=dtype) for _ in range(n)]
    zero_lists(state, [*xpa, *xpf])
    return state, xpa, xpf


# ---------------------------------------------------------------------------------------------- operands
def apply_linear(op, x, *, relu2=False, residual=None, out=None, static=False):
    """Apply a projection operand of the pack: a quantised module (epilogues fused through its rwkv7_forward_* hooks,
    as the reference's dispatch probes them: rwkv7_hf/native_jit_graph_dispatch.py:487-523), a dense ``[out,in]``
    weight tensor, or an ``nn.Linear`` (fp16 / bf16: this library's GEMM from 64 rows up, its row kernel up to 8; else
    one library GEMM).  ``static``: a call of a layer step, where the kernel launched just before on this stream does not write
    a dense weight."""
    if isinstance(op, _QUANT_TYPES):
        if relu2:
            if hasattr(op, "rwkv7_forward_relu2"):
                return op.rwkv7_forward_relu2(x)
            return torch.relu(op(x)) ** 2
        if residual is not None:
            return op.rwkv7_forward_add(x, residual)
        if out is not None:
            return op.rwkv7_forward_into(x, out)
        return op(x)
    weight, bias = (op, None) if isinstance(op, torch.Tensor) else (op.weight, op.bias)
    rows = x.numel() // int(x.shape[-1])
    if rows >= _gemm.MIN_ROWS and _gemm.takes(x, weight) and (bias is None or bias.dtype == x.dtype):
        # many rows over a dense fp16 / bf16 weight: this library's tensor-core GEMM, epilogue fused
        return _gemm.dense_linear(x, weight, bias, relu2=relu2, residual=residual, out=out)
    N = int(weight.shape[0])
    whole = lambda t: t is None or (t.dtype == x.dtype and t.is_contiguous() and t.numel() == rows * N)
    # (inside a layer step, which is opaque to autograd and traces as a whole, nothing is there to follow)
    seen = not static and rows <= _rowsk.MAX_ROWS and _rowsk.followed(*(t for t in (x, weight, residual) if t is not None))
    if (bias is None and not seen and _rowsk.takes_dense(x, weight) and whole(residual) and whole(out)
            and _rowsk.prefers_dense(rows, int(weight.shape[1]), N, relu2 or residual is not None, static)):
        epi = _lib.EPI_RELU2 if relu2 else _lib.EPI_ADD if residual is not None else _lib.EPI_NONE
        y, = _rowsk.rows_gemv((x.reshape(rows, -1),), (weight,), out_features=(N,), fmts=(_rowsk.DENSE,), epilogues=(epi,),
                              residuals=(None if relu2 else residual,), outs=None if out is None else (out.reshape(rows, N),),
                              static_weights=static)
        return y.reshape(*x.shape[:-1], N) if out is None else out
    y = F.linear(x, weight, bias)
    if relu2:
        y = torch.relu(y) ** 2
    elif residual is not None:
        y = y + residual
    if out is not None:
        out.copy_(y)
        return out
    return y


def _weight_of(op):
    return op if isinstance(op, torch.Tensor) else op.weight


def _out_features(op):
    return int(op.shape[0]) if isinstance(op, torch.Tensor) else int(op.out_features)


def _rkv_tiled(ops, xs):
    """The tiled weights of r / k / v when all three are int4 (or row-wise int8) projections of one shape that the
    tensor-core decode kernel takes in one launch; None otherwise."""
    int4 = all(isinstance(m, _q.MM4Linear) for m in ops)
    int8 = all(isinstance(m, _q.MM8Linear) and m.sm7x_rowwise for m in ops)
    if not (int4 or int8) or any(m.bias is not None for m in ops):
        return None
    if len({(m.in_features, m.out_features) for m in ops}) != 1:
        return None
    tiled = [m.tiled_for(x_) for m, x_ in zip(ops, xs)]
    return None if any(t is None for t in tiled) else tiled


def _rkv_launch(ops, xs, tiled):
    if isinstance(ops[0], _q.MM8Linear):
        return _q.w8_tiled_linear_group(xs, tiled, [m.row_scale for m in ops], ops[0].out_features, ops[0].in_features)
    return _q.w4_tiled_linear_group(xs, tiled, ops[0].out_features, ops[0].in_features)


def rkv_grouped(ops, xr, xk, xv):
    """r / k / v through one grouped launch where ``_rkv_tiled`` has their weights; None otherwise."""
    tiled = _rkv_tiled(ops, (xr, xk, xv))
    return None if tiled is None else _rkv_launch(ops, (xr, xk, xv), tiled)


def _rows_operand(op, x):
    """``(fmt, weight, scale, out_features)`` when the projection ``op`` of the few rows ``x`` runs on the row kernel."""
    if isinstance(op, _q.MM4Linear) or (isinstance(op, _q.MM8Linear) and op.sm7x_rowwise):
        ok = (op.bias is None and x.is_contiguous() and int(x.shape[-1]) == op.in_features
              and _q.few_rows_quant(int(x.shape[0]), op.in_features, op.out_features, 4 if isinstance(op, _q.MM4Linear) else 8))
        tiled = op.tiled_for(x) if ok else None
        if tiled is None:
            return None
        return (_rowsk.INT4, tiled, None, op.out_features) if isinstance(op, _q.MM4Linear) else \
            (_rowsk.INT8, tiled, op.row_scale, op.out_features)
    weight = op if isinstance(op, torch.Tensor) else op.weight if isinstance(op, nn.Linear) and op.bias is None else None
    if weight is None or not _rowsk.takes_dense(x, weight):
        return None
    return _rowsk.DENSE, weight, None, int(weight.shape[0])


def rows_projections(ops, xs, epilogues=None):
    """The projections ``ops[i](xs[i])`` of a few rows in one launch, or None when one of them does not take that route.
    For the inside of a layer step: the kernel before it writes activations only."""
    if xs[0].dim() != 2 or not 1 <= int(xs[0].shape[0]) <= _rowsk.MAX_ROWS or xs[0].dtype not in (torch.float16, torch.bfloat16):
        return None
    got = [_rows_operand(o, x) for o, x in zip(ops, xs)]
    if any(g is None for g in got):
        return None
    return _rowsk.rows_gemv(xs, [g[1] for g in got], out_features=[g[3] for g in got], fmts=[g[0] for g in got],
                            scales=[g[2] for g in got], epilogues=epilogues, static_weights=True)


class StepContext:
    """What a layer step needs beyond the pack when it runs inside a larger program: side streams for the
    independent branches of the layer, and the sum over tensor-parallel ranks.  The default context is a single
    GPU with one side stream per device."""

    def __init__(self, side_stream=None, all_reduce=None, tp_world: int = 1, tp_rank: int = 0, lane: int = 0,
                 stream_base: int = 0, slot_ids=None, row_sum=None, idle_slot: int = -1):
        # slot_ids (int32 [B] on the device): the recurrent buffers handed to the layer step are slot pools
        # ([capacity, ...]) and batch row b lives in pool row slot_ids[b]; rows in idle_slot only pad the batch
        self.slot_ids, self.idle_slot = slot_ids, int(idle_slot)
        self._side_stream = side_stream
        self._all_reduce = all_reduce
        # row_sum(partial, lane) -> tp_comm.PeerRowSum or None: the communicator whose row kernels take the sum over
        # ranks in themselves.  defer_sum (set by step_batched between layers): the layer may return its UNSUMMED
        # ffn.value partial and raise `pending`; the next layer's first kernel then sums it.
        self._row_sum = row_sum
        self.defer_sum = False
        self.pending = False
        self.tp_world, self.tp_rank, self.lane, self.stream_base = int(tp_world), int(tp_rank), int(lane), int(stream_base)
        self._own = {}

    def side_stream(self, device, index: int):
        if self._side_stream is not None:
            return self._side_stream(device, self.stream_base + index)
        st = self._own.get((device, index))
        if st is None:
            st = self._own[(device, index)] = torch.cuda.Stream(device=device)
        return st

    def all_reduce(self, t):
        return t if self._all_reduce is None else self._all_reduce(t, self.lane)

    def row_sum(self, partial):
        if self.tp_world == 1 or self._row_sum is None or partial.dim() != 2:
            return None
        return self._row_sum(partial, self.lane)


_DEFAULT_CONTEXT = StepContext()


def _lora_leads(op, rows: int, features: int) -> bool:
    """Whether the LoRA chain stays on the main stream when r / k / v are three products like ``op`` (of ``features`` inputs)."""
    # The longer branch leads: it starts on the programmatic edge of the kernel before it.  The chain is two launches whatever the width,
    # the products grow with it.  us a step, dense fp16 / bf16, chain first -> r first, at 9 / 16 / 32 / 48 / 63 rows (library GEMMs):
    # 768 wide 617 / 633 / 656 / 679 / 705 -> 652 / 669 / 690 / 708 / 729; 1536 1270 / 1313 / 1437 / 1499 / 1790 -> 1358 / 1315 / 1509 /
    # 1612 / 1715; 2048 1492 / 1539 / 1733 / 2014 / 1990 -> 1540 / 1590 / 1731 / 1885 / 2022; 2560 2486 / 2576 / 2799 / 3208 / 3312 -> 2417 /
    # 2504 / 2793 / 3045 / 3086.  At 64 / 128 / 256 rows (this library's GEMM): 768 1124 / 1213 / 1139 -> 1135 / 1219 / 1132; 1024 2297 / 2653 /
    # 2585 -> 2262 / 2484 / 2381; 2560 5835 / 6595 / 6936 -> 5634 / 6176 / 6442.  Affine int8, 2560 wide, 12 / 32 / 64 rows 10350 / 19217 / 9218 ->
    # 10190 / 19055 / 9235.  int8 x int8 (a quantiser and a product each), 12 / 64 rows: 7332 / 4913 -> 7312 / 4861 on one card, 7519 /
    # 5120 -> 8317 / 5497 on another.
    if isinstance(op, _q.A8W8Linear):
        return True
    return _out_features(op) * features < (2048 * 2048 if rows < _gemm.MIN_ROWS else 1024 * 1024)


def _wide_projections(ctx, x, ops, xs, downs, ups, down_x):
    """r / k / v and the LoRA pre-activations of a layer step on parallel branches (of the decode graph once captured):
    ``[r, k, v, w, a, g(, v_gate)]``."""
    main = torch.cuda.current_stream(x.device)
    # (tiled weights that are built on first use belong to the stream that outlives the branches: ahead of the fork)
    tiled = _rkv_tiled(ops, xs)
    fork = main.record_event()
    used = []

    def branch(i, ts, run):
        st = ctx.side_stream(x.device, i)
        st.wait_event(fork)
        used.append(st)
        with torch.cuda.stream(st):
            y = run()
        for t in ts:
            t.record_stream(st)
        return y

    def lora_chain(lean=False):
        hs = _lora.small_gemm_group(down_x, [_weight_of(w) for w in downs], acts=(1, 0, 2, 0)[:len(downs)], lean=lean)
        return _lora.small_gemm_group(hs, [_weight_of(w) for w in ups], lean=lean)

    if tiled is not None:
        # int4 / int8 r / k / v of equal shape: one launch streams all three weight sets (one pipeline fill, no split-K
        # exchange).  The LoRA chain is two launches long and leads, behind the kernel that made its inputs; they branch off
        lora = lora_chain(lean=int(x.shape[0]) > 16)
        branched = rkv = branch(0, xs, lambda: _rkv_launch(ops, xs, tiled))
    elif _lora_leads(ops[0], int(x.shape[0]), int(xs[0].shape[-1])):
        # independent projections on separate branches: the tail of one overlaps the ramp-up of the next
        lora = lora_chain()
        branched = rkv = [branch(i, (t,), lambda: apply_linear(o, t)) for i, (o, t) in enumerate(zip(ops, xs))]
    else:
        # they are the longer branch: r leads, and the LoRA kernels leave them the SMs' shared memory
        lora = branch(0, down_x, lambda: lora_chain(lean=True))
        k, v = (branch(i, (xs[i],), lambda: apply_linear(ops[i], xs[i])) for i in (1, 2))
        rkv, branched = [apply_linear(ops[0], xs[0]), k, v], (k, v, *lora)
    for st in used:
        main.wait_stream(st)
    _used_on(main, *branched)
    return [*rkv, *lora]


def _used_on(stream, *ts):
    """Results allocated on a branch and used on ``stream``: their memory waits for that use.  (Not under capture: the pool is
    the graph's own there, and every branch of a later layer starts behind the stream that used them.)"""
    if not torch.cuda.is_current_stream_capturing():
        for t in ts:
            t.record_stream(stream)


def block_ip_batched(x, state, xpa, xpf, v_first, p, sparse_ffn_out=None, fp16_elapsed=None,
                     fp16_advance_elapsed=False, route_observer=None, *, context: StepContext | None = None):
    """One layer for ``B`` sequences from its pack tuple, recurrent buffers updated in place
    (rwkv7_hf/native_jit_decode.py:481-901: same arguments, same return value).

    ``x [B,D]`` residual stream in, new residual stream out; ``state [B,H,N,N]`` (fp32, or fp16 with the
    ``fp16_elapsed`` int32 ``[B]`` phase counters of the FP16-state lane), ``xpa``/``xpf [B,D]`` and ``v_first [B,A]``
    are overwritten (with ``context.slot_ids`` they are slot pools ``[capacity, ...]`` and only the rows named there change).  Every launch is capturable in a CUDA graph.  ``sparse_ffn_out`` and ``route_observer`` belong to
    the reference's sparse-FFN experiment and must be None."""
    if sparse_ffn_out is not None or route_observer is not None:
        raise NotImplementedError("the sparse-FFN route of the reference is not part of this library")
    if len(p) != PACK_SLOTS:
        raise ValueError(f"a layer pack has {PACK_SLOTS} slots, got {len(p)}")
    (i, H, N, eps, has_pre,
     pre_w, pre_b, an_w, an_b, fn_w, fn_b,
     x_r, x_w, x_k, x_v, x_a, x_g, k_k, k_a, r_k,
     Rw, Kw, Vw, Ow, w1, w2, w0, a1, a2, a0, v1, v2, v0, g1, g2,
     gn_w, gn_b, fx_k, fK, fV, RKVw) = p
    ctx = context or _DEFAULT_CONTEXT
    if has_pre:
        x = _nm.layer_norm(x, pre_w, pre_b)
    slots = ctx.slot_ids
    rows_comm = ctx.row_sum(x)
    if ctx.pending and rows_comm is None:
        ctx.pending = False
        x = ctx.all_reduce(x)
    if ctx.pending:
        # x is the previous layer's ffn.value partial: the sum over ranks happens inside this kernel
        ctx.pending = False
        x, (xr, xw, xk, xv, xa, xg) = rows_comm.attn_norm_mix6(x, xpa, an_w, an_b, (x_r, x_w, x_k, x_v, x_a, x_g),
                                                              slot_ids=slots)
    else:
        xr, xw, xk, xv, xa, xg = _nm.fused_attn_norm_mix6_decode(x, xpa, an_w, an_b, x_r, x_w, x_k, x_v, x_a, x_g,
                                                                 slot_ids=slots)
    first = int(i) == 0
    downs, ups = ((w1, a1, g1), (w2, a2, g2)) if first else ((w1, a1, g1, v1), (w2, a2, g2, v2))
    down_x = (xw, xa, xg) if first else (xw, xa, xg, xv)
    # a few rows: r / k / v and the LoRA "down" products in one launch, the "up" products in the next (if they qualify: decided
    # before the first launch, whose results would be thrown away)
    few = None
    if all(_rowsk.takes_weight(_weight_of(u), x.dtype) and int(_weight_of(u).shape[1]) == _out_features(d) for u, d in zip(ups, downs)):
        few = rows_projections((Rw, Kw, Vw) + downs, (xr, xk, xv) + down_x,
                               ([_lib.EPI_NONE] * 3 + [_lib.EPI_TANH, _lib.EPI_NONE, _lib.EPI_SIGMOID, _lib.EPI_NONE])[:3 + len(downs)])
    if few is not None:
        r, k, v = few[:3]
        lora = rows_projections(ups, few[3:])
    else:
        r, k, v, *lora = _wide_projections(ctx, x, (Rw, Kw, Vw), (xr, xk, xv), downs, ups, down_x)
    w_raw, a_pre, g = lora[:3]
    extra = dict(v_out=v_first) if first else dict(v_first=v_first, v_gate=lora[3], v_gate_bias=v0, v_gate_is_raw=True)
    elapsed = fp16_elapsed if state.dtype == torch.float16 else None
    # the kernel launched just before the recurrence is a projection: it never writes the state
    out, _ = _rec.fused_recurrent_output_prepare_raw(
        r, w_raw, k, v, a_pre, state, g, k_k, k_a, r_k, gn_w, gn_b, eps=float(eps), new_state=state, w_bias=w0, a_bias=a0,
        a_is_raw=True, state_prefetch=True, elapsed=elapsed,
        advance_elapsed=bool(fp16_advance_elapsed) and elapsed is not None, slot_ids=slots, idle_slot=ctx.idle_slot, **extra)
    attn = apply_linear(Ow, out, static=True)
    if rows_comm is not None:
        x, mixed = rows_comm.ffn_add_norm_mix(x, attn, xpf, fn_w, fn_b, fx_k, slot_ids=slots)
    else:
        x, mixed = _nm.fused_ffn_add_norm_mix_decode(x, ctx.all_reduce(attn), xpf, fn_w, fn_b, fx_k, slot_ids=slots)
    hidden = apply_linear(fK, mixed, relu2=True, static=True)
    if ctx.tp_world > 1:
        # the residual rides in rank 0's partial sum (the projection's add epilogue): no extra add kernel
        part = apply_linear(fV, hidden, residual=x if ctx.tp_rank == 0 else None, static=True)
        if rows_comm is not None and ctx.defer_sum:
            ctx.pending = True
            return part
        return ctx.all_reduce(part)
    return apply_linear(fV, hidden, residual=x, static=True)


def step_batched(model, x, state, xpa, xpf, v_first, packs, *, fp16_elapsed=None, context: StepContext | None = None):
    """All layers of one decode step from their packs (rwkv7_hf/native_jit_decode.py:56-68 ``step_batched``): returns
    ``(x, state, xpa, xpf, v_first)`` with the buffers updated in place.  ``model`` is unused (kept for the
    reference's argument order)."""
    last = len(packs) - 1
    for li, p in enumerate(packs):
        if context is not None:
            context.defer_sum = li != last  # between layers the sum moves into the next layer's first kernel
        x = block_ip_batched(x, state[li], xpa[li], xpf[li], v_first, p, fp16_elapsed=fp16_elapsed,
                             fp16_advance_elapsed=li == last, context=context)
    return x, state, xpa, xpf, v_first
