"""Projections over a few rows (csrc/row_gemv.cu): up to eight independent ones, dense or quantised, in one launch with
their activation / residual epilogues.  What a decode step of a few sequences runs instead of one library GEMM per
projection and pointwise kernels behind it (rwkv7_hf/native_jit_graph_dispatch.py:487-523 probes for such fused forms)."""
from __future__ import annotations

import ctypes

import torch
from torch.autograd import forward_ad
from torch.utils._python_dispatch import _get_current_dispatch_mode

from . import _lib
from ._util import dt_code, ptr, require_cuda, stream_ptr

DENSE, INT4, INT8 = 0, 1, 2
MAX_ROWS = 8
MAX_PROBLEMS = 8


def takes_dense(x, weight) -> bool:
    """``x @ weight.T`` with a dense weight: fp16 / bf16 CUDA operands of one dtype, contiguous and 16-byte aligned, few
    rows (anything else keeps its library GEMM)."""
    return (takes_weight(weight, x.dtype) and x.is_cuda and x.is_contiguous() and int(x.shape[-1]) == int(weight.shape[1])
            and x.data_ptr() % 16 == 0 and 1 <= x.numel() // int(weight.shape[1]) <= MAX_ROWS)


def takes_weight(weight, dtype) -> bool:
    """The part of ``takes_dense`` that the weight decides, for activations of ``dtype``."""
    return (weight.is_cuda and weight.dtype == dtype and dtype in (torch.float16, torch.bfloat16) and weight.dim() == 2
            and weight.is_contiguous() and weight.numel() > 0 and int(weight.shape[1]) % 8 == 0 and weight.data_ptr() % 16 == 0)


def followed(*ts) -> bool:
    """Whether more than the values of ``ts`` counts: a gradient or tangent to propagate, a functorch transform, a trace, a
    dispatch mode, a tensor subclass.  A kernel behind ctypes is opaque to all of these; a library GEMM is not."""
    return ((torch.is_grad_enabled() and any(t.requires_grad for t in ts)) or forward_ad._current_level >= 0
            or torch._C._are_functorch_transforms_active() or torch.jit.is_tracing() or torch.compiler.is_compiling()
            or _get_current_dispatch_mode() is not None or any(type(t) not in (torch.Tensor, torch.nn.Parameter) for t in ts))


def prefers_dense(rows: int, K: int, N: int, fused: bool, early: bool) -> bool:
    """Whether one dense product of ``rows`` rows on its own is faster here than as a library GEMM with pointwise kernels behind
    it.  ``fused``: an epilogue rides in it; ``early``: its weights may be requested under the kernel before it.  Library
    against this kernel in us, fp16, 1 / 8 rows:

    * a short K leaves the reads of x and the epilogue: 64 -> 2560 2.4 / 2.8 against 1.9 / 4.2, + residual 3.6 against 2.3 / 6.0; 256 ->
      2048 at 0.82 / 0.97 of the library's time, + residual 0.58 / 0.73;
    * more channels than a wave of CTAs takes: 2560 -> 2560 8.1 / 7.7 against 4.5 / 4.8, but 2560 -> 10240 10.8 against 12.3 / 12.9; 768 ->
      32768 10.7 against 10.1 / 11.4; 1024 -> 8192 5.6 against 4.2 / 4.4, 4096 -> 5120 10.5 against 10.1 / 10.5;
    * early, behind a norm kernel and with relu^2: 2560 -> 10240 13.9 / 14.2 against 12.4 / 12.9, 4096 -> 16384 25.6 / 26.7 against 23.2 / 24.0, 8192 ->
      8192 26.3 / 26.8 against 23.1 / 23.6; but 5120 -> 20480 37.4 against 41.3 / 42.4, and 20480 -> 5120 + residual 48.2 against 51.3 / 53.1."""
    if K < (32 if fused else 64) * rows or K * N > 1 << 26:
        return False
    if early:
        return N <= 16384
    return N <= 4096 or (N <= 8192 and (K <= 1024 or (fused and K * N <= 1 << 25)))


def _check_problem(i, x, w, N, fmt, scale, residual, out):
    """The kernel takes sizes from ``x`` and ``N`` alone: every other operand has to hold as much."""
    M, K = (int(v) for v in x.shape)
    holds = lambda t, n: t.is_contiguous() and t.numel() * t.element_size() >= n
    if fmt == DENSE:
        if tuple(w.shape) != (N, K) or w.dtype != x.dtype or not w.is_contiguous():
            raise ValueError(f"rows_gemv: weight {i} must be a contiguous [{N}, {K}] in the activation dtype, got {tuple(w.shape)}")
    elif fmt in (INT4, INT8):
        need = int((_lib.lib.rwkv7_w4g_tiled_bytes if fmt == INT4 else _lib.lib.rwkv7_w8_tiled_bytes)(K, N))
        if need <= 0 or not holds(w, need):
            raise ValueError(f"rows_gemv: weight {i} is no tiled copy of [{N}, {K}]")
    else:
        raise ValueError(f"rows_gemv: unknown weight format {fmt}")
    if fmt == INT8 and (scale is None or scale.dtype != x.dtype or not holds(scale, N * scale.element_size())):
        raise ValueError(f"rows_gemv: scale {i} must be [{N}] in the activation dtype")
    if residual is not None and (residual.dtype != x.dtype or residual.numel() != M * N or not residual.is_contiguous()):
        raise ValueError(f"rows_gemv: residual {i} must be a contiguous [{M}, {N}] in the activation dtype")
    if out is not None and not holds(out, M * N * x.element_size()):
        raise ValueError(f"rows_gemv: output {i} must be a contiguous [{M}, {N}]")


def rows_gemv(xs, weights, *, out_features, fmts, scales=None, residuals=None, outs=None, epilogues=None, static_weights=False):
    """``outs[i] = epilogue_i(xs[i] [M,K_i] @ W_i.T)`` in one launch.  ``weights[i]`` is dense ``[N,K]`` or a tiled copy
    (``quant.w4_repack_tiled`` / ``w8_repack_tiled``).  ``static_weights``: no weight is written by the kernel launched
    just before this call on the stream."""
    n = len(xs)
    if not 1 <= n <= MAX_PROBLEMS or any(x.dim() != 2 for x in xs):
        raise ValueError(f"rows_gemv takes 1..{MAX_PROBLEMS} inputs [rows, features]")
    M = int(xs[0].shape[0])
    scales = list(scales) if scales is not None else [None] * n
    residuals = list(residuals) if residuals is not None else [None] * n
    epilogues = list(epilogues) if epilogues is not None else [_lib.EPI_NONE] * n
    if any(int(x.shape[0]) != M or x.dtype != xs[0].dtype or not x.is_contiguous() for x in xs):
        raise ValueError("rows_gemv: all inputs need the same row count and dtype, contiguous")
    if any(len(v) != n for v in (weights, out_features, fmts, scales, residuals, epilogues)) or (outs is not None and len(outs) != n):
        raise ValueError("rows_gemv: one weight, output width, format, scale, residual, epilogue and output per input")
    for i, (x, w, N, fmt) in enumerate(zip(xs, weights, out_features, fmts)):
        _check_problem(i, x, w, int(N), fmt, scales[i], residuals[i], None if outs is None else outs[i])
    require_cuda(*xs, *weights, *scales, *residuals, *(outs or ()), what="rows_gemv")
    if outs is None:
        outs = [torch.empty((M, N), device=xs[0].device, dtype=xs[0].dtype) for N in out_features]
    arr = lambda ts: _lib.ptr_array([ptr(t) for t in ts])
    (xp, k0), (wp, k1), (sp, k2), (rp, k3), (op, k4) = (arr(t) for t in (xs, weights, scales, residuals, outs))
    IA = ctypes.c_int * n
    _lib.check(_lib.lib.rwkv7_rows_gemv(n, xp, wp, sp, rp, op, IA(*[int(x.shape[1]) for x in xs]), IA(*out_features), IA(*fmts),
                                        IA(*epilogues), M, dt_code(xs[0]), int(bool(static_weights)), stream_ptr(xs[0])),
               "rows_gemv")
    return outs
