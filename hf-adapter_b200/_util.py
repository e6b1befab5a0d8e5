"""Host-side helpers shared by the operator wrappers."""
from __future__ import annotations

import contextlib
import gc

import torch

from . import _lib

_DT = {torch.float16: _lib.F16, torch.bfloat16: _lib.BF16, torch.float32: _lib.F32}


def dt_code(t: torch.Tensor) -> int:
    try:
        return _DT[t.dtype]
    except KeyError:
        raise ValueError(f"unsupported activation dtype {t.dtype}") from None


def stream_ptr(t: torch.Tensor) -> int:
    # (the stream object that torch.cuda.current_stream builds first costs several times this call, once per launch)
    return torch._C._cuda_getCurrentRawStream(t.get_device())


def require_cuda(*tensors, what: str) -> None:
    """There is no CPU path in this package: every tensor must live on one CUDA device."""
    dev = None
    for t in tensors:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError(f"{what}: tensors must be CUDA tensors (this package has no CPU fallback)")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise ValueError(f"{what}: tensors must be on the same device")


def same_dtype(first, *rest, what: str) -> None:
    for t in rest:
        if t is not None and t.dtype != first.dtype:
            raise ValueError(f"{what}: dtype mismatch ({t.dtype} vs {first.dtype})")


def zero_lists(*lists) -> None:
    """Zeros into every tensor of lists that are of one type each, many tensors a launch (20 M elements each time) and not one: a prefill
    begins with the buffers of all layers, and the GPU idles meanwhile.  Large fp32 tensors are filled one by one: the fill of one
    tensor runs at 6 TB/s there, the other form at 4.5, and the launches no longer show."""
    # us, together / one by one: 32 fp32 tensors of 1 MiB 18 / 161, of 8 74 / 165, of 24 190 / 206, of 32 246 / 269, of 48 370 / 336, of 64 486 / 402; in fp16 of
    # 24 MiB 211 / 335, of 64 539 / 666
    for ts in lists:
        if not ts:
            continue
        if ts[0].element_size() == 4 and ts[0].numel() > 10 << 20 and min(t.numel() for t in ts) > 10 << 20:
            for t in ts:
                t.zero_()
        else:
            torch._foreach_zero_(ts)


def ptr(t):
    return 0 if t is None else t.data_ptr()


def no_fallback(force_fallback: bool, what: str) -> None:
    if force_fallback:
        raise RuntimeError(f"{what}: force_fallback=True requests the pure-PyTorch path, which this package does not ship")


@contextlib.contextmanager
def capture(graph):
    """``torch.cuda.graph(graph)`` with the cyclic collector held off: a model that was dropped leaves its own graphs in a
    reference cycle, and a graph that the collector destroys in the middle of a capture invalidates that capture."""
    on = gc.isenabled()
    gc.disable()
    try:
        with torch.cuda.graph(graph):
            yield
    finally:
        if on:
            gc.enable()
