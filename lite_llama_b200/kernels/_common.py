"""Shared plumbing for the ctypes shims: dtype codes, stream handle, scratch buffers."""

from __future__ import annotations

import functools

import torch

from .. import _lib

F16, BF16, F32 = 0, 1, 2

_DTYPE_CODE = {torch.float16: F16, torch.bfloat16: BF16}
_FLOAT_CODE = {torch.float16: F16, torch.bfloat16: BF16, torch.float32: F32}


def lib():
    return _lib.load()


def check(rc: int) -> None:
    _lib.check(rc)


def dtype_code(t: torch.Tensor, what: str) -> int:
    try:
        return _DTYPE_CODE[t.dtype]
    except KeyError:
        raise ValueError(f"{what} must be float16 or bfloat16, got {t.dtype}") from None


def float_code(t: torch.Tensor, what: str) -> int:
    """Dtype code for the entry points that also run in true 32-bit."""
    try:
        return _FLOAT_CODE[t.dtype]
    except KeyError:
        raise ValueError(f"{what} must be float16, bfloat16 or float32, got {t.dtype}") from None


def require_cuda(*tensors: torch.Tensor) -> None:
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise ValueError(
                "lite_llama_b200 kernels run on CUDA tensors only (there is no CPU fallback); "
                f"got a tensor on {t.device}"
            )


# A decode step calls a few dozen of these shims eagerly, and a launch takes the GPU 4 - 20 us: what a shim does in Python
# beside the launch (4.5 us) is kept to single C calls.  torch.cuda.current_stream() alone costs 3.2 us, a torch.no_grad()
# decorator 1.2 us, a reshape that changes nothing 1 us.
def stream_handle() -> int:
    """The current stream of the current device."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def no_grad(fn):
    """``torch.no_grad()`` as a decorator, without its context object; free where gradients are off already."""

    @functools.wraps(fn)
    def call(*args, **kwargs):
        if not torch.is_grad_enabled():
            return fn(*args, **kwargs)
        torch._C._set_grad_enabled(False)
        try:
            return fn(*args, **kwargs)
        finally:
            torch._C._set_grad_enabled(True)

    return call


def as_rows(t: torch.Tensor) -> torch.Tensor:
    """``t`` with its leading dimensions joined (``t`` itself if it is a matrix already)."""
    return t if t.dim() == 2 and t.size(1) else t.reshape(-1, t.shape[-1])


def own_rows(t: torch.Tensor) -> torch.Tensor:
    """The matrix ``t`` with rows that follow one another.  ``contiguous`` alone leaves the row stride of a one-row matrix,
    which may be anything (the width of the matrix it was sliced from, or 1); ``view`` makes it the row's length."""
    return t.contiguous().view(-1, t.size(1))


def unrows(y: torch.Tensor, like: torch.Tensor) -> torch.Tensor:
    """The matrix ``y`` with the leading dimensions of ``like``."""
    return y if like.dim() == 2 else y.view(*like.shape[:-1], y.shape[-1])


def weights_written() -> None:
    """Between the conversion or copy of a weight-side tensor and a GEMM that reads it: the GEMMs request their weights before
    the previous kernel has finished (csrc/common.cuh, programmatic dependent launch)."""
    check(lib().b2l_weights_written(stream_handle()))


@functools.lru_cache(maxsize=4096)
def quant_gemm_workspace_bytes(kind: int, m: int, n: int, k: int, group: int, device: int) -> int:
    """Workspace of a quantised GEMM: a function of the sizes and the device's SM count."""
    return lib().b2l_quant_gemm_workspace_bytes(kind, m, n, k, group)


def current_device() -> int:
    return torch._C._cuda_getDevice()


def index_width(t: torch.Tensor, what: str) -> int:
    if t.dtype == torch.int32:
        return 4
    if t.dtype == torch.int64:
        return 8
    raise ValueError(f"{what} must be int32 or int64, got {t.dtype}")


def ptr(t: torch.Tensor | None) -> int | None:
    return None if t is None else t.data_ptr()


# Split-K tickets: one persistent zeroed int32 buffer per device. Kernels leave it zeroed, and all
# launches are serialised on the current stream (the reference drives one stream per process too).
_COUNTERS: dict[int, torch.Tensor] = {}
_NUM_COUNTERS = 16384


def counters(device: torch.device) -> torch.Tensor:
    idx = device.index if device.index is not None else torch.cuda.current_device()
    buf = _COUNTERS.get(idx)
    if buf is None:
        buf = torch.zeros(_NUM_COUNTERS, dtype=torch.int32, device=device)
        _COUNTERS[idx] = buf
    return buf


# Stream-K partial sums of the quantised GEMMs travel through a workspace with flag-in-data words (csrc/gemm_quant.cu):
# the buffer must be all-zero when a launch starts and every launch leaves it all-zero, so it is persistent and zeroed
# once -- same contract (and same one-stream assumption) as the ticket counters above. A buffer that has to grow is
# replaced, never freed: a captured CUDA graph may still hold its address.
_ZEROED: dict[int, torch.Tensor] = {}
_ZEROED_RETIRED: list[torch.Tensor] = []


def zeroed_workspace(nbytes: int, device: torch.device) -> torch.Tensor | None:
    if nbytes <= 0:
        return None
    idx = device.index if device.index is not None else torch.cuda.current_device()
    buf = _ZEROED.get(idx)
    if buf is None or buf.numel() < nbytes:
        if buf is not None:
            _ZEROED_RETIRED.append(buf)
        size = max(int(nbytes), 2 * buf.numel() if buf is not None else 0, 1 << 24)
        buf = torch.zeros(size, dtype=torch.uint8, device=device)
        _ZEROED[idx] = buf
    return buf


def workspace(nbytes: int, device: torch.device) -> torch.Tensor | None:
    """Scratch allocated through torch's caching allocator (graph-safe, like the reference's
    ``torch.empty`` scratch in flashdecoding.py:350-358)."""
    if nbytes <= 0:
        return None
    return torch.empty(nbytes, dtype=torch.uint8, device=device)
