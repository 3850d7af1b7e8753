"""The native form of the hot shims (csrc/host/fast_calls.cpp).

Each function takes the plain form of its shim's call and returns None for every other form; the shim then goes on in Python.
Where the extension is missing or was built for another header, source, interpreter or torch, every call goes on in Python.
"""

from __future__ import annotations

import ctypes

import torch

from ..build import fast_tag
from . import _common

# the order of the function table in fast_calls.cpp
_ABI = ("b2l_quant_gemm_workspace_bytes", "b2l_linear_workspace_bytes", "b2l_w8a16_matmul", "b2l_w4a16_matmul_packed",
        "b2l_linear", "b2l_w8a8_gemm", "b2l_quantize_activations_int8", "b2l_skip_rmsnorm", "b2l_skip_rmsnorm_quant_int8",
        "b2l_swiglu", "b2l_last_error")
NAMES = ("w8a16", "w4a16_packed", "linear", "w8a8", "quantize", "norm", "norm_quant", "swiglu")


def _address(name: str) -> int:
    fn = getattr(_common.lib(), name)
    return ctypes.cast(fn, ctypes.c_void_p).value or 0 if isinstance(fn, ctypes._CFuncPtr) else 0


def _python(*_args) -> None:
    """The extension is not there."""


def _table() -> dict:
    try:
        from .. import _fast
        wanted = fast_tag(torch.__version__)
    except (ImportError, OSError):          # not built, or its source is not there to compare with
        return {}
    if getattr(_fast, "built_for", None) != wanted:
        return {}
    _fast.init(*map(_address, _ABI), _common.zeroed_workspace, _common.counters)
    return {name: getattr(_fast, name) for name in NAMES}


def _first(name: str):
    """Stands in for ``name`` until the first call on the GPU, which needs the library loaded in any case."""
    def call(*args):
        if not args[0].is_cuda:
            return None
        table = _table()
        globals().update({n: table.get(n, _python) for n in NAMES})
        return globals()[name](*args)
    return call


w8a16, w4a16_packed, linear, w8a8, quantize, norm, norm_quant, swiglu = map(_first, NAMES)
