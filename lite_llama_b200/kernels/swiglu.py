"""SiLU(gate) * up (reference: lite_llama/kernels/swiglu.py:45-65)."""

from __future__ import annotations

import torch

from . import _native
from ._common import as_rows, check, float_code, lib, no_grad, require_cuda, stream_handle, unrows


def swiglu_forward(a, b):
    c = _native.swiglu(a, b)
    return _swiglu_forward(a, b) if c is None else c


@no_grad
def _swiglu_forward(a, b):
    require_cuda(a, b)
    n_cols = a.shape[-1]
    a2, b2 = as_rows(a), as_rows(b) if b.shape[-1] == n_cols else b.reshape(-1, n_cols)
    if a2.stride(-1) != 1:
        a2 = a2.contiguous()
    if b2.stride(-1) != 1:
        b2 = b2.contiguous()
    code = float_code(a2, "a")
    c = a.new_empty((a2.shape[0], n_cols))
    check(
        lib().b2l_swiglu(
            c.data_ptr(), a2.data_ptr(), b2.data_ptr(), a2.shape[0], n_cols, a2.stride(0), b2.stride(0), c.stride(0),
            code, stream_handle(),
        )
    )
    return unrows(c, a)
