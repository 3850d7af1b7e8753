"""Fused residual-add + RMSNorm (reference: lite_llama/kernels/skip_rmsnorm.py:192-234)."""

from __future__ import annotations

import torch

from . import _native
from ._common import check, dtype_code, lib, no_grad, ptr, require_cuda, stream_handle


def skip_rmsnorm(X, residual, weight, eps=1e-5):
    """``(Y, residual)``: ``residual += X`` in place, ``Y = rmsnorm(residual) * weight``.

    With ``residual=None`` this is plain RMSNorm and ``X`` is echoed back as the second value,
    exactly like the reference (skip_rmsnorm.py:219,234). The last dim is normalised; any leading
    shape is accepted (the per-head q/k norm passes ``[tokens, heads, head_dim]``).
    """
    return _native.norm(X, residual, weight, eps) or _skip_rmsnorm(X, residual, weight, eps)


@no_grad
def _skip_rmsnorm(X, residual, weight, eps):
    require_cuda(X, residual, weight)
    orig_shape = X.shape
    n = orig_shape[-1]
    # matrices go through as they are (unless the results would inherit a requires_grad); all rows follow one another, whatever
    # stride a single one claims
    flat = len(orig_shape) == 2 and not X.requires_grad and X.is_contiguous() and \
        (residual is None or (residual.shape == orig_shape and not residual.requires_grad and residual.is_contiguous()))
    x2 = X if flat else X.contiguous().view(-1, n)
    code = dtype_code(x2, "X")
    if weight.dtype != x2.dtype:
        raise ValueError(f"weight dtype {weight.dtype} must match X dtype {x2.dtype}")
    w = weight.contiguous()
    y = torch.empty_like(x2)
    r2 = None
    if residual is not None:
        if residual.dtype != x2.dtype:
            raise ValueError(f"residual dtype {residual.dtype} must match X dtype {x2.dtype}")
        # aliases the caller's residual when it is contiguous
        r2 = residual if flat else residual.contiguous().view(-1, n)
    check(
        lib().b2l_skip_rmsnorm(
            y.data_ptr(), x2.data_ptr(), ptr(r2), w.data_ptr(), x2.shape[0], n, n, n, n, float(eps), code, stream_handle(),
        )
    )
    if flat:
        return y, (x2 if r2 is None else r2)
    if r2 is not None:
        return y.view(orig_shape), r2.view(orig_shape)
    return y.view(orig_shape), x2.view(orig_shape)


def can_fuse_int8_quant(n: int) -> bool:
    """Shapes the fused norm + int8 quantisation kernel takes (16-byte rows kept in registers)."""
    return n % 8 == 0 and n <= 16384


def skip_rmsnorm_quant_int8(X, residual, weight, eps=1e-5):
    """``skip_rmsnorm`` whose output goes straight into a SmoothQuant GEMM: returns ``(q int8 [rows, n],
    scales fp32 [rows], residual)`` -- the per-token dynamic quantisation of the (fp16-rounded) norm output
    (reference: skip_rmsnorm.py:192-234 then quantization/w8a8.py:35-68), bit-identical to calling the two ops,
    in one launch and without writing the fp16 activations."""
    out = _native.norm_quant(X, residual, weight, eps)
    if out is not None:
        return *out, (X if residual is None else residual)
    return _skip_rmsnorm_quant_int8(X, residual, weight, eps)


@no_grad
def _skip_rmsnorm_quant_int8(X, residual, weight, eps):
    require_cuda(X, residual, weight)
    orig_shape = X.shape
    n = orig_shape[-1]
    # matrices go through as they are (unless the results would inherit a requires_grad); all rows follow one another, whatever
    # stride a single one claims
    flat = len(orig_shape) == 2 and not X.requires_grad and X.is_contiguous() and \
        (residual is None or (residual.shape == orig_shape and not residual.requires_grad and residual.is_contiguous()))
    x2 = X if flat else X.contiguous().view(-1, n)
    code = dtype_code(x2, "X")
    if weight.dtype != x2.dtype:
        raise ValueError(f"weight dtype {weight.dtype} must match X dtype {x2.dtype}")
    if not can_fuse_int8_quant(n):
        raise ValueError(f"skip_rmsnorm_quant_int8 needs n % 8 == 0 and n <= 16384, got {n}")
    w = weight.contiguous()
    r2 = None
    if residual is not None:
        if residual.dtype != x2.dtype:
            raise ValueError(f"residual dtype {residual.dtype} must match X dtype {x2.dtype}")
        r2 = residual.contiguous().view(-1, n)
    q = torch.empty((x2.shape[0], n), dtype=torch.int8, device=x2.device)
    s = torch.empty((x2.shape[0],), dtype=torch.float32, device=x2.device)
    check(
        lib().b2l_skip_rmsnorm_quant_int8(
            q.data_ptr(), s.data_ptr(), x2.data_ptr(), ptr(r2), w.data_ptr(), x2.shape[0], n, n, n, n, float(eps), code,
            stream_handle(),
        )
    )
    return q, s, (r2.view(orig_shape) if r2 is not None else x2.view(orig_shape))
