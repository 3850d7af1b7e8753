"""silu(a) * b in 16-byte units of one and of two rows a thread against the scalar form: the same bits, odd row counts, rows that
follow one another or not, units past the last block of a row."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,n", [(1, 8), (2, 2048), (295, 64), (296, 64), (297, 72), (301, 4104), (3, 140000), (65600, 16)])
def test_units_and_scalars_agree(rows, n, dtype):
    import lite_llama_b200.kernels as K

    wide = torch.randn(rows, 2 * n, device="cuda", dtype=dtype) * 4
    got = K.swiglu_forward(wide[:, :n], wide[:, n:])
    odd = torch.empty(rows * (2 * n + 1), device="cuda", dtype=dtype).view(rows, 2 * n + 1)      # rows off the boundary
    odd[:, 1:] = wide
    assert torch.equal(got, K.swiglu_forward(odd[:, 1:n + 1], odd[:, n + 1:]))
    a, b = wide.double().split(n, 1)
    want = a * torch.sigmoid(a) * b
    # one rounding to the activation type; the 32-bit exponential and divide are within 1e-5
    assert ((got.double() - want).abs() <= want.abs() * (torch.finfo(dtype).eps / 2 + 1e-5) + 1e-6).all()
