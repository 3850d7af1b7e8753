"""One-row activations that are views: a row of a wider matrix, a transposed column.  Their row stride is arbitrary (PyTorch
ignores it, ``contiguous`` keeps it), so what reaches a kernel has to carry the stride of the row itself.  Every result is the
one of a plain copy, bit for bit."""

from __future__ import annotations

import pytest
import torch

K_DIM, WIDE = 256, 259                    # 259: no multiple of 8 elements


def row_of_wide(device: str, k: int = K_DIM) -> torch.Tensor:
    g = torch.Generator().manual_seed(5)
    return torch.randn(4, k + WIDE - K_DIM, generator=g).half().to(device)[:1, :k]


def transposed_column(device: str, k: int = K_DIM) -> torch.Tensor:
    g = torch.Generator().manual_seed(6)
    return torch.randn(k, 1, generator=g).half().to(device).t()


VIEWS = [row_of_wide, transposed_column]


@pytest.mark.parametrize("view", VIEWS)
def test_a_single_row_gets_its_own_length_as_stride(view):
    from lite_llama_b200.kernels._common import as_rows, own_rows

    x = view("cpu")
    assert x.is_contiguous() and x.stride(0) != K_DIM           # so contiguous() alone changes nothing
    a = own_rows(as_rows(x))
    assert a.stride() == x.reshape(-1, K_DIM).stride() == (K_DIM, 1) and a.data_ptr() == x.data_ptr()


def test_as_rows_passes_matrices_through():
    from lite_llama_b200.kernels._common import as_rows, own_rows

    for t in (torch.zeros(4, 64), torch.zeros(4, 67)[:, :64], torch.zeros(1, 64)):
        assert as_rows(t) is t
    assert as_rows(torch.zeros(2, 3, 64)).shape == (6, 64) and as_rows(torch.zeros(64)).shape == (1, 64)
    assert as_rows(torch.zeros(0, 64)).shape == (0, 64)
    assert own_rows(torch.zeros(4, 67)[:, :64]).stride() == (64, 1) and own_rows(torch.zeros(0, 64)).shape == (0, 64)


def calls():
    import lite_llama_b200.kernels as K

    torch.manual_seed(0)
    n, k = 384, K_DIM
    w = torch.randn(n, k, device="cuda", dtype=torch.float16)
    q4 = torch.randint(-2**31, 2**31 - 1, (n, k // 8), device="cuda", dtype=torch.int64).int()
    s4, z4 = torch.rand(n, k // 128, device="cuda"), torch.randint(0, 16, (n, k // 128), device="cuda").float()
    packed = K.w4a16_pack(q4, s4, z4)
    q8 = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
    s8 = torch.rand(n, 1, device="cuda")
    norm = torch.randn(k, device="cuda", dtype=torch.float16)
    return {
        "linear": lambda x: K.linear(x, w),
        "w4a16_matmul": lambda x: K.w4a16_matmul(x, q4, s4, z4),
        "w4a16_matmul_packed": lambda x: K.w4a16_matmul_packed(x, packed),
        "w8a16_matmul": lambda x: K.w8a16_matmul(x, q8, s8, group_n=1, group_k=k),
        "smoothquant_matmul": lambda x: K.smoothquant_matmul(x, q8, s8),
        "swiglu_forward": lambda x: K.swiglu_forward(x, x),
        "skip_rmsnorm": lambda x: K.skip_rmsnorm(x, None, norm)[0],
        "skip_rmsnorm_residual": lambda x: K.skip_rmsnorm(x.clone(), x, norm)[0],
    }


@pytest.mark.gpu
@pytest.mark.timeout(180)
@pytest.mark.parametrize("view", VIEWS)
@pytest.mark.parametrize("name", ["linear", "w4a16_matmul", "w4a16_matmul_packed", "w8a16_matmul", "smoothquant_matmul",
                                  "swiglu_forward", "skip_rmsnorm", "skip_rmsnorm_residual"])
def test_one_row_views(name, view):
    call = calls()[name]
    x = view("cuda")
    want = call(torch.empty(1, K_DIM, device="cuda", dtype=torch.float16).copy_(x))
    got = call(x)
    assert got.shape == want.shape and torch.equal(got, want)
