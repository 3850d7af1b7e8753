"""Weights that a projection converts or copies on the way to its kernel.  The kernels request weights before the previous
kernel has finished, so the shim has to enqueue ``b2l_weights_written`` between such a copy and the GEMM, and only then."""

from __future__ import annotations

import pytest
import torch

N, K_DIM = 128, 256


def tensors(device: str):
    g = torch.Generator().manual_seed(3)
    x = torch.randn(5, K_DIM, generator=g).half()
    q4 = torch.randint(-2**31, 2**31 - 1, (N, K_DIM // 8), generator=g, dtype=torch.int64).int()
    s4 = torch.rand(N, K_DIM // 128, generator=g).half().float()
    z4 = torch.randint(0, 16, (N, K_DIM // 128), generator=g).float()
    q8 = torch.randint(-127, 128, (N, K_DIM), generator=g, dtype=torch.int8)
    s8 = torch.rand(N, 1, generator=g).half().float()
    w = torch.randn(N, K_DIM, generator=g).half()
    return [t.to(device) for t in (x, q4, s4, z4, q8, s8, w)]


def strided(t: torch.Tensor) -> torch.Tensor:
    """The same values with a last stride of 2."""
    return t.repeat_interleave(2, -1)[..., ::2]


def variants(device: str):
    """name -> (call on tensors as the kernel takes them, the same call on tensors that need a conversion or copy)"""
    import lite_llama_b200.kernels as K

    x, q4, s4, z4, q8, s8, w = tensors(device)
    w4 = lambda *a: (lambda: K.w4a16_matmul(x, *a))                                     # noqa: E731
    return {
        "w4a16_tables_fp16": (w4(q4, s4, z4), w4(q4, s4.half(), z4.half())),
        "w4a16_zeros_fp16": (w4(q4, s4, z4), w4(q4, s4, z4.half())),
        "w4a16_zeros_transposed": (w4(q4, s4, z4), w4(q4, s4, z4.t().contiguous().t())),
        "w4a16_qweight_strided": (w4(q4, s4, z4), w4(strided(q4), s4, z4)),
        "w8a16_scales_fp16": (lambda: K.w8a16_matmul(x, q8, s8, group_n=1, group_k=K_DIM),
                              lambda: K.w8a16_matmul(x, q8, s8.half(), group_n=1, group_k=K_DIM)),
        "w8a8_qweight_strided": (lambda: K.smoothquant_matmul(x, q8, s8), lambda: K.smoothquant_matmul(x, strided(q8), s8)),
        "linear_weight_strided": (lambda: K.linear(x, w), lambda: K.linear(x, strided(w))),
    }


NAMES = ["w4a16_tables_fp16", "w4a16_zeros_fp16", "w4a16_zeros_transposed", "w4a16_qweight_strided", "w8a16_scales_fp16",
         "w8a8_qweight_strided", "linear_weight_strided"]
GEMMS = {"b2l_linear", "b2l_w8a8_gemm", "b2l_w4a16_matmul", "b2l_w8a16_matmul"}


class Recorder:
    """Stands in for the library: remembers the names of the calls."""

    def __init__(self) -> None:
        self.calls: list[str] = []

    def __getattr__(self, name):
        def call(*_args):
            self.calls.append(name)
            return 0
        return call


@pytest.mark.parametrize("name", NAMES)
def test_the_order_is_kept_exactly_where_a_copy_was_made(name, monkeypatch):
    from lite_llama_b200.kernels import _common, linear as _  # noqa: F401
    import sys

    rec = Recorder()
    mods = [sys.modules["lite_llama_b200.kernels." + m] for m in
            ("_common", "linear", "quantization.w4a16", "quantization.w8a16", "quantization.w8a8")]
    fakes = {"lib": lambda: rec, "check": lambda rc: None, "require_cuda": lambda *t: None, "stream_handle": lambda: 0,
             "counters": lambda d: torch.zeros(1, dtype=torch.int32), "workspace": lambda n, d: None,
             "zeroed_workspace": lambda n, d: None, "current_device": lambda: 0, "quant_gemm_workspace_bytes": lambda *a: 0}
    for m in mods:
        for attr, fake in fakes.items():
            if hasattr(m, attr):
                monkeypatch.setattr(m, attr, fake)
    plain, converted = variants("cpu")[name]
    plain()
    assert "b2l_weights_written" not in rec.calls
    rec.calls.clear()
    converted()
    order = [c for c in rec.calls if c in GEMMS | {"b2l_weights_written"}]
    assert order[0] == "b2l_weights_written" and order[1] in GEMMS and len(order) == 2, order


@pytest.mark.gpu
@pytest.mark.timeout(180)
@pytest.mark.parametrize("name", NAMES)
def test_converted_weights_back_to_back(name):
    plain, converted = variants("cuda")[name]
    want = plain()
    got = [converted() for _ in range(50)]                  # every call converts again, into recycled memory
    assert all(torch.equal(y, want) for y in got)
