"""W4A16 projections of up to 8 tokens (csrc/gemm_quant_decode.cu) against a 64-bit product: fewer strips than SMs, several
chunks of strips per CTA, a last strip past N, warps with no, one and several slices of k, groups of 128 and 512, biases.
Tolerance: one rounding to fp16 (2^-11 as a 2-norm bound) on top of fp32 accumulation."""

from __future__ import annotations

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(180)]


def K():
    import lite_llama_b200.kernels as k

    return k


def case(m, n, k, group):
    q = torch.randint(-(2**31), 2**31 - 1, (n, k // 8), device="cuda", dtype=torch.int64).to(torch.int32)
    s = torch.rand(n, k // group, device="cuda") * 4e-3 + 1e-3
    z = torch.randint(0, 16, (n, k // group), device="cuda").float()
    codes = torch.stack([(q >> (4 * j)) & 15 for j in range(8)], -1).view(n, k // group, group).double()
    w = ((codes - z.double()[..., None]) * s.double()[..., None]).view(n, k)
    return q, s, z, w, torch.randn(m, k, device="cuda", dtype=torch.float16)


@pytest.mark.parametrize("m", [1, 7, 8])
@pytest.mark.parametrize("n,k,group", [(16, 256, 128), (130, 512, 128), (4104, 4096, 128), (20000, 1024, 512), (2360, 14336, 128)])
@pytest.mark.parametrize("bias", [None, torch.float16, torch.float32])
def test_int4_decode(m, n, k, group, bias):
    q, s, z, w, x = case(m, n, k, group)
    b = None if bias is None else torch.randn(n, device="cuda", dtype=bias)
    got = K().w4a16_matmul_packed(x, K().w4a16_pack(q, s, z, group_size=group), bias=b).double()
    want = x.double() @ w.T + (0.0 if b is None else b.double())
    assert ((got - want).norm() / want.norm()).item() < 2.0**-11
    assert torch.equal(got, K().w4a16_matmul(x, q, s, z, group_size=group, bias=b).double())      # same products, same order


@pytest.mark.parametrize("m,n,k", [(1, 130, 512), (8, 4104, 4096)])
def test_int4_decode_zero_points_that_are_not_whole(m, n, k):
    """One fractional zero point per row at random groups, and one beyond what the conversion can hold."""
    q, s, z, _, x = case(m, n, k, 128)
    z[torch.arange(n), torch.randint(0, k // 128, (n,))] += 0.37
    z[5, 1] = 1500.0
    codes = torch.stack([(q >> (4 * j)) & 15 for j in range(8)], -1).view(n, k // 128, 128).double()
    want = x.double() @ ((codes - z.double()[..., None]) * s.double()[..., None]).view(n, k).T
    for got in (K().w4a16_matmul(x, q, s, z, group_size=128), K().w4a16_matmul_packed(x, K().w4a16_pack(q, s, z, group_size=128))):
        assert ((got.double() - want).norm() / want.norm()).item() < 2.0**-11


@pytest.mark.parametrize("m,n,k", [(1, 32, 256), (5, 2600, 4096), (8, 28672, 4096), (3, 30, 8192)])
def test_int4_decode_swiglu_is_gemm_then_swiglu(m, n, k):
    from lite_llama_b200.kernels.quantization import interleave_gate_up

    q, s, z, _, x = case(m, n, k, 128)
    wide = K().w4a16_matmul_packed(x, K().w4a16_pack(q, s, z, group_size=128))
    want = K().swiglu_forward(wide[:, : n // 2], wide[:, n // 2 :])
    packed = K().w4a16_pack(interleave_gate_up(q), interleave_gate_up(s), interleave_gate_up(z), group_size=128)
    for _ in range(3):          # back to back: the next launch fetches its weights while this one runs
        got = K().w4a16_matmul_packed(x, packed, swiglu=True)
        assert torch.equal(got, want)
