"""The CTA-pair GEMMs of prompt-sized batches (csrc/gemm_pair.cu) against a 64-bit product, at the edges of their tiles:
token counts around the 256-row tile, output counts that end inside a 64-wide store box, a K tail, one tile per pair and
several.  Tolerance: one rounding of the result to 16 bits (2^-9 relative for bf16, 2^-12 for fp16 as a 2-norm bound) on
top of fp32 accumulation, which is orders of magnitude below it."""

from __future__ import annotations

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(180)]

REL = {torch.float16: 2.0**-11, torch.bfloat16: 2.0**-8}


def K():
    import lite_llama_b200.kernels as k

    return k


def rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


# 129 tokens x 10240 outputs: the fewest tokens and (40 wide tiles of 256) about the fewest tiles the pair kernel takes
EDGES = [(129, 10240, 192), (256, 10248, 64), (257, 5128, 392), (511, 5112, 1000), (1000, 4096, 520), (2049, 4104, 256)]


@pytest.mark.parametrize("m,n,k", EDGES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bias", [False, True])
def test_linear_pair_tiles(m, n, k, dtype, bias):
    x = torch.randn(m, k, device="cuda", dtype=dtype)
    w = torch.randn(n, k, device="cuda", dtype=dtype)
    b = torch.randn(n, device="cuda", dtype=dtype) if bias else None
    want = x.double() @ w.double().T + (b.double() if bias else 0.0)
    assert rel(K().linear(x, w, b), want) < REL[dtype]


@pytest.mark.parametrize("m,n,k", [(129, 10240, 192), (256, 10248, 64), (511, 5112, 1008), (2049, 4104, 256)])
@pytest.mark.parametrize("bias", [False, True])
def test_int8_pair_tiles(m, n, k, bias):
    qa = torch.randint(-127, 128, (m, k), device="cuda", dtype=torch.int8)
    qw = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
    sa, sw = torch.rand(m, device="cuda") * 1e-2, torch.rand(n, device="cuda") * 1e-2
    b = torch.randn(n, device="cuda") if bias else None
    want = (qa.double() @ qw.double().T) * sa.double()[:, None] * sw.double() + (b.double() if bias else 0.0)
    assert rel(K().smoothquant_matmul_prequant(qa, sa, qw, sw, bias=b), want) < REL[torch.float16]


def test_linear_forms_the_pair_kernel_does_not_take():
    """Output counts that are no multiple of 8 stay on the one-SM kernel; strided activations and weights go either way."""
    x = torch.randn(600, 512, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(10250, 512, device="cuda", dtype=torch.bfloat16)
    assert rel(K().linear(x, w), x.double() @ w.double().T) < REL[torch.bfloat16]
    xs, ws = x[:, 64:320], w[:10240, 128:384]
    assert rel(K().linear(xs, ws), xs.double() @ ws.double().T) < REL[torch.bfloat16]
