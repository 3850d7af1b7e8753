"""Prompt attention with two query tiles per CTA (csrc/flash_attention_tc.cu) against 64 bits: lengths around the 128-token
blocks, sequences of no, one and many blocks, more sequences than a warp has lanes, even groups (two heads per CTA) and odd ones
(two blocks of a head, the second of which may be missing).  Tolerance: probabilities and results are rounded to 16 bits
(2^-12 and 2^-9 each as 2-norm bounds)."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(180)]

LENGTHS = [[700, 129, 0, 128, 257, 1, 640, 383], [1100], [256] * 5, [130 + 7 * i for i in range(40)], [2000, 3]]


def K():
    import lite_llama_b200.kernels as k

    return k


@pytest.mark.parametrize("lens", LENGTHS)
@pytest.mark.parametrize("hq,hk", [(32, 8), (28, 4), (24, 24), (10, 2)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_two_tiles_per_cta(lens, hq, hk, dtype):
    d, total, longest = 128, sum(lens), max(lens)
    if -(-longest // 128) * hq * len(lens) <= 148:
        pytest.skip("few blocks stay with one tile per CTA")
    qkv = torch.randn(total, (hq + 2 * hk) * d, device="cuda", dtype=dtype)
    q, k, v = (t.unflatten(1, (-1, d)) for t in qkv.split([hq * d, hk * d, hk * d], 1))
    index = torch.int64 if hk == 4 else torch.int32
    n = torch.tensor(lens, device="cuda", dtype=index)
    start = (n.cumsum(0) - n).to(index)
    scale = 1.0 / math.sqrt(d)
    got = K().flash_attention2_no_pad(q, k, v, scale * math.log2(math.e), start, n, longest)
    assert torch.equal(K().flash_attention2_no_pad(q, k, v, scale * math.log2(math.e), start, n, longest), got)
    diff = norm = 0.0
    for i, m in enumerate(lens[:12]):
        if m == 0:
            continue
        a = int(start[i])
        qi, ki, vi = (t[a : a + m].double().transpose(0, 1) for t in (q, k, v))
        s = (qi.view(hk, -1, m, d) @ ki.transpose(1, 2)[:, None] * scale).masked_fill(
            torch.ones(m, m, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
        want = (s.softmax(-1) @ vi[:, None]).reshape(hq, m, d).transpose(0, 1)
        diff += (got[a : a + m].double() - want).square().sum().item()
        norm += want.square().sum().item()
    assert math.sqrt(diff / norm) < (2.0**-11 if dtype == torch.float16 else 2.0**-8)


@pytest.mark.parametrize("lens", [[200], [0, 300, 0, 129], [40 + i for i in range(70)]])
@pytest.mark.parametrize("hq,hk", [(16, 2), (9, 3)])
def test_a_bound_far_above_the_lengths(lens, hq, hk):
    """The bound decides how many blocks there might be, not what comes out: the same bits as with the next larger bound whose
    grid is as large, in about the same time."""
    q = torch.randn(sum(lens), hq, 128, device="cuda", dtype=torch.float16)
    k, v = torch.randn(2, sum(lens), hk, 128, device="cuda", dtype=torch.float16)
    n = torch.tensor(lens, device="cuda", dtype=torch.int32)
    start = (n.cumsum(0) - n).int()
    call = lambda bound: K().flash_attention2_no_pad(q, k, v, 0.1275, start, n, bound)                      # noqa: E731
    near = -(-150 // (hq * len(lens))) * 128 + 256
    got, want = call(32768), call(near)
    assert got.isfinite().all() and torch.equal(got, want)

    def time(bound):
        graph, a, b = torch.cuda.CUDAGraph(), *(torch.cuda.Event(enable_timing=True) for _ in range(2))
        with torch.cuda.graph(graph):
            for _ in range(20):
                call(bound)
        best = float("inf")
        for _ in range(5):
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert time(32768) < 2 * time(near)                 # the scheduler of every CTA walked through all levels: up to 6 times


def test_large_scores_rescale_the_sums():
    """Scores that grow along the keys by far more than the 2^8 that the running maximum may lag behind, and a row of one size."""
    d, m, h = 128, 900, 24
    q = torch.zeros(m, h, d, device="cuda", dtype=torch.float16)
    k, v = torch.zeros_like(q), torch.randn(m, h, d, device="cuda", dtype=torch.float16)
    q[:, :, 0], k[:, :, 0] = 8.0, torch.linspace(-30, 30, m, device="cuda")[:, None]
    q[5] = 0.0
    n, start = torch.tensor([m], device="cuda"), torch.zeros(1, device="cuda", dtype=torch.int64)
    got = K().flash_attention2_no_pad(q, k, v, math.log2(math.e), start, n, m).double()
    s = (q.double().transpose(0, 1) @ k.double().permute(1, 2, 0)).masked_fill(
        torch.ones(m, m, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    want = (s.softmax(-1) @ v.double().transpose(0, 1)).transpose(0, 1)
    assert ((got - want).norm() / want.norm()).item() < 2.0**-10
