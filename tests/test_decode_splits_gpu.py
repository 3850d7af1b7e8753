"""Decode attention at the edges of its split rule (csrc/flash_decoding.cu): one split, the plain merge (up to 8), the merge
of many (9, more than a warp's 32), rows of 512 bytes and of 4 KB, against attention in 64 bits.  Tolerance: probabilities and
result rounded to 16 bits (2^-10 as a 2-norm bound for fp16)."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(180)]


@pytest.mark.parametrize("batch,context", [(1, 60), (1, 520), (1, 580), (1, 2100), (3, 5000), (32, 700), (98, 130), (99, 130), (300, 90)])
@pytest.mark.parametrize("heads,kv_heads,d", [(32, 8, 128), (14, 2, 64)])
def test_split_counts(batch, context, heads, kv_heads, d):
    import lite_llama_b200.kernels as K

    lens = [context - (i * (context - context // 2)) // batch for i in range(batch)]
    pool = torch.randn(batch * context, 2 * kv_heads, d, device="cuda", dtype=torch.float16)
    q = torch.randn(batch, heads, d, device="cuda", dtype=torch.float16)
    table = torch.arange(batch * context, device="cuda", dtype=torch.int32).view(batch, context)
    rows = torch.arange(batch, device="cuda", dtype=torch.int32)
    got = K.flash_decoding(q, pool[:, :kv_heads], pool[:, kv_heads:], 1 / math.sqrt(d), table, rows,
                           torch.tensor(lens, device="cuda", dtype=torch.int32), context)
    kv = pool.view(batch, context, 2, kv_heads, d).double()
    k, v = (t.permute(0, 2, 1, 3).repeat_interleave(heads // kv_heads, 1) for t in (kv[:, :, 0], kv[:, :, 1]))
    s = (q.double()[:, :, None] * k).sum(-1) / math.sqrt(d)
    dead = torch.arange(context, device="cuda")[None] >= torch.tensor(lens, device="cuda")[:, None]
    want = (s.masked_fill(dead[:, None], float("-inf")).softmax(-1)[..., None] * v).sum(2)
    assert ((got.double() - want).norm() / want.norm()).item() < 2.0**-10
