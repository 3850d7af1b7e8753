"""Decode attention in shares (csrc/flash_decoding.cu): CTAs that take items of one row or equal shares of all rows, as the
lengths on the device say, against attention in 64 bits.  Tolerance: probabilities and result rounded to 16 bits (2^-10 as a
2-norm bound for fp16, eight times that for bf16)."""

from __future__ import annotations

import math
import random

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(180)]

HEADS = [(32, 8, 128), (32, 32, 128), (40, 8, 128), (64, 16, 64)]       # one block of kv heads, four, five heads each, two of 64


def lengths(kind: str, batch: int, bound: int) -> list[int]:
    rng = random.Random(batch + bound)
    return {
        "full": [bound] * batch,                                         # equal shares
        "ragged": [rng.randint(1, bound) for _ in range(batch)],
        "fifth": [bound // 5] * batch,                                   # items of four tiles or more
        "few": [max(1, bound // 50)] * batch,                            # items of two tiles
        "one long": [bound] + [17] * (batch - 1),
        "holes": [0 if rng.random() < 0.4 else rng.randint(1, bound) for _ in range(batch)],
        "none": [0] * batch,
    }[kind]


def check(batch, bound, lens, heads, kv_heads, d, dtype, wide, split_pools):
    import lite_llama_b200.kernels as K

    index = torch.int64 if wide else torch.int32
    rows = batch * bound
    if split_pools:
        k, v = (torch.randn(rows, kv_heads, d, device="cuda", dtype=dtype) for _ in range(2))
    else:
        pool = torch.randn(rows, 2 * kv_heads, d, device="cuda", dtype=dtype)
        k, v = pool[:, :kv_heads], pool[:, kv_heads:]
    q = torch.randn(batch, heads, d, device="cuda", dtype=dtype)
    table = torch.randperm(rows, device="cuda").int().view(batch, bound)
    order = torch.randperm(batch, device="cuda")
    got = K.flash_decoding(q, k, v, 1 / math.sqrt(d), table, order.to(index), torch.tensor(lens, device="cuda", dtype=index), bound)
    want = torch.zeros(batch, heads, d, device="cuda", dtype=torch.float64)
    for b, n in enumerate(lens):
        if n:
            at = table[order[b], :n].long()
            kk, vv = (t[at].double().permute(1, 0, 2).repeat_interleave(heads // kv_heads, 0) for t in (k, v))
            want[b] = torch.einsum("hn,hnd->hd", (torch.einsum("hd,hnd->hn", q[b].double(), kk) / math.sqrt(d)).softmax(-1), vv)
    if not any(lens):
        assert not got.any()
        return
    assert all(not got[b].any() for b, n in enumerate(lens) if n == 0)
    assert ((got.double() - want).norm() / want.norm()).item() < (2.0**-10 if dtype is torch.float16 else 2.0**-7)


@pytest.mark.parametrize("heads,kv_heads,d", HEADS)
@pytest.mark.parametrize("kind", ["full", "ragged", "fifth", "few", "one long", "holes", "none"])
def test_shares_of_any_lengths(heads, kv_heads, d, kind):
    # rows handled by a lane each, by four lanes' worth, by threads; 13 tiles per SM and more
    for batch, bound in ((8, 4001), (32, 1000), (100, 460), (130, 250)):
        check(batch, bound, lengths(kind, batch, bound), heads, kv_heads, d, torch.float16, batch == 32, batch == 100)


def test_shares_in_bf16_at_the_most_rows():
    check(1024, 33, lengths("ragged", 1024, 33), 32, 8, 128, torch.bfloat16, False, False)
    check(1024, 65, lengths("holes", 1024, 65), 32, 8, 128, torch.bfloat16, True, False)
