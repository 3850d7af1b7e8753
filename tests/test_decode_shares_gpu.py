"""Decode attention in shares (csrc/flash_decoding.cu): CTAs that take a split with tokens each, or equal shares of all rows, as the
lengths on the device say, against attention in 64 bits.  Tolerance: probabilities and result rounded to 16 bits (2^-10 as a
2-norm bound for fp16, eight times that for bf16)."""

from __future__ import annotations

import math
import random

import pytest
import torch

from test_decode_plan_cpu import SHARES, plan

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(180)]

# one block of kv heads, four, five heads each, two blocks of 64, two warps of query heads to each kv head
HEADS = [(32, 8, 128), (32, 32, 128), (40, 8, 128), (64, 16, 64), (80, 4, 128)]


def lengths(kind: str, batch: int, bound: int) -> list[int]:
    rng = random.Random(batch + bound)
    return {
        "full": [bound] * batch,                                         # equal shares
        "ragged": [rng.randint(1, bound) for _ in range(batch)],
        "fifth": [bound // 5] * batch,
        "few": [max(1, bound // 50)] * batch,                            # a split each
        "one long": [bound] + [17] * (batch - 1),
        "holes": [0 if rng.random() < 0.4 else rng.randint(1, bound) for _ in range(batch)],
        "none": [0] * batch,
    }[kind]


def inputs(batch, bound, heads, kv_heads, d, dtype, layout="pool"):
    rows = batch * bound
    if layout == "pool":
        pool = torch.randn(rows, 2 * kv_heads, d, device="cuda", dtype=dtype)
        k, v = pool[:, :kv_heads], pool[:, kv_heads:]
    elif layout == "two":
        k, v = (torch.randn(rows, kv_heads, d, device="cuda", dtype=dtype) for _ in range(2))
    else:                                                                # a head's key and value side by side: a copy per head
        pool = torch.randn(rows, kv_heads, 2 * d, device="cuda", dtype=dtype)
        k, v = pool[..., :d], pool[..., d:]
    q = torch.randn(batch, heads, d, device="cuda", dtype=dtype)
    table = torch.randperm(rows, device="cuda").int().view(batch, bound)
    return q, k, v, table, torch.randperm(batch, device="cuda")


def run(q, k, v, table, order, lens, bound, wide=False):
    import lite_llama_b200.kernels as K

    index = torch.int64 if wide else torch.int32
    lens = torch.tensor(lens, device="cuda", dtype=index)
    return K.flash_decoding(q, k, v, 1 / math.sqrt(q.shape[2]), table, order.to(index), lens, bound)


def exact(q, k, v, table, order, lens):
    batch, heads, d = q.shape
    want = torch.zeros(batch, heads, d, device="cuda", dtype=torch.float64)
    for b, n in enumerate(lens):
        if n:
            at = table[order[b], :n].long()
            kk, vv = (t[at].double().permute(1, 0, 2).repeat_interleave(heads // k.shape[1], 0) for t in (k, v))
            want[b] = torch.einsum("hn,hnd->hd", (torch.einsum("hd,hnd->hn", q[b].double(), kk) / math.sqrt(d)).softmax(-1), vv)
    return want


def splits_fit(batch, heads, kv_heads, d, bound, lens) -> bool:
    p = plan(batch, heads, kv_heads, d, bound)
    return sum(-(-n // p.tokens) for n in lens) * p.blocks <= p.grid


def check(batch, bound, lens, heads, kv_heads, d, dtype, wide=False, layout="pool", shares=True):
    assert not shares or plan(batch, heads, kv_heads, d, bound).form == SHARES
    data = inputs(batch, bound, heads, kv_heads, d, dtype, layout)
    got = run(*data, lens, bound, wide)
    assert torch.equal(got, run(*data, lens, bound, wide))
    assert all(not got[b].any() for b, n in enumerate(lens) if n == 0)
    if any(lens):
        want = exact(*data, lens)
        assert ((got.double() - want).norm() / want.norm()).item() < (2.0**-10 if dtype is torch.float16 else 2.0**-7)


@pytest.mark.parametrize("heads,kv_heads,d", HEADS)
@pytest.mark.parametrize("kind", ["full", "ragged", "fifth", "few", "one long", "holes", "none"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_shares_of_any_lengths(heads, kv_heads, d, kind, dtype):
    # fewer rows than a warp has lanes, as many, more than the smaller blocks have threads; 13 tiles per SM and more
    for batch, bound in ((8, 8001), (32, 2000), (100, 700), (170, 400)):
        if batch * bound * kv_heads > 1 << 20:
            bound //= 2
        check(batch, bound, lengths(kind, batch, bound), heads, kv_heads, d, dtype, batch == 32, "two" if batch == 100 else "pool")


@pytest.mark.parametrize("heads,kv_heads,d", HEADS[:4])
@pytest.mark.parametrize("kind", ["full", "ragged", "fifth", "few", "one long", "holes", "none"])
def test_lengths_around_the_line_of_the_shares(heads, kv_heads, d, kind):
    for batch, bound in ((8, 4001), (32, 1000), (100, 460), (130, 250)):
        lens = lengths(kind, batch, bound)
        check(batch, bound, lens, heads, kv_heads, d, torch.float16, batch == 32, "two" if batch == 100 else "pool", shares=False)


def test_rows_of_a_single_split_in_bf16():
    check(1024, 33, lengths("ragged", 1024, 33), 32, 8, 128, torch.bfloat16, shares=False)
    check(1024, 65, lengths("holes", 1024, 65), 32, 8, 128, torch.bfloat16, True, shares=False)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind", ["ragged", "holes", "one long", "few"])
def test_shares_of_the_most_rows(kind, dtype):
    # 888 rows of one block of kv heads would be cut into a single split each; a thread owns several rows
    check(887, 200, lengths(kind, 887, 200), 32, 8, 128, dtype, kind == "holes")


@pytest.mark.parametrize("kind", ["ragged", "few"])
@pytest.mark.parametrize("heads,kv_heads,d", HEADS)
def test_shares_of_heads_that_are_not_packed(heads, kv_heads, d, kind):
    check(32, 2000, lengths(kind, 32, 2000), heads, kv_heads, d, torch.float16, layout="per head")


@pytest.mark.parametrize("heads,kv_heads,d", HEADS)
@pytest.mark.parametrize("kind", ["few", "one long"])
def test_rows_do_not_depend_on_the_others_where_the_splits_fit(heads, kv_heads, d, kind):
    """Up to a split per CTA, rows are cut as by the grid of splits (which folds its merge when asked to): the same bits."""
    import lite_llama_b200.kernels.flashdecoding as F

    batch, bound = 32, 2000
    data = inputs(batch, bound, heads, kv_heads, d, torch.float16)
    lens = lengths(kind, batch, bound)[:28] + [0] * 4
    others = [n if b % 3 == 0 else (b * 7) % 48 for b, n in enumerate(lens[:28])] + [0] * 4
    assert splits_fit(batch, heads, kv_heads, d, bound, lens) and splits_fit(batch, heads, kv_heads, d, bound, others)
    got = run(*data, lens, bound)
    assert torch.equal(got[::3], run(*data, others, bound)[::3])
    F._FOLD = True
    try:
        assert torch.equal(got, run(*data, lens, bound))
    finally:
        F._FOLD = False


@pytest.mark.parametrize("heads,kv_heads,d", HEADS)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind", ["full", "few"])
def test_infinite_values_stay_infinite(heads, kv_heads, d, dtype, kind):
    """Every probability is one that 16 bits hold, so an infinite value makes its column infinite, and only infinite values of both
    signs make it NaN; the other columns do not notice."""
    batch, bound = 32, 2000
    q, k, v, table, order = inputs(batch, bound, heads, kv_heads, d, dtype)
    q = q * 0.1
    lens = lengths(kind, batch, bound)
    for b, n in enumerate(lens):
        tokens = table[order[b], torch.randint(0, n - 1, (3,), device="cuda")].long()   # (a last one also stands for those beyond the row)
        v[tokens, b % kv_heads, b % 7] = math.inf
        v[tokens, b % kv_heads, b % 7 + 8] = -math.inf
        if b % 2 and n > 1:
            v[table[order[b], 0].long(), b % kv_heads, b % 7 + 16] = math.inf
            v[table[order[b], n - 1].long(), b % kv_heads, b % 7 + 16] = -math.inf
    assert plan(batch, heads, kv_heads, d, bound).form == SHARES
    got, want = run(q, k, v, table, order, lens, bound), exact(q, k, v, table, order, lens)
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got.isnan(), want.isnan()) and want.isinf().any()
    assert torch.equal(got[got.isinf()].double(), want[want.isinf()])
    ok = want.isfinite()
    assert ((got[ok].double() - want[ok]).norm() / want[ok].norm()).item() < (2.0**-10 if dtype is torch.float16 else 2.0**-7)


@pytest.mark.parametrize("heads,kv_heads,d", HEADS)
def test_a_workspace_for_the_splits_alone_is_enough(heads, kv_heads, d):
    """A caller of the C entry may have sized it for [batch, heads, splits] partial rows and their statistics."""
    from lite_llama_b200 import _lib

    batch, bound = 32, 2000
    q, k, v, table, order = inputs(batch, bound, heads, kv_heads, d, torch.float16)
    lens, order, out = torch.full((batch,), bound, device="cuda").int(), order.int(), torch.empty_like(q)
    p = plan(batch, heads, kv_heads, d, bound)
    nbytes = batch * heads * p.splits * (d + 1) * 4 + 16
    ws = torch.empty(nbytes + 64, dtype=torch.uint8, device="cuda")
    ws[nbytes:] = 7

    def call(size):
        return _lib.load().b2l_flash_decoding(
            out.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), table.data_ptr(), order.data_ptr(), 4, lens.data_ptr(), 4, batch,
            heads, kv_heads, d, bound, d**-0.5, q.stride(0), q.stride(1), k.stride(0), k.stride(1), v.stride(0), v.stride(1),
            table.stride(0), 1, out.stride(0), out.stride(1), ws.data_ptr(), size, None, 0, 0, torch.cuda.current_stream().cuda_stream)

    assert p.form == SHARES and call(nbytes - 1) != 0
    _lib.check(call(nbytes))
    want = exact(q, k, v, table, order, [bound] * batch)
    assert ((out.double() - want).norm() / want.norm()).item() < 2.0**-10
    assert (ws[nbytes:] == 7).all()


def test_a_captured_step_follows_the_lengths():
    """One graph, replayed with lengths whose splits fit the CTAs and with others, in turn: nothing of a replay is left for the next."""
    batch, bound, heads, kv_heads, d = 32, 2000, 32, 8, 128
    data = inputs(batch, bound, heads, kv_heads, d, torch.float16)
    lens = torch.full((batch,), bound, device="cuda").int()
    import lite_llama_b200.kernels as K

    q, k, v, table, order = data
    call = lambda: K.flash_decoding(q, k, v, d**-0.5, table, order.int(), lens, bound)  # noqa: E731
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    for kind in ("full", "few", "ragged", "one long", "none", "holes", "few", "full"):
        want = lengths(kind, batch, bound)
        lens.copy_(torch.tensor(want).int())
        graph.replay()
        assert torch.equal(out, run(*data, want, bound))
