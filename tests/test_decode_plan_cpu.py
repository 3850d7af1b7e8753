"""Split plan of decode attention (csrc/flash_decoding.cu), read off its workspace: a function of sizes alone, no GPU.

Lengths are device data and ``max_actual_seq_len`` is only a bound (a captured graph's bucket, or one long sequence among
short ones), so a row of the longest possible length has to be cut into enough splits whatever the other rows are."""

from __future__ import annotations

import ctypes
from typing import NamedTuple

import pytest

from lite_llama_b200 import _lib


def splits(batch: int, heads: int, kv_heads: int, d: int, longest: int) -> int:
    nbytes = _lib.load().b2l_flash_decoding_workspace_bytes(batch, heads, kv_heads, d, longest)
    return max(1, (nbytes - 16) // (batch * heads * (d + 1) * 4))


# (batch, bucket, longest split in tokens): six CTAs per SM of 148 over the rows' kv-head blocks (one block of 8 heads of
# 128), in tiles of 16 tokens, at least four tiles each
@pytest.mark.parametrize("batch,bucket,longest_split", [
    (1, 4096, 64), (8, 4096, 64), (12, 4096, 64), (32, 2048, 80), (32, 4096, 160), (64, 4096, 304), (128, 4096, 592),
    (256, 4096, 1024),
])
def test_one_long_sequence_is_cut_whatever_the_batch(batch, bucket, longest_split):
    n = splits(batch, 32, 8, 128, bucket)
    assert -(-bucket // n) <= longest_split, (n, bucket)


SPLITS, CLUSTER, SHARES = 0, 1, 2


class Plan(NamedTuple):
    form: int
    splits: int      # per row
    tokens: int      # per split
    grid: int        # CTAs of the shares
    blocks: int      # of kv heads


def plan(batch: int, heads: int, kv_heads: int, d: int, longest: int) -> Plan:
    out = (ctypes.c_int * 5)()
    _lib.check(_lib.load().b2l_flash_decoding_plan(batch, heads, kv_heads, d, longest, out, None))
    return Plan(*out)


# on 148 SMs: 13 tiles of 16 tokens per CTA (six with several blocks of kv heads), with one or two CTAs to an SM by shared memory and
# two splits or more; as many CTAs as fit at once, by registers as well (nine warps of heads of 128: one to an SM)
@pytest.mark.parametrize("batch,heads,kv_heads,d,longest,form,grid", [
    (1, 32, 8, 128, 200, CLUSTER, 0), (1, 32, 8, 128, 2000, SPLITS, 0), (32, 32, 8, 128, 480, SPLITS, 0),
    (32, 32, 8, 128, 1000, SHARES, 148), (887, 32, 8, 128, 200, SHARES, 148), (888, 32, 8, 128, 200, SPLITS, 0),
    (32, 28, 4, 128, 2000, SHARES, 296), (32, 14, 2, 64, 2000, SPLITS, 0), (8, 32, 32, 128, 600, SHARES, 148),
    (64, 16, 8, 256, 2000, SPLITS, 0), (32, 80, 4, 128, 2000, SHARES, 148), (32, 64, 4, 128, 2000, SHARES, 296),
    (16, 80, 4, 128, 2000, SPLITS, 0), (64, 64, 16, 64, 2000, SHARES, 296),
])
def test_form(batch, heads, kv_heads, d, longest, form, grid):
    p = plan(batch, heads, kv_heads, d, longest)
    assert (p.form, p.grid) == (form, grid)


@pytest.mark.parametrize("batch,bucket", [(8, 4096), (32, 2048), (32, 4096), (128, 4096), (256, 4096)])
def test_shares_cut_a_long_row_no_coarser_than_the_splits(batch, bucket):
    """Alone with tokens, a row of the longest length is cut into its splits, a CTA each; where those are more than the CTAs it is
    cut into a share per CTA."""
    p = plan(batch, 32, 8, 128, bucket)
    assert p.form == SHARES and p.splits == splits(batch, 32, 8, 128, bucket) and p.splits * p.tokens >= bucket
    assert p.splits * p.blocks <= p.grid or -(-bucket // p.grid) <= p.tokens
