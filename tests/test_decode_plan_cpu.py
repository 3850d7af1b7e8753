"""Split plan of decode attention (csrc/flash_decoding.cu), read off its workspace: a function of sizes alone, no GPU.

Lengths are device data and ``max_actual_seq_len`` is only a bound (a captured graph's bucket, or one long sequence among
short ones), so a row of the longest possible length has to be cut into enough splits whatever the other rows are."""

from __future__ import annotations

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
