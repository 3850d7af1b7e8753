"""Which kernel takes a quantised GEMM (csrc/gemm_quant.cu), a function of sizes alone: no GPU, 148 SMs."""

from __future__ import annotations

import ctypes

import pytest

from lite_llama_b200 import _lib

INT4, FP8, INT8 = 0, 1, 2
STREAMING, DECODE, BATCH, PAIRS, WIDE = range(5)

# 256 tokens per tile with int4 weights in groups of 128 and of 384 (where they divide k) and with one 8-bit scale per row: whole waves of
# 74 pairs, a last tile of one half between tiles of two (the accumulators' turn shifts by an odd number of segments), a last wave cut
# in two with full and with short second parts, rows of y that no 8-byte store fits, an odd number of steps, two tokens in a half
WIDE_TILES = [(385, 18944, 3456), (257, 9470, 3456), (1537, 9470, 3456), (1153, 19200, 1408), (2000, 9734, 1920), (130, 18942, 3456)]

# (m, n, k): pairs that share a tile, with int4 and 8-bit weights in groups of 128 and with one scale per row; the last part shorter, a k
# that no four parts of whole int4 blocks share, tokens that end within the four a thread stores, a tile of one half (64 tokens) or less
SHARED_TILES = {(65, 2560, 2176): (3, 4), (65, 2560, 2560): 4, (129, 1302, 4864): 4, (67, 256, 16384): 4, (100, 5376, 2432): 3, (128, 4096, 14336): 3,
                (200, 4096, 3200): 2, (257, 2600, 3328): 2, (500, 1730, 3200): 2, (256, 4096, 4096): 2}


def form(kind: int, m: int, n: int, k: int, group_k: int, swiglu: bool = False) -> tuple[int, int]:
    """Kernel, and pairs of SMs that share a tile."""
    out = (ctypes.c_int * 2)()
    _lib.check(_lib.load().b2l_quant_gemm_form(kind, m, n, k, group_k, int(swiglu), out, None))
    return out[0], out[1]


@pytest.mark.parametrize("m,n,k", WIDE_TILES)
def test_wide_tiles(m, n, k):
    assert form(INT4, m, n, k, 128) == form(INT4, m, n, k, 128, True) == (WIDE, 1)
    assert form(FP8, m, n, k, k) == form(INT8, m, n, k, k) == (WIDE, 1)
    if k % 384 == 0:
        assert form(INT4, m, n, k, 384) == (WIDE, 1)
    assert form(FP8, m, n, k, 128) == (PAIRS, 1)


@pytest.mark.parametrize("m,n,k", SHARED_TILES)
def test_shared_tiles(m, n, k):
    pairs = SHARED_TILES[m, n, k]
    int4, pairs = pairs if isinstance(pairs, tuple) else (pairs, pairs)
    for swiglu in (False, True):
        assert form(INT4, m, n, k, 128, swiglu) == form(INT4, m, n, k, k, swiglu) == (PAIRS, int4)
    assert form(FP8, m, n, k, 128) == form(FP8, m, n, k, k) == form(INT8, m, n, k, k) == (PAIRS, pairs)


@pytest.mark.parametrize("kind,m,n,k,group,swiglu,kernel", [
    (INT4, 8, 4096, 4096, 128, False, DECODE), (INT4, 64, 4096, 4096, 128, False, BATCH), (FP8, 33, 4096, 4096, 128, False, BATCH),
    (INT4, 72, 4096, 14336, 192, False, STREAMING), (INT4, 72, 12800, 4096, 128, False, PAIRS),
    # one weight tile: half of a pair is padding
    (INT4, 2821, 128, 8192, 128, False, STREAMING), (FP8, 2821, 64, 8192, 128, False, STREAMING), (INT4, 2000, 128, 8192, 128, False, PAIRS),
    # a short k, whose end of a tile nothing covers, and fewer waves in all
    (INT4, 1024, 9728, 896, 128, False, PAIRS), (INT4, 1024, 9728, 896, 128, True, WIDE), (INT4, 1081, 2776, 384, 128, False, PAIRS),
    (FP8, 1410, 2088, 576, 576, False, PAIRS), (INT8, 463, 24408, 256, 256, False, PAIRS), (INT4, 1146, 20984, 256, 128, False, PAIRS),
    (INT4, 1664, 4096, 14336, 128, False, PAIRS), (INT4, 1024, 4096, 14336, 128, False, WIDE), (INT4, 4096, 28672, 4096, 128, False, WIDE),
    (INT8, 2048, 28672, 4096, 4096, False, WIDE), (FP8, 2048, 28672, 4096, 128, False, PAIRS), (FP8, 1664, 4096, 14336, 128, False, PAIRS),
])
def test_kernel(kind, m, n, k, group, swiglu, kernel):
    assert form(kind, m, n, k, group, swiglu)[0] == kernel


@pytest.mark.parametrize("rows,group,tile", [(32, 128, 64), (48, 128, 64), (49, 128, 128), (32, 256, 64), (33, 256, 128), (33, 4096, 128)])
def test_rows_of_an_expert_tile(rows, group, tile):
    from lite_llama_b200.kernels.fused_moe import _pair_tile

    assert _pair_tile(rows * 16, 16, group) == tile
