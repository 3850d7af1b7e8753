"""Dispatch of the dense and int8 projections (csrc/gemm_dense.cu), a function of sizes alone: no GPU, 148 SMs."""

from __future__ import annotations

import ctypes
from typing import NamedTuple

import pytest

from lite_llama_b200 import _lib


class Plan(NamedTuple):
    pairs: bool      # SM pairs instead of the one-SM kernel, whose plan the rest is
    tokens: int      # per tile
    parts: int       # of k
    blocks: int      # of 64 k (16 bits) or 128 k (int8) per part
    accumulate: int  # blocks per accumulation


def plan(m: int, n: int, k: int, elem_bytes: int) -> Plan:
    out = (ctypes.c_int * 5)()
    _lib.check(_lib.load().b2l_linear_plan(m, n, k, elem_bytes, out, None))
    return Plan(bool(out[0]), *out[1:])


@pytest.mark.parametrize("m,n,k,elem_bytes,tokens,pairs", [
    # 65 - 128 tokens: a second wave of the smaller tile ...
    (65, 9728, 896, 2, 128, False), (128, 18944, 192, 2, 128, False), (100, 9600, 320, 2, 128, False), (100, 14336, 448, 1, 128, False),
    # ... unless several of them share an SM over so short a k
    (65, 9728, 128, 2, 64, False), (100, 14336, 192, 2, 64, False), (65, 9728, 256, 1, 64, False), (128, 12288, 128, 1, 64, False),
    # more tokens and a short k: as many tiles as there are SMs, and the pairs where that is more than one wave
    (257, 4864, 128, 2, 64, False), (400, 4864, 256, 2, 128, True), (700, 5120, 256, 1, 128, True),
    (300, 5120, 256, 1, 64, False), (513, 2304, 448, 2, 64, True),
])
def test_token_tiles(m, n, k, elem_bytes, tokens, pairs):
    p = plan(m, n, k, elem_bytes)
    assert (p.tokens, p.pairs) == (tokens, pairs)


@pytest.mark.parametrize("m,n,k", [(64, 896, 4864), (33, 512, 8192), (17, 896, 4864), (48, 1000, 2104), (16, 240, 10160), (64, 64, 4096)])
def test_fewer_parts_of_k_accumulate_as_before(m, n, k):
    """Where k is cut in fewer parts than SMs and blocks would allow for, an accumulation is as long as those parts."""
    p, blocks = plan(m, n, k, 2), -(-k // 64)
    most = min(148 // -(-n // 128), blocks // 4, 32)
    assert p.parts < most and p.accumulate == -(-blocks // most) and p.blocks % p.accumulate == 0


@pytest.mark.parametrize("m,n,k,elem_bytes", [(64, 896, 4864, 1), (64, 3584, 3584, 2), (16, 128, 4096, 2), (128, 4096, 4096, 2)])
def test_one_accumulation_per_part_elsewhere(m, n, k, elem_bytes):
    p = plan(m, n, k, elem_bytes)
    assert p.accumulate == p.blocks
