"""Rotation and cache write in 16-byte units against the form for any even stride: rows that start off a 16-byte boundary, head
dims with and without whole units per half, both index widths.  The same bits, and nothing written beside the rows."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("batch,seq,hq,hkv,d", [(1, 1, 32, 8, 128), (3, 7, 5, 1, 48), (2, 1, 40, 8, 256), (1, 3, 3, 3, 24),
                                                (129, 1, 2, 1, 16)])
def test_aligned_and_unaligned_rows_agree(batch, seq, hq, hkv, d, dtype):
    import lite_llama_b200.kernels as K

    n, heads = batch * seq, hq + 2 * hkv
    qkv = torch.randn(n, heads * d, device="cuda", dtype=dtype)
    cos, sin = torch.randn(2, batch, seq, d, device="cuda", dtype=dtype)
    rows = torch.randperm(3 * n, device="cuda")[:n]
    results = []
    for pad, width in ((0, torch.int64), (2, torch.int32), (8, torch.int32)):        # 2: every row off the boundary
        buf = torch.full((n * (heads * d + pad) + pad,), 7.0, device="cuda", dtype=dtype)
        at = buf[pad:].view(n, heads * d + pad)[:, : heads * d]
        at.copy_(qkv)
        pool = torch.full((3 * n, 2 * hkv, d), -3.0, device="cuda", dtype=dtype)
        q, k, v = (t.unflatten(1, (-1, d)) for t in at.split([hq * d, hkv * d, hkv * d], 1))
        K.rope_kv_write(q, k, v, cos, sin, rows.to(width), pool, batch, seq)
        assert (buf[:pad] == 7).all() and (pad == 0 or (buf[pad:].view(n, -1)[:, heads * d:] == 7).all())
        results.append((at.clone(), pool))
    for got in results[1:]:
        assert torch.equal(got[0], results[0][0]) and torch.equal(got[1], results[0][1])
    at, pool = results[0]
    assert torch.equal(pool[rows].flatten(1), at[:, hq * d:])                        # rotated keys, then values as they came
    assert torch.equal(at[:, (hq + hkv) * d:], qkv[:, (hq + hkv) * d:])
    untouched = torch.ones(3 * n, dtype=torch.bool, device="cuda")
    untouched[rows] = False
    assert (pool[untouched] == -3).all()
    x = qkv[:, :hq * d].double().view(n, hq, d)
    c, s = (t.view(n, 1, d)[..., : d // 2].double() for t in (cos, sin))
    a, b = x.chunk(2, -1)
    want = torch.cat([a * c - b * s, b * c + a * s], -1).flatten(1)
    # two roundings to the activation type per element, each of a value below |a c| + |b s|
    bound = 2 * torch.finfo(dtype).eps * torch.cat([(a * c).abs() + (b * s).abs(), (b * c).abs() + (a * s).abs()], -1).flatten(1)
    assert ((at[:, : hq * d].double() - want).abs() <= bound + 1e-6).all()
