"""Decode attention whose splits are one cluster, against 64-bit attention: the first and last lengths of its range and their
neighbours, empty rows, rows shorter than one split, head groups with and without padding, scattered caches."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bound", [16, 64, 65, 256, 257, 2000])     # one split, clusters, splits with a merge of their own
@pytest.mark.parametrize("fold", [False, True])
def test_an_empty_row_is_zero_whatever_the_bound(bound, fold, monkeypatch):
    import sys

    import lite_llama_b200.kernels as K

    monkeypatch.setattr(sys.modules["lite_llama_b200.kernels.flashdecoding"], "_FOLD", fold)
    q = torch.randn(3, 8, 64, device="cuda", dtype=torch.float16)
    pool = torch.randn(3 * bound, 4, 64, device="cuda", dtype=torch.float16)
    table = torch.arange(3 * bound, device="cuda", dtype=torch.int32).view(3, bound)
    lens = torch.tensor([bound, 0, 1], device="cuda")
    scratch = [torch.full((3, 8, 64), float("nan"), device="cuda", dtype=torch.float16) for _ in range(8)]
    del scratch                                                      # what the result's memory held before
    got = K.flash_decoding(q, pool[:, :2], pool[:, 2:], 0.125, table, torch.arange(3, device="cuda"), lens, bound)
    assert not got[1].any()
    torch.testing.assert_close(got[2].view(2, 4, 64), pool[2 * bound, 2:, None].expand(2, 4, 64), rtol=0, atol=0)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("batch,hq,hkv,d", [(1, 32, 8, 128), (3, 14, 2, 64), (18, 28, 4, 128), (4, 8, 8, 32), (1, 40, 1, 64),
                                            (2, 6, 2, 256)])
@pytest.mark.parametrize("bound", [64, 65, 129, 200, 256, 257])
def test_cluster_splits(bound, batch, hq, hkv, d, dtype):
    import lite_llama_b200.kernels as K

    gen = torch.Generator().manual_seed(bound * 31 + d)
    lens = torch.randint(1, bound + 1, (batch,), generator=gen)
    lens[0] = bound
    if batch > 2:
        lens[1], lens[2] = 0, 1
    q = torch.randn(batch, hq, d, generator=gen).to(dtype).cuda()
    pool = torch.randn(batch * bound + 5, 2 * hkv, d, generator=gen).to(dtype).cuda()
    table = torch.randperm(batch * bound, generator=gen).int().view(batch, bound).cuda() + 5
    slots = torch.randperm(batch, generator=gen).cuda()
    args = (pool[:, :hkv], pool[:, hkv:], d ** -0.5, table, slots, lens.cuda(), bound)
    got = K.flash_decoding(q, *args)
    assert torch.equal(got, K.flash_decoding(q, *args))
    for b in range(batch):
        n = int(lens[b])
        if n == 0:
            assert not got[b].any()
            continue
        rows = table[slots[b], :n].long()
        k, v = pool[rows, :hkv].double(), pool[rows, hkv:].double()
        s = torch.einsum("hgd,nhd->hgn", q[b].double().view(hkv, hq // hkv, d), k) * d ** -0.5
        want = torch.einsum("hgn,nhd->hgd", s.softmax(-1), v).reshape(hq, d)
        # probabilities and the result are rounded to the activation type, scores carry 32-bit sums
        eps = torch.finfo(dtype).eps
        assert float((got[b].double() - want).norm() / want.norm()) < 1.5 * eps
        assert float((got[b].double() - want).abs().max()) < 4 * eps * float(v.abs().max())
