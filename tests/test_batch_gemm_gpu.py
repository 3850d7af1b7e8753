"""The quantised projections of decode batches (csrc/gemm_quant_batch.cu) against a 64-bit product, where the kernel can go
wrong: token counts around its tiles of 16 / 32 / 48 / 64, one block of k and odd numbers of 128-k steps, rows past the last
tile, tiles shared by several CTAs in equal parts and in unequal ones, CTAs with parts of several tiles.  Tolerance: one
rounding of the result to fp16 (2^-12 as a 2-norm bound) on top of fp32 accumulation, orders of magnitude below it."""

from __future__ import annotations

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(180)]

REL = 2.0**-11
TOKENS = [9, 16, 17, 32, 33, 48, 49, 64]
# n, k: a single step; an odd step count (half a block left over); many sharers; equal splits; more tiles than SMs, where CTAs
# take parts of two or three tiles; the same with an odd step count
SHAPES = [(130, 128), (1000, 384), (896, 4864), (2048, 2048), (20100, 1280), (19100, 640)]


def K():
    import lite_llama_b200.kernels as k

    return k


def rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


def int4_case(n, k, group, m):
    q = torch.randint(-(2**31), 2**31 - 1, (n, k // 8), device="cuda", dtype=torch.int64).to(torch.int32)
    s = torch.rand(n, k // group, device="cuda") * 4e-3 + 1e-3
    z = torch.randint(0, 16, (n, k // group), device="cuda").float()
    codes = torch.stack([(q >> (4 * j)) & 15 for j in range(8)], -1).view(n, k // group, group).double()
    w = ((codes - z.double()[..., None]) * s.double()[..., None]).view(n, k)
    return q, s, z, w, torch.randn(m, k, device="cuda", dtype=torch.float16)


@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("group", [128, 256, 384])
def test_int4_batches(n, k, group):
    if k % group:
        pytest.skip("groups divide k")
    q, s, z, w, x64 = int4_case(n, k, group, 64)
    packed = K().w4a16_pack(q, s, z, group_size=group)
    for i, m in enumerate(TOKENS):
        x = x64[:m]
        b = (None, torch.randn(n, device="cuda", dtype=torch.float16), torch.randn(n, device="cuda"))[i % 3]
        got = K().w4a16_matmul_packed(x, packed, bias=b)
        assert rel(got, x.double() @ w.T + (0.0 if b is None else b.double())) < REL, m
        assert torch.equal(K().w4a16_matmul_packed(x, packed, bias=b), got), m
        other = K().w4a16_matmul(x, q, s, z, group_size=group, bias=b)           # the reference's layout
        if m <= 48 or n <= 148 * 128:                                            # else the streaming kernel's
            assert torch.equal(other, got), m


@pytest.mark.parametrize("n,k", [(1000, 384), (2048, 2048)])
def test_int4_batches_with_zero_points_that_are_not_whole(n, k):
    q, s, z, w, x64 = int4_case(n, k, 128, 64)
    off = torch.rand_like(z) * (torch.rand_like(z) < 0.1)              # a tenth of the groups
    w = w - (off * s).double().repeat_interleave(128, 1)
    for m in TOKENS:
        got = K().w4a16_matmul(x64[:m], q, s, z + off, group_size=128)
        assert rel(got, x64[:m].double() @ w.T) < REL, m
        assert torch.equal(K().w4a16_matmul(x64[:m], q, s, z + off, group_size=128), got), m


@pytest.mark.parametrize("m", [9, 64])
def test_int4_tables_of_any_stride(m):
    """The scales and zero points of the reference's layout as views: one row for all, rows that overlap, groups along the rows,
    rows with a gap, a start that is no multiple of 16 bytes."""
    n, k, groups = 300, 1024, 8
    q, s, z, _, x = int4_case(n, k, 128, m)
    flat_s, flat_z = torch.rand(8 * n, device="cuda") * 4e-3 + 1e-3, torch.randint(0, 16, (8 * n,), device="cuda").float()
    views = [lambda t: t[:groups].expand(n, groups), lambda t: t.as_strided((n, groups), (4, 1)),
             lambda t: t[: n * groups].view(groups, n).t(), lambda t: t.repeat(2).as_strided((n, groups), (12, 1)),
             lambda t: t[1:].as_strided((n, groups), (4, 1))]
    for view in views:
        sv, zv = view(flat_s), view(flat_z)
        want = K().w4a16_matmul(x, q, sv.contiguous(), zv.contiguous(), group_size=128)
        assert torch.equal(K().w4a16_matmul(x, q, sv, zv, group_size=128), want)


@pytest.mark.parametrize("n,k", SHAPES)
def test_int4_batches_with_activation_are_gemm_then_swiglu(n, k):
    from lite_llama_b200.kernels.quantization import interleave_gate_up

    q, s, z, _, x64 = int4_case(n, k, 128, 64)
    packed = K().w4a16_pack(*(interleave_gate_up(t) for t in (q, s, z)), group_size=128)
    for m in TOKENS:
        wide = K().w4a16_matmul_packed(x64[:m], packed)                # (gate_0, up_0, gate_1, ...)
        want = K().swiglu_forward(wide[:, 0::2].contiguous(), wide[:, 1::2].contiguous())
        assert torch.equal(K().w4a16_matmul_packed(x64[:m], packed, swiglu=True), want), m


@pytest.mark.parametrize("n,k", SHAPES + [(300, 400)])                 # 400: the last step is partly past k
@pytest.mark.parametrize("fmt", ["fp8_block", "fp8_channel", "int8_channel", "int8_group_n"])
def test_w8_batches(n, k, fmt):
    x64 = torch.randn(64, k, device="cuda", dtype=torch.float16)
    if fmt.startswith("fp8"):
        q = (torch.randn(n, k, device="cuda") * 60).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        w = q.view(torch.float8_e4m3fn).double()
    else:
        q = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
        w = q.double()
    gn, gk = {"fp8_block": (128, 128), "int8_group_n": (48, k)}.get(fmt, (1, k))
    s = torch.rand((n + gn - 1) // gn, (k + gk - 1) // gk, device="cuda") * 1e-3 + 1e-4
    w = w * s.double().repeat_interleave(gn, 0)[:n].repeat_interleave(gk, 1)[:, :k]
    for m in [1, 8] + TOKENS:
        got = K().w8a16_matmul(x64[:m], q, s, group_n=gn, group_k=gk)
        assert rel(got, x64[:m].double() @ w.T) < REL, m
        assert torch.equal(K().w8a16_matmul(x64[:m], q, s, group_n=gn, group_k=gk), got), m


@pytest.mark.parametrize("m", [24, 64])
def test_infinities_pass_through_shared_tiles(m):
    """2048 x 2048 has several CTAs per tile: an infinite or undefined partial sum arrives as what it is."""
    q = torch.ones(2048, 2048, device="cuda", dtype=torch.int8)
    q[:, 7::16] = -1
    x = torch.zeros(m, 2048, device="cuda", dtype=torch.float16)
    x[0, 1600], x[1, 1607], x[2, 3] = float("inf"), float("inf"), float("nan")
    x[3, 5], x[3, 2000] = float("inf"), float("-inf")
    got = K().w8a16_matmul(x, q, torch.ones(2048, 1, device="cuda"), group_n=1, group_k=2048)
    assert (got[0] == float("inf")).all() and (got[1] == float("-inf")).all()
    assert got[2].isnan().all() and got[3].isnan().all() and (got[4:] == 0).all()


@pytest.mark.parametrize("m", [1, 16, 33, 64])
@pytest.mark.parametrize("n,k", [(2048, 2048), (20100, 1280)])        # equal parts of a tile; parts of several tiles
def test_partial_sums_keep_their_bits(m, n, k):
    """Every product is a multiple of 12.5 and every sum of them below 2^17, so 32-bit sums are exact in any order, and the halves
    of k cancel.  A partial sum that loses its last bit between CTAs leaves a remainder."""
    q = torch.full((n, k), 100, device="cuda", dtype=torch.int8)
    half = torch.randint(1, 16, (m, k // 2), device="cuda").half() / 2
    x = torch.cat([half, -half.flip(1)], 1)
    got = K().w8a16_matmul(x, q, torch.full((n, 1), 0.25, device="cuda"), group_n=1, group_k=k)
    assert not got.any()


def test_workspace_is_left_clean_and_a_smaller_one_takes_the_streaming_kernel():
    import lite_llama_b200.kernels._common as c
    from lite_llama_b200 import _lib

    lib = _lib.load()
    n, k, m = 2048, 4096, 64
    x = torch.randn(m, k, device="cuda", dtype=torch.float16)
    q = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
    s = torch.rand(n // 128, k // 128, device="cuda") * 1e-3
    want = K().w8a16_matmul(x, q, s, group_n=128, group_k=128)
    full = lib.b2l_quant_gemm_workspace_bytes(2, m, n, k, 128)
    cnt = c.counters(x.device)
    for nbytes in (full, full // 2, 0):
        ws, out = torch.zeros(full, dtype=torch.uint8, device="cuda"), torch.empty(m, n, device="cuda", dtype=torch.float16)
        rc = lib.b2l_w8a16_matmul(out.data_ptr(), x.data_ptr(), q.data_ptr(), 0, s.data_ptr(), None, 0, m, n, k, 128, 128,
                                  k, k, s.stride(0), s.stride(1), n, ws.data_ptr(), nbytes, cnt.data_ptr(), cnt.numel(),
                                  c.stream_handle())
        torch.cuda.synchronize()
        assert (ws == 0).all() and (cnt == 0).all()
        if rc == 0:                       # less than the streaming kernel needs is refused, as before
            assert rel(out, want.double()) < REL
        else:
            assert nbytes < full
    assert rc != 0
