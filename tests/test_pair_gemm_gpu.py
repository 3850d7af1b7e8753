"""The CTA-pair GEMMs of prompt-sized batches (csrc/gemm_pair.cu) against a 64-bit product, at the edges of their tiles:
token counts around the 256-row tile, output counts that end inside a 64-wide store box, a K tail, one tile per pair and
several.  Tolerance: one rounding of the result to 16 bits (2^-9 relative for bf16, 2^-12 for fp16 as a 2-norm bound) on
top of fp32 accumulation, which is orders of magnitude below it."""

from __future__ import annotations

import pytest
import torch

from test_quant_form_cpu import FP8, INT4, INT8, SHARED_TILES, WIDE, WIDE_TILES, form

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(180)]

REL = {torch.float16: 2.0**-11, torch.bfloat16: 2.0**-8}


def K():
    import lite_llama_b200.kernels as k

    return k


def rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


# 129 tokens x 10240 outputs: the fewest tokens and (40 wide tiles of 256) about the fewest tiles the pair kernel takes.  The
# 4104 outputs of 511 tokens run in 66 tiles of 128 outputs.  2049 x 4104 (153 wide tiles) and 700 x 6400 (150 tiles of 128)
# give the 74 pairs a second and a third tile, the accumulators taken in turn
EDGES = [(129, 10240, 192), (256, 10248, 64), (257, 5128, 392), (511, 5112, 1000), (1000, 4096, 520), (2049, 4104, 256),
         (511, 4104, 392), (300, 4104, 1008), (1000, 2056, 72), (700, 6400, 136)]


@pytest.mark.parametrize("m,n,k", EDGES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bias", [False, True])
def test_linear_pair_tiles(m, n, k, dtype, bias):
    x = torch.randn(m, k, device="cuda", dtype=dtype)
    w = torch.randn(n, k, device="cuda", dtype=dtype)
    b = torch.randn(n, device="cuda", dtype=dtype) if bias else None
    want = x.double() @ w.double().T + (b.double() if bias else 0.0)
    got = K().linear(x, w, b)
    assert rel(got, want) < REL[dtype] and torch.equal(K().linear(x, w, b), got)


@pytest.mark.parametrize("m,n,k", [(129, 10240, 192), (256, 10248, 64), (511, 5112, 1008), (2049, 4104, 256),
                                   (511, 4104, 400), (300, 4104, 1008), (700, 6400, 144)])
@pytest.mark.parametrize("bias", [False, True])
def test_int8_pair_tiles(m, n, k, bias):
    qa = torch.randint(-127, 128, (m, k), device="cuda", dtype=torch.int8)
    qw = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
    sa, sw = torch.rand(m, device="cuda") * 1e-2, torch.rand(n, device="cuda") * 1e-2
    b = torch.randn(n, device="cuda") if bias else None
    want = (qa.double() @ qw.double().T) * sa.double()[:, None] * sw.double() + (b.double() if bias else 0.0)
    assert rel(K().smoothquant_matmul_prequant(qa, sa, qw, sw, bias=b), want) < REL[torch.float16]


def test_linear_forms_the_pair_kernel_does_not_take():
    """Output counts that are no multiple of 8 stay on the one-SM kernel; strided activations and weights go either way."""
    x = torch.randn(600, 512, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(10250, 512, device="cuda", dtype=torch.bfloat16)
    assert rel(K().linear(x, w), x.double() @ w.double().T) < REL[torch.bfloat16]
    xs, ws = x[:, 64:320], w[:10240, 128:384]
    assert rel(K().linear(xs, ws), xs.double() @ ws.double().T) < REL[torch.bfloat16]


# ---- quantised weights (csrc/gemm_quant_pair.cu): 256-row x 128-token tiles, 128 k per operand stage ----
# m: one token over / under a tile, 64-token edge of the dispatch; n: rows past the last tile; k: an odd number of stages
# (half a raw block is left over), one and several stages per scale group.  129 x 5128: the wave rule leaves scale groups to
# the streaming kernel and gives one scale per row to the pair kernel; 129 x 18944 is the pair kernel's either way.  From
# 129 x 18944 on there are 148 to 304 tiles for 74 pairs: what a pair carries from one tile to the next (ring phases, stage
# and raw-block counts of the conversion groups, accumulator in turn), and a short last tile after full ones
QUANT_EDGES = [(65, 10240, 128), (127, 10140, 384), (129, 5128, 640), (500, 2600, 256), (1000, 1300, 896),
               (129, 18944, 640), (1000, 9728, 896), (1153, 5128, 384), (1100, 9728, 768)]


def int4_case(n, k, group, m):
    q = torch.randint(-(2**31), 2**31 - 1, (n, k // 8), device="cuda", dtype=torch.int64).to(torch.int32)
    s = torch.rand(n, k // group, device="cuda") * 4e-3 + 1e-3
    z = torch.randint(0, 16, (n, k // group), device="cuda").float()
    codes = torch.stack([(q >> (4 * j)) & 15 for j in range(8)], -1).view(n, k // group, group).double()
    w = ((codes - z.double()[..., None]) * s.double()[..., None]).view(n, k)
    return q, s, z, w, torch.randn(m, k, device="cuda", dtype=torch.float16)


@pytest.mark.parametrize("m,n,k", QUANT_EDGES)
@pytest.mark.parametrize("group", [128, 256])
@pytest.mark.parametrize("bias", [None, torch.float16, torch.float32])
def test_int4_pair_tiles(m, n, k, group, bias):
    if k % group:
        pytest.skip("groups divide k")
    q, s, z, w, x = int4_case(n, k, group, m)
    b = None if bias is None else torch.randn(n, device="cuda", dtype=bias)
    packed = K().w4a16_pack(q, s, z, group_size=group)
    got = K().w4a16_matmul_packed(x, packed, bias=b)
    assert rel(got, x.double() @ w.T + (0.0 if b is None else b.double())) < REL[torch.float16]
    assert torch.equal(K().w4a16_matmul_packed(x, packed, bias=b), got)


@pytest.mark.parametrize("m,n,k", QUANT_EDGES)
def test_int4_pair_swiglu_is_gemm_then_swiglu(m, n, k):
    from lite_llama_b200.kernels.quantization import interleave_gate_up

    q, s, z, _, x = int4_case(n, k, 128, m)
    wide = K().w4a16_matmul_packed(x, K().w4a16_pack(q, s, z, group_size=128))
    want = K().swiglu_forward(wide[:, : n // 2], wide[:, n // 2 :])
    packed = K().w4a16_pack(interleave_gate_up(q), interleave_gate_up(s), interleave_gate_up(z), group_size=128)
    assert torch.equal(K().w4a16_matmul_packed(x, packed, swiglu=True), want)


@pytest.mark.parametrize("m,n,k", QUANT_EDGES + [(300, 5000, 400)])       # 400: the last stage is partly past k
@pytest.mark.parametrize("fmt", ["fp8_block", "fp8_channel", "int8_channel", "int8_group_n"])
def test_w8_pair_tiles(m, n, k, fmt):
    x = torch.randn(m, k, device="cuda", dtype=torch.float16)
    if fmt.startswith("fp8"):
        q = (torch.randn(n, k, device="cuda") * 60).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        w = q.view(torch.float8_e4m3fn).double()
    else:
        q = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
        w = q.double()
    gn, gk = {"fp8_block": (128, 128), "int8_group_n": (48, k)}.get(fmt, (1, k))
    s = torch.rand((n + gn - 1) // gn, (k + gk - 1) // gk, device="cuda") * 1e-3
    w = w * s.double().repeat_interleave(gn, 0)[:n].repeat_interleave(gk, 1)[:, :k]
    b = torch.randn(n, device="cuda")
    got = K().w8a16_matmul(x, q, s, group_n=gn, group_k=gk, bias=b)
    assert rel(got, x.double() @ w.T + b.double()) < REL[torch.float16]


@pytest.mark.parametrize("m", [1, 31, 33, 64])
@pytest.mark.parametrize("n,k", [(10140, 528), (4096, 4096), (19210, 528)])      # 64 tokens of the last: the pair kernel's tiles
@pytest.mark.parametrize("fp8", [True, False])
def test_w8_per_channel_decode_tiles(m, n, k, fp8):
    x = torch.randn(m, k, device="cuda", dtype=torch.float16)
    if fp8:
        q = (torch.randn(n, k, device="cuda") * 60).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        w = q.view(torch.float8_e4m3fn).double()
    else:
        q = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
        w = q.double()
    s = torch.rand(n, 1, device="cuda") * 1e-3
    got = K().w8a16_matmul(x, q, s, group_n=1, group_k=k)
    assert rel(got, x.double() @ (w * s.double()).T) < REL[torch.float16]


# ---- routed experts (b2l_moe_sort / b2l_moe_gather / b2l_moe_pair_gemm) ----
@pytest.mark.parametrize("fmt", ["fp8", "int8"])
@pytest.mark.parametrize("hidden,inter,gn,gk", [(256, 128, 128, 128), (400, 208, 16, 512), (1024, 320, 64, 128),
                                                (2176, 1152, 128, 128)])
@pytest.mark.parametrize("idle", [0, 30])
def test_experts_with_runs_around_the_tile(fmt, hidden, inter, gn, gk, idle):
    """Runs of 0, 1, 16, 17, 32, 33, 127, 128, 129 and 300 rows; outputs and intermediate columns past the last tile.  With 30
    idle experts beside them the rows per expert are few enough for tiles of 64 rows.  2176 x 1152: 108 to 153 tiles for 74
    pairs and odd stage counts, so pairs go from one expert's tile to another's."""
    runs = [0, 1, 16, 17, 32, 33, 127, 128, 129, 300] + [0] * idle
    E, top_k = len(runs), 1
    ids = torch.cat([torch.full((n,), e) for e, n in enumerate(runs)])
    ids = ids[torch.randperm(ids.numel())].view(-1, top_k).cuda()
    T = ids.shape[0]
    x = torch.randn(T, hidden, device="cuda", dtype=torch.float16)

    def weight(n, k):
        if fmt == "fp8":
            q = (torch.randn(E, n, k, device="cuda") * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
            raw, q = q.view(torch.uint8), q.double()
        else:
            raw = torch.randint(-127, 128, (E, n, k), device="cuda", dtype=torch.int8)
            q = raw.double()
        s = torch.rand(E, -(-n // gn), -(-k // gk), device="cuda") * 5e-4
        return raw, s, q * s.double().repeat_interleave(gn, 1)[:, :n].repeat_interleave(gk, 2)[:, :, :k]

    w1, s1, d1 = weight(2 * inter, hidden)
    w2, s2, d2 = weight(hidden, inter)
    tw = torch.rand(T, top_k, device="cuda").half()
    def call():
        return K().fused_moe(x, w1, w2, tw, ids, w1_scale=s1, w2_scale=s2, group_n=gn, group_k=gk)

    got = call()
    assert torch.equal(call(), got)          # the order of an expert's rows may differ, their values not
    want = torch.empty(T, hidden, dtype=torch.float64, device="cuda")
    for e in range(E):
        t = (ids[:, 0] == e).nonzero()[:, 0]
        g, u = (x[t].double() @ d1[e].T).half().double().chunk(2, -1)
        a = (torch.nn.functional.silu(g) * u).half().double()
        want[t] = (a @ d2[e].T) * tw[t].double()
    assert rel(got, want) < 2 * REL[torch.float16]        # two roundings to 16 bits between the products, one at the end


@pytest.mark.parametrize("slots,experts,width", [(1, 1, torch.int32), (255, 3, torch.int64), (4000, 130, torch.int32),
                                                 (700, 2048, torch.int64)])
def test_moe_sort_lists_every_valid_slot_once(slots, experts, width):
    from lite_llama_b200 import _lib

    L = _lib.load()
    ids = torch.randint(-1, experts + 1, (slots,), device="cuda", dtype=width)       # -1 and `experts` belong to nobody
    most = L.b2l_moe_sort_max_tiles(slots, 128, experts)
    order = torch.full((slots + 1,), -7, dtype=torch.int32, device="cuda")
    table = torch.full((1 + 3 * most,), -7, dtype=torch.int32, device="cuda")
    _lib.check(L.b2l_moe_sort(order.data_ptr(), table.data_ptr(), ids.data_ptr(), ids.element_size(), slots, 128, experts,
                              torch.cuda.current_stream().cuda_stream))
    order, table, ids = order.tolist(), table.tolist(), ids.tolist()
    valid = [i for i, e in enumerate(ids) if 0 <= e < experts]
    assert order[slots] == len(valid) and sorted(order[: len(valid)]) == valid
    assert table[0] <= most
    row = 0
    for t in range(table[0]):
        e, first, rows = table[1 + 3 * t : 4 + 3 * t]
        assert first == row and 1 <= rows <= 128 and all(ids[s] == e for s in order[first : first + rows])
        row += rows
    assert row == len(valid)


# ---- the 16-byte forms of two element-wise kernels against the forms for any alignment ----
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k", [(1, 2048), (3, 8192), (2, 8200), (5, 18944), (2, 32768), (2, 32776)])
def test_quantiser_in_vectors_equals_the_scalar_one(m, k, dtype):
    x = torch.randn(m, k + 8, device="cuda", dtype=dtype)
    x[0, 3], x[-1, :8] = 30.0, 0.0
    q, s = K().quantize_activations_int8(x[:, :k])                    # 16-byte rows
    q2, s2 = K().quantize_activations_int8(x[:, 1 : k + 1])           # the same kernel family on unaligned rows ...
    xs = torch.empty(m, k + 9, device="cuda", dtype=dtype)
    xs[:, 1 : k + 1] = x[:, :k]
    q3, s3 = K().quantize_activations_int8(xs[:, 1 : k + 1])          # ... and on the same values, unaligned
    assert torch.equal(q, q3) and torch.equal(s, s3)
    assert q2.shape == q.shape and s2.shape == s.shape
    want = (x[:, :k].float().abs().amax(-1) / 127.0)
    assert torch.equal(s, torch.where(want > 0, want, torch.ones_like(want)))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tokens,n,top_k", [(1, 8, 1), (3, 2048, 8), (70, 264, 9), (5, 100, 8), (445, 8, 1),
                                            (300, 264, 9), (120, 2048, 8), (500, 100, 8)])
@pytest.mark.parametrize("addend", [False, True])
def test_expert_sum_in_vectors(tokens, n, top_k, addend, dtype):
    from lite_llama_b200 import _lib

    L = _lib.load()
    x = torch.randn(tokens, top_k, n, device="cuda", dtype=dtype)
    add = torch.randn(tokens, n, device="cuda", dtype=dtype) if addend else None
    out = torch.empty(tokens, n, device="cuda", dtype=dtype)
    _lib.check(L.b2l_moe_sum(out.data_ptr(), x.data_ptr(), add.data_ptr() if addend else None, tokens, n, top_k,
                             0 if dtype == torch.float16 else 1, torch.cuda.current_stream().cuda_stream))
    acc = torch.zeros(tokens, n, device="cuda")
    for k in range(top_k):
        acc = acc + x[:, k].float()
    assert torch.equal(out, (acc + add.float() if addend else acc).to(dtype))


# ---- how long one accumulation in tensor memory runs where a scale covers all of k ----
# (m, n, k, k values per accumulation): parts of k as 148 SMs / (n / 128 x m / 64 tiles) leave them
@pytest.mark.parametrize("m,n,k,chain", [(16, 4096, 4096, 1024), (64, 6144, 4096, 1408), (128, 4096, 4096, 2048),
                                         (96, 4096, 14336, 7168), (192, 2048, 4096, 1408)])
@pytest.mark.parametrize("fp8", [True, False])
def test_per_channel_accumulations_are_no_longer_than_the_parts_of_k(m, n, k, chain, fp8):
    """Positive values, so that the accumulator's rounding shows as a mean deviation, far above that of the rounding to fp16.
    One addition of 16 products loses less than 2^-23 of the partial sum; over twice the chain and more it exceeds the bound
    for int8."""
    x = torch.rand(m, k, device="cuda").mul_(0.5).add_(0.5).half()
    if fp8:
        q = (torch.rand(n, k, device="cuda") * 100 + 20).to(torch.float8_e4m3fn).view(torch.uint8)
        w = q.view(torch.float8_e4m3fn).double()
    else:
        q = torch.randint(1, 127, (n, k), device="cuda", dtype=torch.int8)
        w = q.double()
    s = torch.rand(n, 1, device="cuda") * 1e-4 + 1e-4
    got, want = K().w8a16_matmul(x, q, s, group_n=1, group_k=k).double(), x.double() @ (w * s.double()).T
    assert abs(((got - want) / want).mean().item()) < chain / 16 * 2.0**-23


# parts of k that had a CTA each (four blocks of 64 on 148 SMs) and now share one: two, three, four of them, the last part shorter
@pytest.mark.parametrize("m,n,k", [(64, 896, 4864), (33, 512, 8192), (64, 512, 8192), (17, 896, 4864), (48, 1000, 2104), (16, 240, 10160)])
def test_linear_accumulates_no_longer_than_the_parts_of_k(m, n, k):
    """Positive values: one addition of 16 products cuts off less than 2^-23 of the partial sum, over 256 k (16 additions) half of
    16 * 2^-23 on average.  The mean over eight inputs leaves 5e-7 of the rounding to fp16; over 640 k and more the bound is missed
    by half and more."""
    dev = 0.0
    for _ in range(8):
        x = torch.rand(m, k, device="cuda").mul_(0.5).add_(0.5).half()
        w = (torch.rand(n, k, device="cuda") + 0.1).half()
        want = x.double() @ w.double().T
        dev += ((K().linear(x, w).double() - want) / want).mean().item() / 8
    assert abs(dev) < 16 * 2.0**-23


@pytest.mark.parametrize("m,n,k", [(1, 136, 64), (17, 1000, 256), (130, 520, 512), (300, 10248, 144), (256, 3584, 2048),
                                   (7, 1000, 256), (33, 520, 4096), (65, 9736, 896), (97, 9736, 128)])
@pytest.mark.parametrize("shift", [0, 1])
def test_int8_scales_in_vectors_and_alone(m, n, k, shift):
    """Scales and bias that start on a 16-byte boundary are loaded in vectors, others one by one: the same result."""
    qa = torch.randint(-127, 128, (m, k), device="cuda", dtype=torch.int8)
    qw = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
    sa, sw, b = ((torch.rand(v + 1, device="cuda") * 1e-2)[shift : shift + v] for v in (m, n, n))
    want = (qa.double() @ qw.double().T) * sa.double()[:, None] * sw.double() + b.double()
    got = K().smoothquant_matmul_prequant(qa, sa, qw, sw, bias=b)
    assert rel(got, want) < REL[torch.float16]
    assert torch.equal(got, K().smoothquant_matmul_prequant(qa, sa.clone(), qw, sw.clone(), bias=b.clone()))


# Clusters of two and four pairs that share a tile: parts of k of unequal length, a k tail, outputs that end inside a tile, one
# to four token tiles, tokens in the first CTA of a pair only
SPLIT_EDGES = [(65, 896, 4872), (128, 3584, 2056), (129, 1000, 2112), (256, 3400, 4200), (700, 776, 4104), (256, 4096, 4232),
               (500, 2056, 8200), (1000, 1800, 5208), (600, 2300, 10248)]


@pytest.mark.parametrize("m,n,k", SPLIT_EDGES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bias", [False, True])
def test_linear_split_over_a_cluster(m, n, k, dtype, bias):
    x = torch.randn(m, k, device="cuda", dtype=dtype)
    w = torch.randn(n, k, device="cuda", dtype=dtype) * 0.05
    b = torch.randn(n, device="cuda", dtype=dtype) if bias else None
    want = x.double() @ w.double().T + (b.double() if bias else 0.0)
    got = K().linear(x, w, b)
    assert rel(got, want) < REL[dtype] and torch.equal(K().linear(x, w, b), got)


@pytest.mark.parametrize("m,n,k", SPLIT_EDGES)
@pytest.mark.parametrize("bias", [False, True])
def test_int8_split_over_a_cluster(m, n, k, bias):
    k = (k + 15) // 16 * 16
    qa = torch.randint(-127, 128, (m, k), device="cuda", dtype=torch.int8)
    qw = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
    sa, sw = torch.rand(m, device="cuda") * 1e-3, torch.rand(n, device="cuda") * 1e-2
    b = torch.randn(n, device="cuda") if bias else None
    want = (qa.double() @ qw.double().T) * sa.double()[:, None] * sw.double() + (b.double() if bias else 0.0)
    assert rel(K().smoothquant_matmul_prequant(qa, sa, qw, sw, bias=b), want) < REL[torch.float16]


# ---- 256 tokens per tile (csrc/gemm_quant_wide.cu): WIDE_TILES reach it, the others lie around its line (the form with the activation
# takes most of them) ----
WIDE_EDGES = [(300, 18944, 384), (513, 12800, 640), (1000, 9734, 128), (769, 9734, 384), (640, 18688, 896), (1537, 3330, 1152)]


@pytest.mark.parametrize("m,n,k", WIDE_EDGES)
@pytest.mark.parametrize("group", [128, 384])
def test_int4_wide_tiles(m, n, k, group):
    if k % group:
        pytest.skip("groups divide k")
    q, s, z, w, x = int4_case(n, k, group, m)
    b = torch.randn(n, device="cuda")
    packed = K().w4a16_pack(q, s, z, group_size=group)
    got = K().w4a16_matmul_packed(x, packed, bias=b)
    assert rel(got, x.double() @ w.T + b.double()) < REL[torch.float16]
    if n > 148 * 64:    # a row's sums do not depend on its tile: the same bits from the kernel of 128 tokens per tile
        assert torch.equal(K().w4a16_matmul_packed(x[:128], packed, bias=b), got[:128])


@pytest.mark.parametrize("m,n,k", WIDE_EDGES)
def test_int4_wide_swiglu_is_gemm_then_swiglu(m, n, k):
    test_int4_pair_swiglu_is_gemm_then_swiglu(m, n, k)


@pytest.mark.parametrize("m,n,k", WIDE_EDGES)
@pytest.mark.parametrize("fmt", ["fp8_block", "fp8_channel", "int8_channel", "int8_group_n"])
def test_w8_wide_tiles(m, n, k, fmt):
    test_w8_pair_tiles(m, n, k, fmt)


@pytest.mark.parametrize("m,n,k", WIDE_TILES)
@pytest.mark.parametrize("group", [128, 384])
def test_int4_tiles_of_256_tokens(m, n, k, group):
    if k % group == 0:
        assert form(INT4, m, n, k, group)[0] == WIDE
    test_int4_wide_tiles(m, n, k, group)


@pytest.mark.parametrize("m,n,k", WIDE_TILES)
def test_int4_swiglu_tiles_of_256_tokens(m, n, k):
    assert form(INT4, m, n, k, 128, True)[0] == WIDE
    test_int4_pair_swiglu_is_gemm_then_swiglu(m, n, k)


@pytest.mark.parametrize("m,n,k", WIDE_TILES)
@pytest.mark.parametrize("fmt", ["fp8_channel", "int8_channel", "int8_group_n"])
def test_w8_tiles_of_256_tokens(m, n, k, fmt):
    assert form(FP8 if fmt.startswith("fp8") else INT8, m, n, k, k)[0] == WIDE
    test_w8_pair_tiles(m, n, k, fmt)


# ---- one-SM kernel (csrc/gemm_dense.cu): 128-token tiles where 64-token tiles would need a second wave (75 - 148 weight tiles), and
# fewer splits of k than there are SMs for where the last CTA of a tile would add up too many
PLAN_EDGES = [(65, 9728, 896), (128, 18944, 192), (100, 9600, 320), (16, 128, 4096), (64, 896, 4864), (33, 512, 8192), (200, 256, 2048)]


@pytest.mark.parametrize("m,n,k", PLAN_EDGES)
def test_linear_token_tiles_and_splits(m, n, k):
    for dtype in (torch.float16, torch.bfloat16):
        test_linear_pair_tiles(m, n, k, dtype, True)


@pytest.mark.parametrize("m,n,k", PLAN_EDGES)
def test_int8_token_tiles_and_splits(m, n, k):
    test_int8_pair_tiles(m, n, k, True)


# ---- several pairs on a tile (csrc/gemm_quant_pair.cu): four up to 15 tiles, three up to 22, two up to 33, by steps of k; and sizes
# that the rule leaves to a pair each or to the streaming kernel
SPLIT_EDGES = list(SHARED_TILES) + [(100, 8192, 1152), (200, 4096, 1408), (500, 1730, 2048), (257, 2600, 1024)]


@pytest.mark.parametrize("m,n,k", SPLIT_EDGES)
@pytest.mark.parametrize("group", [128, 256, 0])
@pytest.mark.parametrize("bias", [None, torch.float16, torch.float32])
def test_int4_shared_tiles(m, n, k, group, bias):
    test_int4_pair_tiles(m, n, k, group or k, bias)


@pytest.mark.parametrize("m,n,k", SPLIT_EDGES)
def test_int4_shared_swiglu_is_gemm_then_swiglu(m, n, k):
    test_int4_pair_swiglu_is_gemm_then_swiglu(m, n, k)


@pytest.mark.parametrize("m,n,k", SPLIT_EDGES + [(300, 1000, 2000)])
@pytest.mark.parametrize("fmt", ["fp8_block", "fp8_channel", "int8_channel", "int8_group_n"])
def test_w8_shared_tiles(m, n, k, fmt):
    test_w8_pair_tiles(m, n, k, fmt)


@pytest.mark.parametrize("idle", [5, 7])      # 52 and 46 rows per expert: either side of the line between tiles of 128 and 64 rows
@pytest.mark.parametrize("fmt", ["fp8", "int8"])
def test_experts_either_side_of_the_smaller_tile(fmt, idle):
    test_experts_with_runs_around_the_tile(fmt, 1024, 384, 128, 128, idle)
