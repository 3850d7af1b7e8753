"""The native form of the hot shims against the general Python form: the same bits where it takes a call, and no answer for
every form that it leaves to Python (which also keeps the error messages)."""

from __future__ import annotations

import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu


def setup_module():
    import lite_llama_b200.kernels as K
    x = torch.ones(2, 8, device="cuda", dtype=torch.float16)
    K.swiglu_forward(x, x)                      # the first call binds


def data(rows: int, n: int, k: int):
    g = torch.Generator().manual_seed(rows * 7 + n)
    x = torch.randn(rows, k, generator=g).half().cuda()
    w = torch.randn(n, k, generator=g).half().cuda()
    q8 = torch.randint(-127, 128, (n, k), generator=g, dtype=torch.int8).cuda()
    s8 = torch.rand(n, 1, generator=g).cuda() * 0.01
    return x, w, q8, s8


def forms(rows: int, n: int, k: int):
    """name -> (native call, general call), both on tensors in the plain form"""
    import sys
    import lite_llama_b200.kernels as K
    from lite_llama_b200.kernels import _native as N

    mod = lambda m: sys.modules["lite_llama_b200.kernels." + m]                      # noqa: E731
    x, w, q8, s8 = data(rows, n, k)
    q4 = torch.randint(-2**31, 2**31 - 1, (n, k // 8), dtype=torch.int64).int().cuda()
    s4, z4 = torch.rand(n, k // 64).cuda() * 0.01, torch.randint(0, 16, (n, k // 64)).float().cuda()
    p = K.w4a16_pack(q4, s4, z4, group_size=64)
    a, sa = mod("quantization.w8a8")._quantize_activations_int8(x)
    norm, w1 = mod("skip_rmsnorm"), w[0].contiguous()
    w4 = lambda t, sw: (t, p.qweight, p.scales, p.zeros, p.n, p.k, 64, p.zeros_foldable, sw)    # noqa: E731
    return {
        "w8a16": (x, lambda t: N.w8a16(t, q8, s8, 1, k), lambda t: mod("quantization.w8a16")._w8a16_matmul(t, q8, s8, 1, k, None)),
        "w4a16": (x, lambda t: N.w4a16_packed(*w4(t, False)), lambda t: mod("quantization.w4a16")._w4a16_matmul_packed(t, p, None, False)),
        "w4a16_swiglu": (x, lambda t: N.w4a16_packed(*w4(t, True)), lambda t: mod("quantization.w4a16")._w4a16_matmul_packed(t, p, None, True)),
        "linear": (x, lambda t: N.linear(t, w), lambda t: mod("linear")._linear(t, w, None)),
        "w8a8": (a, lambda t: N.w8a8(t, sa, q8, s8, True),
                 lambda t: mod("quantization.w8a8")._smoothquant_matmul_prequant(t, sa, q8, s8, None, torch.bfloat16)),
        "quantize": (x, N.quantize, mod("quantization.w8a8")._quantize_activations_int8),
        "norm": (x, lambda t: N.norm(t, None, w1, 1e-5), lambda t: norm._skip_rmsnorm(t, None, w1, 1e-5)),
        "norm_residual": (x, lambda t: N.norm(t, x.flip(0), w1, 1e-5), lambda t: norm._skip_rmsnorm(t, x.flip(0), w1, 1e-5)),
        "norm_quant": (x, lambda t: N.norm_quant(t, x.flip(0), w1, 1e-5),
                       lambda t: norm._skip_rmsnorm_quant_int8(t, x.flip(0), w1, 1e-5)[:2]),
        "swiglu": (x, lambda t: N.swiglu(t, x.flip(0)), lambda t: mod("swiglu")._swiglu_forward(t, x.flip(0))),
    }


NAMES = ["w8a16", "w4a16", "w4a16_swiglu", "linear", "w8a8", "quantize", "norm", "norm_residual", "norm_quant", "swiglu"]


def same(a, b) -> None:
    for u, v in zip(a, b, strict=True) if isinstance(a, tuple) else [(a, b)]:
        assert u.dtype == v.dtype and u.shape == v.shape and u.stride() == v.stride() and u.requires_grad == v.requires_grad
        assert torch.equal(u, v)


@pytest.mark.parametrize("rows,n,k", [(1, 128, 128), (5, 200, 192), (70, 256, 512), (300, 1032, 256)])
@pytest.mark.parametrize("name", NAMES)
def test_native_and_general_form_agree(name, rows, n, k):
    x, native, general = forms(rows, n, k)[name]
    got = native(x)
    assert got is not None
    same(got, general(x))


class Seen(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class Dispatched(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class Sub(torch.Tensor):
    pass


@pytest.mark.parametrize("name", NAMES)
def test_forms_left_to_python(name):
    x, native, _ = forms(5, 128, 128)[name]
    wide = torch.cat([x, x], 1)
    assert native(x[None]) is None                                     # three dimensions
    assert native(x.new_empty((0, 128))) is None                       # no rows
    assert native(wide[:, ::2]) is None                                # columns that do not follow one another
    assert native(x.as_subclass(Sub)) is None
    assert native(x.cpu()) is None
    assert native(x.float() if name != "swiglu" else x.double()) is None
    with Seen():
        assert native(x) is None
    with Dispatched():
        assert native(x) is None
    if name in ("w8a16", "w4a16", "w4a16_swiglu", "linear"):
        assert native(wide.view(-1)[4:4 + x.numel()].view(x.shape)) is None          # rows off a 16-byte boundary
    if name.startswith("norm"):
        assert native(x.clone().requires_grad_()) is None
        assert native(wide[:, :128]) is None


def test_errors_keep_their_text():
    import lite_llama_b200.kernels as K
    x, w, q8, s8 = data(4, 128, 128)
    for bad in (lambda: K.linear(x, w.bfloat16()), lambda: K.w8a16_matmul(x.bfloat16(), q8, s8, group_n=1, group_k=128),
                lambda: K.skip_rmsnorm(x, None, w[0].bfloat16()), lambda: K.smoothquant_matmul_prequant(x, s8, q8, s8)):
        with pytest.raises(ValueError, match="must"):
            bad()


def test_native_calls_inside_a_graph_and_on_another_stream():
    x, native, general = forms(5, 256, 256)["linear"]
    want = general(x)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = native(x)
    side.synchronize()
    assert torch.equal(got, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = native(x)
    x2 = x.flip(0).clone()
    x.copy_(x2)
    graph.replay()
    assert torch.equal(out, general(x2))


@pytest.mark.parametrize("name", ["w8a16", "w4a16", "linear", "w8a8", "quantize", "norm", "norm_quant", "swiglu"])
def test_an_allocation_that_fails_is_an_out_of_memory_error(name):
    """ModelRunner falls back to eager steps on this type.  The inputs are there before the allocator is closed to new segments,
    and every result needs one of its own (more than 10 MB)."""
    from lite_llama_b200.kernels import _native as N
    import lite_llama_b200.kernels as K

    m, n, k = 16384, 2048, 1024
    x, w = torch.ones(m, k, device="cuda", dtype=torch.float16), torch.ones(n, k, device="cuda", dtype=torch.float16)
    q8, xq, s = w.to(torch.int8), x.to(torch.int8), torch.ones(m, device="cuda")
    p = K.w4a16_pack(torch.zeros(n, k // 8, device="cuda", dtype=torch.int32), s[:1].expand(n, k // 128).contiguous(),
                     torch.zeros(n, k // 128, device="cuda"), group_size=128)
    call = {
        "w8a16": lambda: N.w8a16(x, q8, s[:n].view(n, 1), 1, k),
        "w4a16": lambda: N.w4a16_packed(x, p.qweight, p.scales, p.zeros, n, k, 128, True, False),
        "linear": lambda: N.linear(x, w),
        "w8a8": lambda: N.w8a8(xq, s, q8, s[:n], False),
        "quantize": lambda: N.quantize(x),
        "norm": lambda: N.norm(x, None, w[0], 1e-5),
        "norm_quant": lambda: N.norm_quant(x, None, w[0], 1e-5),
        "swiglu": lambda: N.swiglu(x, x),
    }[name]
    assert call() is not None
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction(1e-6)
    try:
        with pytest.raises(torch.cuda.OutOfMemoryError):
            call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert call() is not None                                          # and nothing is left behind
