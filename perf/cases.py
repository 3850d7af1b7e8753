"""The work a serving process gives this framework, as a list of measurable cases.

Every case goes through public entry points (``lite_llama_b200.kernels``, ``ModelRunner``) with the geometries of the
presets (``executor/model_config.py``) and random weights in the storage formats the kernels take.  Kinds:

``step``         one decode step of a whole (shallow) int4 model through ``ModelRunner.forward`` and its captured graph
``prompt``       one prompt pass of the same model (padded rectangle of ragged prompts), logits of the last tokens
``int4_mlp``     norm -> gate|up with the fused activation -> down, int4 weights in groups of 128
``w8_proj``      the two attention projections of a layer with 8-bit weights and 16-bit activations
``w8a8_mlp``     SmoothQuant feed-forward: 8-bit weights and per-token 8-bit activations
``dense_mlp``    the feed-forward in fp16 / bf16
``prefill_attn`` causal attention over ragged prompts
``decode_attn``  one query per sequence over the paged cache
``moe``          routing and routed SwiGLU experts, fp8 blocks or fp16

Weights of the small-token cases are stacked over several layers so that a pass reads more than the L2 cache holds,
as a decode step of the full model does.
"""

from __future__ import annotations

import math

import torch

from lite_llama_b200 import kernels as K
from lite_llama_b200.executor import ModelRunner
from lite_llama_b200.executor.decoder import DecoderWeights, LayerWeights
from lite_llama_b200.executor.model_config import PRESETS
from lite_llama_b200.kernels.quantization import interleave_gate_up
from lite_llama_b200.quantization import LinearWeights

EPS = 1e-5
GROUP = 128
LOG2E = 1.4426950408889634
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
# (hidden, intermediate) of the dense presets; the third one is the 0.5B geometry, which no tile size divides
MLPS = ((4096, 14336), (3584, 18944), (896, 4864), (4096, 12288))
# (query heads, key/value heads, head size) of the presets
HEADS = ((32, 8, 128), (28, 4, 128), (14, 2, 64), (32, 4, 128))


def listed() -> list[dict]:
    return [
        # a single user's chat: every launch of a decode step counts
        {"name": "step_int4_b1", "kind": "step", "preset": "llama-3-8b", "layers": 8, "batch": 1, "context": 200},
        # the headline serving batch, sequences of different ages
        {"name": "step_int4_b32", "kind": "step", "preset": "llama-3-8b", "layers": 8, "batch": 32, "context": 1000},
        # prompts of a new batch, padded to the longest
        {"name": "prompt_int4_4x512", "kind": "prompt", "preset": "llama-3-8b", "layers": 2, "batch": 4, "context": 512},
        # a few sequences decoding: the feed-forward alone, weight streaming
        {"name": "int4_mlp_7", "kind": "int4_mlp", "hidden": 4096, "inter": 14336, "tokens": 7, "layers": 4},
        # a long prompt batch through int4 weights: tensor-core work
        {"name": "int4_mlp_4000", "kind": "int4_mlp", "hidden": 4096, "inter": 14336, "tokens": 4000, "layers": 1},
        # fp8 checkpoint with 128 x 128 scale blocks, a medium decode batch
        {"name": "fp8_proj_64", "kind": "w8_proj", "hidden": 4096, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "format": "fp8_block", "tokens": 64, "layers": 6},
        # SmoothQuant model in continuous batching, 256 concurrent requests
        {"name": "w8a8_mlp_256", "kind": "w8a8_mlp", "hidden": 3584, "inter": 18944, "tokens": 256, "layers": 2},
        # unquantised weights, a full prompt batch
        {"name": "bf16_mlp_4096", "kind": "dense_mlp", "hidden": 4096, "inter": 14336, "tokens": 4096, "layers": 1,
         "dtype": "bf16"},
        # prompt attention, sequences of different lengths
        {"name": "prefill_attn_4x2048", "kind": "prefill_attn", "heads": 32, "kv_heads": 8, "head_dim": 128, "batch": 4,
         "context": 2048, "dtype": "fp16"},
        # decode attention over a filled cache
        {"name": "decode_attn_32x2000", "kind": "decode_attn", "heads": 32, "kv_heads": 8, "head_dim": 128, "batch": 32,
         "context": 2000, "dtype": "fp16"},
        # routed experts, decode batch: nearly every expert is read for a few rows each
        {"name": "moe_fp8_32", "kind": "moe", "hidden": 2048, "inter": 768, "experts": 128, "top_k": 8, "format": "fp8",
         "tokens": 32},
        # routed experts, prompt batch
        {"name": "moe_fp8_2000", "kind": "moe", "hidden": 2048, "inter": 768, "experts": 128, "top_k": 8, "format": "fp8",
         "tokens": 2000},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng) -> dict:
    kind = rng.choice(("step", "prompt", "int4_mlp", "int4_mlp", "w8_proj", "w8_proj", "w8a8_mlp", "dense_mlp",
                       "prefill_attn", "decode_attn", "moe", "moe"))
    if kind == "step":
        return {"kind": kind, "preset": rng.choice(("llama-3-8b", "qwen3-8b")), "layers": rng.randint(4, 8),
                "batch": _log_int(rng, 1, 64), "context": _log_int(rng, 20, 2000)}
    if kind == "prompt":
        batch = _log_int(rng, 1, 8)
        return {"kind": kind, "preset": rng.choice(("llama-3-8b", "qwen3-8b")), "layers": 2, "batch": batch,
                "context": _log_int(rng, 16, 2048 // batch)}
    if kind in ("int4_mlp", "w8a8_mlp", "dense_mlp"):
        hidden, inter = rng.choice(MLPS)
        tokens = _log_int(rng, 1, 3000)
        case = {"kind": kind, "hidden": hidden, "inter": inter, "tokens": tokens, "layers": 1 if tokens > 500 else 2}
        if kind == "dense_mlp":
            case["dtype"] = rng.choice(("fp16", "bf16"))
        return case
    if kind == "w8_proj":
        hidden = rng.choice((4096, 3584, 2048))
        tokens = _log_int(rng, 1, 3000)
        heads, kv_heads, head_dim = rng.choice((HEADS[0], HEADS[1], HEADS[3]))
        return {"kind": kind, "hidden": hidden, "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim,
                "format": rng.choice(("fp8_block", "fp8_channel", "int8_channel")), "tokens": tokens,
                "layers": 1 if tokens > 500 else 4}
    if kind == "moe":
        return {"kind": kind, "hidden": 2048, "inter": 768, "experts": rng.choice((64, 128)),
                "top_k": rng.choice((4, 8)), "format": rng.choice(("fp8", "fp8", "fp16")), "tokens": _log_int(rng, 1, 2000)}
    heads, kv_heads, head_dim = rng.choice(HEADS)
    case = {"kind": kind, "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim}
    if kind == "prefill_attn":
        case["batch"] = _log_int(rng, 1, 16)
        case["context"] = _log_int(rng, 16, 8000 // case["batch"])
    else:
        case["batch"] = _log_int(rng, 1, 64)
        case["context"] = _log_int(rng, 16, min(8000, 64000 // case["batch"]))
    case["dtype"] = rng.choice(("fp16", "bf16"))
    return case


# ------------------------------------------------------------------------------------------------ raw tensors
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, *shape, std=1.0, dtype=torch.float16) -> torch.Tensor:
    return torch.empty(shape, device="cuda", dtype=torch.float32).normal_(0.0, std, generator=gen).to(dtype)


def _norm_weight(gen, n: int, dtype) -> torch.Tensor:
    return (1.0 + _normal(gen, n, std=0.1, dtype=torch.float32)).to(dtype)


def _int4(gen, n: int, k: int):
    """An int4 checkpoint tensor: (qweight [n, k/8] int32, scales, zeros fp32 [n, k/128]) of normal weights."""
    w = torch.empty((n, k // GROUP, GROUP), device="cuda").normal_(0.0, 0.02, generator=gen)
    lo, hi = torch.aminmax(w, dim=-1)
    scale = (hi - lo) / 15.0
    zero = (-lo / scale).round().clamp_(0, 15)
    codes = w.div_(scale[..., None]).add_(zero[..., None]).round_().clamp_(0, 15).to(torch.int32).view(n, k // 8, 8)
    q = codes[..., 0].clone()
    for j in range(1, 8):
        q |= codes[..., j] << (4 * j)
    return q, scale.contiguous(), zero.contiguous()


def _int4_exact(raw) -> torch.Tensor:
    q, s, z = raw
    n = q.shape[0]
    codes = torch.stack([(q >> (4 * j)) & 15 for j in range(8)], dim=-1).view(n, -1, GROUP)
    return ((codes - z.double()[..., None]) * s.double()[..., None]).view(n, -1)


def _w8(gen, n: int, k: int, fmt: str):
    """(qweight, scales, group_n, group_k)"""
    if fmt == "fp8_block":
        q = _normal(gen, n, k, std=60.0, dtype=torch.float32).clamp_(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        s = torch.empty(((n + 127) // 128, (k + 127) // 128), device="cuda").uniform_(2e-4, 5e-4, generator=gen)
        return q, s, 128, 128
    s = torch.empty((n, 1), device="cuda").uniform_(2e-4, 5e-4, generator=gen)
    w = _normal(gen, n, k, std=40.0, dtype=torch.float32)
    if fmt == "fp8_channel":
        return w.clamp_(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8), s, 1, k
    return w.round_().clamp_(-127, 127).to(torch.int8), s, 1, k


def _w8_exact(q: torch.Tensor, s: torch.Tensor, gn: int, gk: int) -> torch.Tensor:
    w = (q.view(torch.float8_e4m3fn) if q.dtype == torch.uint8 else q).double()
    n, k = w.shape[-2:]
    s = s.double().repeat_interleave(gn, dim=-2).repeat_interleave(gk, dim=-1)
    return w * s[..., :n, :k]


def _raw_mlp(case: dict, seed: int) -> dict:
    """What an MLP stack is made of, in the formats a checkpoint has."""
    gen = _gen(seed)
    h, i, dt = case["hidden"], case["inter"], DTYPES[case.get("dtype", "fp16")]
    layers = []
    for _ in range(case["layers"]):
        norm = _norm_weight(gen, h, dt)
        if case["kind"] == "int4_mlp":
            layers.append((norm, _int4(gen, 2 * i, h), _int4(gen, h, i)))
        elif case["kind"] == "w8a8_mlp":
            layers.append((norm, _w8(gen, 2 * i, h, "int8_channel"), _w8(gen, h, i, "int8_channel")))
        else:
            layers.append((norm, _normal(gen, 2 * i, h, std=0.02, dtype=dt), _normal(gen, h, i, std=0.02, dtype=dt)))
    return {"layers": layers, "x": _normal(gen, case["tokens"], h, dtype=dt), "res": _normal(gen, case["tokens"], h, dtype=dt)}


def _raw_proj(case: dict, seed: int) -> dict:
    gen = _gen(seed)
    q = case["heads"] * case["head_dim"]
    rows = q + 2 * case["kv_heads"] * case["head_dim"]
    layers = [(_w8(gen, rows, case["hidden"], case["format"]), _w8(gen, case["hidden"], q, case["format"]))
              for _ in range(case["layers"])]
    return {"layers": layers, "x": [_normal(gen, case["tokens"], case["hidden"]) for _ in layers],
            "a": [_normal(gen, case["tokens"], q) for _ in layers]}


def _lengths(case: dict) -> list[int]:
    """Ragged sequence lengths: the longest is ``context``, the others go down to half of it."""
    b, c = case["batch"], case["context"]
    return [c - (i * (c - c // 2)) // b for i in range(b)]


def _raw_attn(case: dict, seed: int) -> dict:
    gen = _gen(seed)
    dt, b, c = DTYPES[case["dtype"]], case["batch"], case["context"]
    hq, hk, d = case["heads"], case["kv_heads"], case["head_dim"]
    lens = torch.tensor(_lengths(case), device="cuda", dtype=torch.int32)
    raw = {"lens": lens, "scale": 1.0 / math.sqrt(d)}
    if case["kind"] == "prefill_attn":           # prompts back to back
        raw["qkv"] = _normal(gen, sum(_lengths(case)), (hq + 2 * hk) * d, dtype=dt)
        raw["start"] = (lens.cumsum(0) - lens).to(torch.int32)
    else:                                        # rows of a sequence lie in a run, as the row allocator hands them out
        raw["table"] = torch.arange(b * c, device="cuda", dtype=torch.int32).view(b, c)
        raw["pool"] = _normal(gen, b * c, 2 * hk, d, dtype=dt)
        raw["q"] = _normal(gen, b, hq, d, dtype=dt)
        raw["slots"] = torch.arange(b, device="cuda", dtype=torch.int32)
    return raw


def _raw_moe(case: dict, seed: int) -> dict:
    gen = _gen(seed)
    e, h, i, t = case["experts"], case["hidden"], case["inter"], case["tokens"]
    if case["format"] == "fp8":
        w1 = _normal(gen, e, 2 * i, h, std=60.0, dtype=torch.float32).to(torch.float8_e4m3fn).view(torch.uint8)
        w2 = _normal(gen, e, h, i, std=60.0, dtype=torch.float32).to(torch.float8_e4m3fn).view(torch.uint8)
        s1 = torch.empty((e, 2 * i // 128, h // 128), device="cuda").uniform_(2e-4, 5e-4, generator=gen)
        s2 = torch.empty((e, h // 128, i // 128), device="cuda").uniform_(2e-4, 5e-4, generator=gen)
    else:
        w1, w2, s1, s2 = _normal(gen, e, 2 * i, h, std=0.02), _normal(gen, e, h, i, std=0.02), None, None
    # logits: every token ranks the experts, some experts are more popular; no two equal, so the choice has one answer
    pref = _normal(gen, t, e, dtype=torch.float32) + _normal(gen, 1, e, std=0.3, dtype=torch.float32)
    logits = (pref.argsort(-1).argsort(-1).float() * (6.0 / e)).half()
    return {"w1": w1, "w2": w2, "s1": s1, "s2": s2, "logits": logits, "x": _normal(gen, t, h)}


def _raw_model(case: dict, seed: int) -> dict:
    cfg = PRESETS[case["preset"]].with_(num_layers=case["layers"], max_seq_len=max(64, case["context"] + 8))
    gen = _gen(seed)
    h = cfg.hidden_size
    layers = []
    for _ in range(cfg.num_layers):
        layers.append({
            "in_norm": _norm_weight(gen, h, torch.float16), "post_norm": _norm_weight(gen, h, torch.float16),
            "qkv": _int4(gen, cfg.q_size + 2 * cfg.kv_size, h), "o": _int4(gen, h, cfg.q_size),
            "gate_up": _int4(gen, 2 * cfg.intermediate_size, h), "down": _int4(gen, h, cfg.intermediate_size),
            "q_norm": _norm_weight(gen, cfg.head_dim, torch.float16) if cfg.use_qk_norm else None,
            "k_norm": _norm_weight(gen, cfg.head_dim, torch.float16) if cfg.use_qk_norm else None})
    b, c = case["batch"], case["context"]
    lens = torch.tensor(_lengths(case), device="cuda", dtype=torch.int32)
    raw = {"cfg": cfg, "layers": layers, "embed": _normal(gen, cfg.vocab_size, h, std=0.5),
           "head": _normal(gen, cfg.vocab_size, h, std=0.02), "norm": _norm_weight(gen, h, torch.float16), "lens": lens}
    width = c if case["kind"] == "prompt" else 1
    raw["ids"] = torch.randint(0, cfg.vocab_size, (b, width), device="cuda", generator=gen)
    if case["kind"] == "step":          # the cache as the prompts left it: rotated keys | values of every earlier token
        raw["cache"] = [_normal(gen, b, c, 2 * cfg.num_kv_heads, cfg.head_dim) for _ in layers]
    return raw


# ------------------------------------------------------------------------------------------------ prepare and run
def _linear4(raw, swiglu: bool = False) -> LinearWeights:
    n, k = raw[0].shape[0], raw[0].shape[1] * 8
    parts = [interleave_gate_up(t) for t in raw] if swiglu else raw
    return LinearWeights("int4", n, k, group_size=GROUP, packed=K.w4a16_pack(*parts, group_size=GROUP), swiglu=swiglu)


def _runner(case: dict, raw: dict) -> dict:
    cfg, b, c = raw["cfg"], case["batch"], case["context"]
    layers = [LayerWeights(input_norm=l["in_norm"], post_norm=l["post_norm"], qkv=_linear4(l["qkv"]), o=_linear4(l["o"]),
                           gate_up=_linear4(l["gate_up"], swiglu=True), down=_linear4(l["down"]), q_norm=l["q_norm"],
                           k_norm=l["k_norm"]) for l in raw["layers"]]
    weights = DecoderWeights(embed=raw["embed"], lm_head=raw["head"], final_norm=raw["norm"], layers=layers)
    runner = ModelRunner(cfg, weights, (b + 1) * cfg.max_seq_len)
    slots = torch.arange(b, device="cuda", dtype=torch.int32)
    state = {"kind": case["kind"], "runner": runner, "ids": raw["ids"]}
    if case["kind"] == "prompt":
        runner.prefill_alloc_kv_cache(c, raw["lens"], slots)
        state["positions"] = torch.arange(c, device="cuda").expand(b, c).contiguous()
        state["last"] = (raw["lens"] - 1).long()
        return state
    runner.enable_cuda_graph((b,), (cfg.max_seq_len,))
    # a prompt of lens - 1 tokens has run; this step's token is the last of lens
    rows = runner.prefill_alloc_kv_cache(c, raw["lens"] - 1, slots)
    for pool, cache in zip(runner.kv_cache_manager.gpu_kv_buffer, raw["cache"]):
        pool[rows.long()] = cache.view(b * c, 2 * cfg.num_kv_heads, cfg.head_dim)
    runner.decode_alloc_kv_cache(b)
    state["positions"] = (raw["lens"].long() - 1).unsqueeze(1)
    return state


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("step", "prompt"):
        return _runner(case, _raw_model(case, seed))
    if kind == "int4_mlp":
        raw = _raw_mlp(case, seed)
        raw["layers"] = [(n, _linear4(gu, swiglu=True).packed, _linear4(dn).packed) for n, gu, dn in raw["layers"]]
    elif kind in ("w8a8_mlp", "dense_mlp"):
        raw = _raw_mlp(case, seed)
    elif kind == "w8_proj":
        raw = _raw_proj(case, seed)
    elif kind == "moe":
        raw = _raw_moe(case, seed)
    else:
        raw = _raw_attn(case, seed)
        hq, hk, d = case["heads"], case["kv_heads"], case["head_dim"]
        if kind == "prefill_attn":
            raw["q"], raw["k"], raw["v"] = (t.unflatten(1, (-1, d)) for t in raw.pop("qkv").split([hq * d, hk * d, hk * d], 1))
        else:
            raw["k"], raw["v"] = raw["pool"][:, :hk], raw["pool"][:, hk:]
    return {**case, **raw}


def run(s):
    kind = s["kind"]
    if kind == "step":
        return s["runner"].forward(s["ids"], s["positions"])
    if kind == "prompt":
        return s["runner"].forward(s["ids"], s["positions"], last_token_index=s["last"])
    if kind == "w8_proj":
        out = []
        for ((wq, sq, gn, gk), (wo, so, on, ok)), x, a in zip(s["layers"], s["x"], s["a"]):
            out.append(K.w8a16_matmul(x, wq, sq, group_n=gn, group_k=gk))
            out.append(K.w8a16_matmul(a, wo, so, group_n=on, group_k=ok))
        return out
    if kind == "prefill_attn":
        return K.flash_attention2_no_pad(s["q"], s["k"], s["v"], s["scale"] * LOG2E, s["start"], s["lens"], s["context"])
    if kind == "decode_attn":
        return K.flash_decoding(s["q"], s["k"], s["v"], s["scale"], s["table"], s["slots"], s["lens"], s["context"])
    if kind == "moe":
        weights, ids = K.route_topk(s["logits"], s["top_k"])
        return K.fused_moe(s["x"], s["w1"], s["w2"], weights, ids, w1_scale=s["s1"], w2_scale=s["s2"],
                           group_n=128 if s["s1"] is not None else 0, group_k=128 if s["s1"] is not None else 0)
    x, residual = s["x"], s["res"].clone()             # the residual stream is updated in place
    for norm, gate_up, down in s["layers"]:
        if kind == "int4_mlp":
            h, residual = K.skip_rmsnorm(x, residual, norm, EPS)
            x = K.w4a16_matmul_packed(K.w4a16_matmul_packed(h, gate_up, swiglu=True), down)
        elif kind == "w8a8_mlp":
            q, scales, residual = K.skip_rmsnorm_quant_int8(x, residual, norm, EPS)
            wide = K.smoothquant_matmul_prequant(q, scales, gate_up[0], gate_up[1])
            x = K.smoothquant_matmul(K.swiglu_forward(wide[:, :s["inter"]], wide[:, s["inter"]:]), down[0], down[1])
        else:
            h, residual = K.skip_rmsnorm(x, residual, norm, EPS)
            wide = K.linear(h, gate_up)
            x = K.linear(K.swiglu_forward(wide[:, :s["inter"]], wide[:, s["inter"]:]), down)
    return x, residual


# ------------------------------------------------------------------------------------------------ what a pass needs
def _active_experts(case: dict) -> float:
    return case["experts"] * (1.0 - (1.0 - case["top_k"] / case["experts"]) ** case["tokens"])


def _int4_bytes(n: int, k: int) -> float:
    return n * k / 2 + n * (k // GROUP) * 8


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("step", "prompt"):
        cfg = PRESETS[case["preset"]]
        b, n, lens = case["batch"], case["layers"], _lengths(case)
        t = sum(lens) if kind == "prompt" else b
        shapes = ((cfg.q_size + 2 * cfg.kv_size, cfg.hidden_size), (cfg.hidden_size, cfg.q_size),
                  (2 * cfg.intermediate_size, cfg.hidden_size), (cfg.hidden_size, cfg.intermediate_size))
        head = cfg.vocab_size * cfg.hidden_size
        weights = n * sum(_int4_bytes(*s) for s in shapes) + 2 * head
        flops = 2.0 * t * n * sum(x * y for x, y in shapes) + 2.0 * b * head
        kv_row = 2 * cfg.kv_size * 2
        kv = n * sum(lens) * kv_row
        flops += 4.0 * n * sum(lens) * cfg.q_size if kind == "step" else 2.0 * n * sum(m * m for m in lens) * cfg.q_size
        return {"bytes": weights + kv + 2.0 * b * cfg.vocab_size + 2.0 * t * cfg.hidden_size, "flops": flops}
    if kind in ("int4_mlp", "w8a8_mlp", "dense_mlp"):
        h, i, t, n = case["hidden"], case["inter"], case["tokens"], case["layers"]
        per = {"int4_mlp": _int4_bytes(2 * i, h) + _int4_bytes(h, i), "w8a8_mlp": 3.0 * h * i + 4 * (2 * i + h),
               "dense_mlp": 6.0 * h * i}[kind]
        return {"bytes": n * per + 4 * 2.0 * t * h, "flops": 6.0 * n * t * h * i}
    if kind == "w8_proj":
        q = case["heads"] * case["head_dim"]
        rows, h, t, n = q + 2 * case["kv_heads"] * case["head_dim"], case["hidden"], case["tokens"], case["layers"]
        return {"bytes": n * (rows * h + h * q + 2.0 * t * (2 * h + rows + q)), "flops": 2.0 * n * t * h * (rows + q)}
    if kind == "moe":
        e, h, i, t = _active_experts(case), case["hidden"], case["inter"], case["tokens"]
        return {"bytes": e * 3.0 * h * i * (1 if case["format"] == "fp8" else 2) + 4.0 * t * h,
                "flops": 6.0 * t * case["top_k"] * h * i}
    lens, t = _lengths(case), sum(_lengths(case))
    q, kv = case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"]
    if kind == "prefill_attn":
        return {"bytes": 2.0 * t * (2 * q + 2 * kv), "flops": 2.0 * sum(n * n for n in lens) * q}
    return {"bytes": 2.0 * t * 2 * kv + 4.0 * case["batch"] * q, "flops": 4.0 * t * q}


def tolerance(case: dict):
    """About four times what the path is off its 64-bit result: activations are rounded to 16 bits between the ops."""
    kind = case["kind"]
    if kind in ("step", "prompt"):                     # 1.4e-3 to 2.2e-3
        return {"rel": 1e-2}
    bf = case.get("dtype") == "bf16"
    if kind in ("prefill_attn", "decode_attn"):        # 2.5e-4 in fp16, eight times that in bf16
        return {"rel": 8e-3 if bf else 1e-3}
    if kind == "w8a8_mlp":                             # activations cut to 8 bits: one ulp before the cut can move a step
        return {"rel": 2e-2}
    if kind == "w8_proj":                              # 2.1e-4: the rounding of the result
        return {"rel": 8e-4}
    if kind == "dense_mlp":
        return {"rel": 2e-2 if bf else 2.5e-3 * math.sqrt(case["layers"])}
    return {"rel": 2.5e-3 * math.sqrt(case.get("layers", 1))}      # 6e-4 a layer, 5e-4 for the experts


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x: torch.Tensor, w: torch.Tensor, eps: float = EPS) -> torch.Tensor:
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _silu_mul(wide: torch.Tensor) -> torch.Tensor:
    g, u = wide.chunk(2, dim=-1)
    return torch.nn.functional.silu(g) * u


def _int8_rows(x: torch.Tensor):
    """Per-row 8-bit activations, rounded towards zero (the stored format of SmoothQuant's dynamic scheme)."""
    scale = x.abs().amax(-1, keepdim=True) / 127.0
    return (x / scale).trunc(), scale


def _exact_attn(q, k, v, scale, causal_from: int | None):
    """``q [n, hq, d]``, ``k`` / ``v [m, hk, d]``; query row r sees keys up to ``causal_from + r`` (None: all)."""
    n, hq, d = q.shape
    m, hk, _ = k.shape
    q = q.view(n, hk, hq // hk, d).permute(1, 2, 0, 3)
    s = q @ k.permute(1, 2, 0)[:, None] * scale
    if causal_from is not None:
        rows, cols = torch.arange(n, device=q.device)[:, None], torch.arange(m, device=q.device)[None, :]
        s = s.masked_fill(cols > rows + causal_from, float("-inf"))
    return (s.softmax(-1) @ v.permute(1, 0, 2)[:, None]).permute(2, 0, 1, 3).reshape(n, hq, d)


def _rope(x: torch.Tensor, pos: torch.Tensor, theta: float) -> torch.Tensor:
    d = x.shape[-1]
    freq = theta ** (-torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    ang = pos.double()[:, None, None] * freq
    a, b = x.chunk(2, -1)
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1)


def _exact_model(case: dict, seed: int):
    raw = _raw_model(case, seed)
    cfg, lens, ids = raw["cfg"], raw["lens"].tolist(), raw["ids"]
    hq, hk, d, eps = cfg.num_heads, cfg.num_kv_heads, cfg.head_dim, cfg.rms_norm_eps
    prompt = case["kind"] == "prompt"
    spans, at = [], 0
    for n in lens:                                     # rows of each sequence among the tokens of this pass
        w = n if prompt else 1
        spans.append((at, at + w))
        at += w
    tok = torch.cat([ids[i, :e - a] for i, (a, e) in enumerate(spans)])
    pos = torch.cat([torch.arange(n, device="cuda") if prompt else torch.tensor([n - 1], device="cuda") for n in lens])
    x = raw["embed"][tok].double()
    for li, l in enumerate(raw["layers"]):
        qkv = _rms(x, l["in_norm"], eps) @ _int4_exact(l["qkv"]).T
        q, k, v = (t.unflatten(1, (-1, d)) for t in qkv.split([cfg.q_size, cfg.kv_size, cfg.kv_size], 1))
        if l["q_norm"] is not None:
            q, k = _rms(q, l["q_norm"], eps), _rms(k, l["k_norm"], eps)
        q, k = _rope(q, pos, cfg.rope_theta), _rope(k, pos, cfg.rope_theta)
        outs = []
        for i, (a, e) in enumerate(spans):
            kk, vv = k[a:e], v[a:e]
            if not prompt:
                past = raw["cache"][li][i, :lens[i] - 1].double()
                kk, vv = torch.cat([past[:, :hk], kk]), torch.cat([past[:, hk:], vv])
            outs.append(_exact_attn(q[a:e], kk, vv, 1.0 / math.sqrt(d), 0 if prompt else None))
        x = x + torch.cat(outs).flatten(1) @ _int4_exact(l["o"]).T
        x = x + _silu_mul(_rms(x, l["post_norm"], eps) @ _int4_exact(l["gate_up"]).T) @ _int4_exact(l["down"]).T
    last = x[[e - 1 for _, e in spans]]
    return (_rms(last, raw["norm"], eps) @ raw["head"].double().T).unsqueeze(1)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("step", "prompt"):
        return _exact_model(case, seed)
    if kind in ("int4_mlp", "w8a8_mlp", "dense_mlp"):
        raw = _raw_mlp(case, seed)
        x, res = raw["x"].double(), raw["res"].double()
        for norm, gu, dn in raw["layers"]:
            res = res + x
            h = _rms(res, norm)
            if kind == "int4_mlp":
                x = _silu_mul(h @ _int4_exact(gu).T) @ _int4_exact(dn).T
            elif kind == "dense_mlp":
                x = _silu_mul(h @ gu.double().T) @ dn.double().T
            else:
                q, s = _int8_rows(h)
                q, s = _int8_rows(_silu_mul((q @ gu[0].double().T) * s * gu[1].double().T))
                x = (q @ dn[0].double().T) * s * dn[1].double().T
        return x, res
    if kind == "w8_proj":
        raw, out = _raw_proj(case, seed), []
        for (qkv, o), x, a in zip(raw["layers"], raw["x"], raw["a"]):
            out += [x.double() @ _w8_exact(*qkv).T, a.double() @ _w8_exact(*o).T]
        return out
    if kind == "moe":
        raw = _raw_moe(case, seed)
        p = raw["logits"].double().softmax(-1)
        w, ids = p.topk(case["top_k"], dim=-1)
        w = w / w.sum(-1, keepdim=True)
        x = raw["x"].double()
        out = torch.zeros_like(x)
        for e in range(case["experts"]):
            t, slot = (ids == e).nonzero(as_tuple=True)
            if t.numel() == 0:
                continue
            w1, w2 = ((raw[n][e].double() if raw[s] is None else _w8_exact(raw[n][e], raw[s][e], 128, 128))
                      for n, s in (("w1", "s1"), ("w2", "s2")))
            out.index_add_(0, t, (_silu_mul(x[t] @ w1.T) @ w2.T) * w[t, slot][:, None])
        return out
    raw = _raw_attn(case, seed)
    hq, hk, d = case["heads"], case["kv_heads"], case["head_dim"]
    lens = _lengths(case)
    if kind == "decode_attn":
        return torch.cat([_exact_attn(raw["q"][i:i + 1].double(), kv[:, :hk], kv[:, hk:], raw["scale"], None)
                          for i, n in enumerate(lens) for kv in (raw["pool"][raw["table"][i, :n].long()].double(),)])
    q, k, v = (t.unflatten(1, (-1, d)) for t in raw["qkv"].split([hq * d, hk * d, hk * d], 1))
    return torch.cat([_exact_attn(*parts, raw["scale"], 0)
                      for parts in zip(*(t.double().split(lens) for t in (q, k, v)))])
