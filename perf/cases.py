"""The work that a user of this package has it do, as cases that can be timed and compared.

Every case goes through the calls a program makes: an NVFP4 Linear module, ``quantize_to_fp4``, the
KV-cache helpers, the chunk attention, the causal DiT's forward, the scheduler.  Sizes are those of
the 5B-shaped causal DiT this package serves (dim 3072, 24 heads of 128, FFN 14336, 880 tokens per
latent frame, 3-frame chunks, 15-frame window, 512 text tokens), of its token and head shards under
sequence parallelism, and of the test suite's reduced configurations; ``draw`` spreads over the
ranges in between.
"""
import math

import torch
import torch.nn as nn

import longlive_b200 as L
from longlive_b200 import dit, ops
from longlive_b200.scheduler import FlowUniPCMultistepScheduler

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # A handful of rows through a projection: the latency of one module call (quantize + GEMM) without work behind it.
        {"name": "linear_17x3072x3072", "kind": "linear", "m": 17, "k": 3072, "n": 3072, "bias": True},
        # One chunk (3 latent frames) through an attention projection: the most frequent Linear of the model.
        {"name": "linear_2640x3072x3072", "kind": "linear", "m": 2640, "k": 3072, "n": 3072, "bias": True},
        # FFN-down over 12 latent frames: the largest Linear (long K, many tokens).
        {"name": "linear_10560x14336x3072", "kind": "linear", "m": 10560, "k": 14336, "n": 3072, "bias": True},
        # The FFN hidden of one chunk through the quantizer alone (a program that runs its own GEMMs or ships activations).
        {"name": "quantize_2640x14336", "kind": "quantize", "m": 2640, "k": 14336, "dtype": "bf16", "rule": "mse"},
        # The KV-cache write of one layer: keys and values of a chunk into their persistent slots.
        {"name": "kv_write_2640x24", "kind": "kv_write", "tokens": 2640, "heads": 24, "rule": "mse"},
        # The cached part of a layer's window as bf16 (callers with an attention of their own).
        {"name": "kv_dequant_4x2640x24", "kind": "kv_dequant", "blocks": 4, "tokens": 2640, "heads": 24, "dtype": "bf16"},
        # Self-attention of a chunk over the full window: 4 cached NVFP4 blocks and the chunk itself.
        {"name": "window_2640x4x24", "kind": "window", "q": 2640, "blocks": 4, "tokens": 2640, "cur": 2640, "heads": 24},
        # The same for one rank of four (6 heads), early in a video: 2 cached blocks.
        {"name": "window_2640x2x6", "kind": "window", "q": 2640, "blocks": 2, "tokens": 2640, "cur": 2640, "heads": 6},
        # Cross-attention of a chunk to the 512 text tokens.
        {"name": "cross_2640x512x24", "kind": "cross", "q": 2640, "keys": 512, "heads": 24},
        # A denoising step (forward and scheduler step) of the whole 30-layer model in the steady state of a streaming rollout,
        # its launches captured in a graph: four of these and a clean forward make a chunk.
        {"name": "denoise_30_layers", "kind": "denoise", "layers": 30, "dim": 3072, "ffn": 14336, "heads": 24, "grid_h": 22, "grid_w": 40,
         "blocks": 5, "past": 4, "text": 512, "graphs": True},
        # The same step of a small image through two layers, launched kernel by kernel (window still filling): the host side of it.
        {"name": "denoise_2_layers_eager", "kind": "denoise", "layers": 2, "dim": 3072, "ffn": 14336, "heads": 24, "grid_h": 11, "grid_w": 20,
         "blocks": 3, "past": 1, "text": 512, "graphs": False},
        # What surrounds the forwards of a chunk: noise to tokens, four scheduler steps, tokens to the latent handed off.
        {"name": "sampler_3x44x80", "kind": "sampler", "channels": 48, "frames": 3, "height": 44, "width": 80, "steps": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "quantize", "quantize", "kv_write", "kv_dequant", "window", "window", "window", "cross",
                       "denoise", "denoise", "sampler"])
    if kind == "linear":
        wide = [256 * rng.randint(1, 56), 256 * rng.randint(1, 16), 3072, 3072]
        return {"kind": kind, "m": _log(rng, 1, 10560), "k": rng.choice(wide), "n": rng.choice([64 * rng.randint(2, 224), 3072, 3072, 14336]),
                "bias": rng.random() < 0.8}
    if kind == "quantize":
        return {"kind": kind, "m": _log(rng, 1, 10560), "k": rng.choice([64 * rng.randint(1, 224), 3072, 14336]),
                "dtype": rng.choice(["bf16", "bf16", "bf16", "fp16"]), "rule": rng.choice(["mse", "mse", "mse", "mae", "abs_max", "static_6", "static_4"])}
    if kind == "kv_write":
        return {"kind": kind, "tokens": _log(rng, 128, 2640), "heads": rng.choice([1, 2, 3, 6, 12, 24]), "rule": rng.choice(["mse", "mse", "static_6"])}
    if kind == "kv_dequant":
        return {"kind": kind, "blocks": rng.randint(1, 8), "tokens": _log(rng, 128, 2640), "heads": rng.choice([2, 3, 6, 12, 24]),
                "dtype": rng.choice(["bf16", "bf16", "fp16", "fp32"])}
    if kind == "window":
        t = _log(rng, 144, 2640)
        return {"kind": kind, "q": t, "blocks": rng.randint(0, 5), "tokens": t, "cur": t, "heads": rng.choice([2, 3, 6, 12, 24, 24])}
    if kind == "cross":
        return {"kind": kind, "q": _log(rng, 48, 5280), "keys": rng.choice([512, 512, rng.randint(16, 512)]), "heads": rng.choice([2, 8, 12, 24, 24])}
    if kind == "denoise":
        graphs = rng.random() < 0.5
        dim, ffn, heads = rng.choice([(3072, 14336, 24), (2048, 8192, 16), (1024, 4096, 8)])
        blocks = rng.randint(2, 5)
        return {"kind": kind, "layers": rng.randint(1, 8) if graphs else rng.randint(1, 3), "dim": dim, "ffn": ffn, "heads": heads,
                "grid_h": rng.randint(6, 22), "grid_w": rng.randint(8, 40), "blocks": blocks, "past": blocks - 1 if graphs else rng.randint(1, blocks - 1),
                "text": 512, "graphs": graphs}
    return {"kind": kind, "channels": rng.choice([16, 48]), "frames": rng.randint(1, 6), "height": 2 * rng.randint(4, 44), "width": 2 * rng.randint(4, 80),
            "steps": rng.randint(1, 8)}


# ---- states ---------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _activation(g, m, k, dtype=torch.bfloat16):
    """N(0, 1) with 0.1 % of the entries scaled by 20: activations with outliers."""
    x = torch.randn(m, k, generator=g, device=DEV)
    return torch.where(torch.rand(m, k, generator=g, device=DEV) < 1e-3, x * 20, x).to(dtype)


def _kv_blocks(g, n, tokens, heads):
    cfg = L.QuantizationConfig(scale_rule="mse")
    return [L.quantize_to_fp4(torch.randn(tokens * heads, 128, generator=g, device=DEV).bfloat16(), cfg) for _ in range(n)]


def _scheduler():
    return FlowUniPCMultistepScheduler(num_train_timesteps=1000, shift=1, use_dynamic_shifting=False)


def _prepare_linear(c, g):
    model = nn.Sequential(nn.Linear(c["k"], c["n"], bias=c["bias"], device=DEV, dtype=torch.bfloat16))
    with torch.no_grad():
        model[0].weight.copy_(torch.randn(c["n"], c["k"], generator=g, device=DEV) * 0.02)
        if c["bias"]:
            model[0].bias.copy_(torch.randn(c["n"], generator=g, device=DEV) * 0.02)
    L.quantize_model_with_filter(model, materialize_for_inference=True, verbose=False)
    return {"model": model.requires_grad_(False), "x": _activation(g, c["m"], c["k"]).unsqueeze(0)}


def _prepare_quantize(c, g):
    return {"x": _activation(g, c["m"], c["k"], DTYPES[c["dtype"]]), "config": L.QuantizationConfig(scale_rule=c["rule"])}


def _prepare_kv_write(c, g):
    rows = c["tokens"] * c["heads"]
    cfg = L.QuantizationConfig(scale_rule=c["rule"])
    k, v = (torch.randn(rows, 128, generator=g, device=DEV).bfloat16() for _ in range(2))
    return {"k": k, "v": v, "config": cfg, "slots": [L.quantize_to_fp4(torch.zeros_like(k), cfg) for _ in range(2)]}


def _prepare_kv_dequant(c, g):
    return {"k": _kv_blocks(g, c["blocks"], c["tokens"], c["heads"]), "v": _kv_blocks(g, c["blocks"], c["tokens"], c["heads"])}


def _prepare_window(c, g):
    bf = lambda n: torch.randn(n, c["heads"] * 128, generator=g, device=DEV).bfloat16()
    return {"k": _kv_blocks(g, c["blocks"], c["tokens"], c["heads"]), "v": _kv_blocks(g, c["blocks"], c["tokens"], c["heads"]),
            "q": bf(c["q"]), "k_cur": bf(c["cur"]), "v_cur": bf(c["cur"])}


def _prepare_cross(c, g):
    bf = lambda n: torch.randn(n, c["heads"] * 128, generator=g, device=DEV).bfloat16()
    return {"q": bf(c["q"]), "k": bf(c["keys"]), "v": bf(c["keys"])}


def _prepare_denoise(c, g):
    """A model in the middle of a rollout: ``past`` chunks cached by clean forwards, the next one begun, and one denoising
    step of it done (which captures the graph the others replay)."""
    cfg = dit.DiTConfig(dim=c["dim"], ffn_dim=c["ffn"], heads=c["heads"], layers=c["layers"], text_len=c["text"], grid_h=c["grid_h"],
                        grid_w=c["grid_w"], frames_per_chunk=3, window_frames=3 * c["blocks"], sink_frames=3)
    model = dit.CausalDiT(cfg, seed=g.initial_seed(), use_graphs=c["graphs"])
    bf = lambda *shape: torch.randn(*shape, generator=g, device=DEV).bfloat16()
    ctx = model.encode_text(bf(cfg.text_len, cfg.text_dim))
    clean = torch.zeros(3, device=DEV)
    for chunk in range(c["past"]):
        model.cache.begin_chunk()
        model.forward(bf(cfg.chunk_tokens, cfg.patch_dim), clean, ctx, 3 * chunk, t_key=(0.0,) * 3)
    model.cache.begin_chunk()
    s = {"model": model, "x": bf(cfg.chunk_tokens, cfg.patch_dim), "ctx": ctx, "frame": 3 * c["past"], "scheduler": _scheduler()}
    _run_denoise(c, s)
    return s


def _prepare_sampler(c, g):
    f, h, w, ch = c["frames"], c["height"] // 2, c["width"] // 2, c["channels"]
    bf = lambda *shape: torch.randn(*shape, generator=g, device=DEV).bfloat16()
    return {"noise": bf(ch, f, 2 * h, 2 * w), "flows": [bf(f * h * w, 4 * ch) for _ in range(c["steps"])],
            "scheduler": _scheduler(),
            "out": torch.empty(ch, f, 2 * h, 2 * w, dtype=torch.bfloat16, device=DEV)}


def prepare(case, seed):
    return {"case": case, **globals()["_prepare_" + case["kind"]](case, _gen(seed))}


# ---- one pass -------------------------------------------------------------------------------------

def _parts(q):
    return q.values, q.scale_factors.view(torch.uint8), q.amax


def _run_linear(c, s):
    return s["model"](s["x"])


def _run_quantize(c, s):
    return _parts(L.quantize_to_fp4(s["x"], s["config"]))


def _run_kv_write(c, s):
    return [_parts(L.quantize_to_fp4(s[name], s["config"], out=slot)) for name, slot in zip("kv", s["slots"])]


def _run_kv_dequant(c, s):
    return [L.dequantize_kv_cache(s[name], c["blocks"], c["heads"], c["tokens"], DTYPES[c["dtype"]], s[name][0].device) for name in "kv"]


def _run_window(c, s):
    return ops.attention_nvfp4kv(s["q"], s["k"], s["v"], c["tokens"], s["k_cur"], s["v_cur"], c["heads"])


def _run_cross(c, s):
    return ops.attention_bf16(s["q"], s["k"], s["v"], c["heads"])


def _run_denoise(c, s):
    # the first denoising step of ``CausalDiT.run_chunk``: the cache block is left to the clean forward that ends the chunk
    sched, x = s["scheduler"], s["x"]
    sched.set_timesteps(4, device="cpu", shift=5.0)
    t = float(sched.timesteps[0])
    flow = s["model"].forward(x, torch.full((3,), t, device=DEV), s["ctx"], s["frame"], t_key=(t,) * 3, write_cache=False)
    return sched.step(flow, t, x, return_dict=False)[0]


def _run_sampler(c, s):
    x = ops.patchify(s["noise"])
    sched = s["scheduler"]
    sched.set_timesteps(c["steps"], device="cpu", shift=5.0)
    for t, flow in zip(sched.timesteps.tolist(), s["flows"]):
        x = sched.step(flow, t, x, return_dict=False)[0]
    return ops.unpatchify(x, s["out"])


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state["case"], state)


# ---- what a pass cannot do without ------------------------------------------------------------------

NVFP4 = 0.5625          # bytes of an NVFP4 value: a 4-bit code and a sixteenth of a scale byte


def work(case):
    c = case
    if c["kind"] == "linear":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2 * m * k + NVFP4 * n * k + 2 * m * n + (2 * n if c["bias"] else 0), "flops": 2 * m * n * k}
    if c["kind"] == "quantize":
        return {"bytes": (2 + NVFP4) * c["m"] * c["k"], "flops": 0}
    if c["kind"] == "kv_write":
        return {"bytes": 2 * (2 + NVFP4) * c["tokens"] * c["heads"] * 128, "flops": 0}
    if c["kind"] == "kv_dequant":
        return {"bytes": 2 * (NVFP4 + DTYPES[c["dtype"]].itemsize) * c["blocks"] * c["tokens"] * c["heads"] * 128, "flops": 0}
    if c["kind"] == "window":
        d = c["heads"] * 128
        cached = c["blocks"] * c["tokens"]
        return {"bytes": d * (4 * c["q"] + 2 * NVFP4 * cached + 4 * c["cur"]), "flops": 4 * c["q"] * (cached + c["cur"]) * d}
    if c["kind"] == "cross":
        d = c["heads"] * 128
        return {"bytes": d * 4 * (c["q"] + c["keys"]), "flops": 4 * c["q"] * c["keys"] * d}
    if c["kind"] == "denoise":
        s, d, f = 3 * c["grid_h"] * c["grid_w"], c["dim"], c["ffn"]
        cached = c["past"] * s
        per_layer = NVFP4 * (6 * d * d + 2 * d * f + 2 * cached * d) + 4 * c["text"] * d
        flops = 2 * s * (6 * d * d + 2 * d * f) + 4 * s * (cached + s + c["text"]) * d
        return {"bytes": c["layers"] * per_layer + 4 * s * 192 + 8 * 192 * d, "flops": c["layers"] * flops + 8 * s * 192 * d}
    n = c["channels"] * c["frames"] * c["height"] * c["width"]
    return {"bytes": 2 * n * (2 + c["steps"]), "flops": 0}


def tolerance(case):
    # codes, scales, dequantized values and scheduler steps are defined operation by operation
    if case["kind"] in ("quantize", "kv_write", "kv_dequant", "sampler"):
        return "exact"
    # NVFP4 operands are exact, sums are fp32, the result is rounded to bf16 once or twice
    if case["kind"] == "linear":
        return {"rel": 4e-3}
    # probabilities and outputs in bf16
    if case["kind"] in ("window", "cross"):
        return {"rel": 1e-2}
    # one bf16 ulp in front of an NVFP4 quantizer flips codes: the flow prediction of two correct implementations differs by 5 to
    # 8 percent whatever the depth, and the step takes 0.06 of it
    return {"rel": 1e-2}
