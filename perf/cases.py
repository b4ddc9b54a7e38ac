"""Timed workloads of the quantized denoising path, each run through the calls a user's program makes.

A case is a plain dict; `kind` says which entry point it goes through:

  linear      nn.QuantizedLinear.__call__ (optionally LoRA-wrapped): one layer on activations of `batch` x `rows`
  attention   ops.fmha / ops.fmha_ex: one attention call on projected q, k, v
  quantize    nn.Linear.to_quantized (encode) and QuantizedLinear.dequantize (decode): load-time work
  flux        Flux1.predict_noise + the Euler update: one denoising step of the dual / single-stream model
  zimage      ZImage.denoise_step: one step of the single-stream model
  qwen        QwenImage.denoise_step: one guidance step (prompt and negative prompt) of the dual-stream model

Model steps run at full width and depth with random-init weights; what a step costs depends on the number of
images, the picture size and the text length, which is what the cases and the draws vary.
"""
from __future__ import annotations

import math

import torch

from mflux_b200 import nn, ops
from mflux_b200.flux import Flux1, FluxConfig
from mflux_b200.lora import LoRALinear
from mflux_b200.qwen import QwenConfig, QwenImage
from mflux_b200.schedulers import LinearScheduler
from mflux_b200.zimage import ZImage, ZImageConfig

DEVICE = "cuda"


def listed() -> list[dict]:
    return [
        # Modulation linear of a single-stream block: two images' conditioning vectors, 256 wide. The smallest call
        # there is: launch latency and the host side of a call.
        _linear("modulation_w8_2rows", rows=2, n=15360, k=256, bits=8),
        # AdaLN linear of a joint block for one image: streams 28 MB of packed weights for one row.
        _linear("adaln_w4_1row", rows=1, n=18432, k=3072, bits=4),
        # Fused q/k/v projection of one prompt's text rows, an odd number of them: a few tiles, not a full GPU.
        _linear("text_qkv_w4_333rows", rows=333, n=9216, k=3072, bits=4),
        # Feed-forward input projection of one 1024x1024 image, the single-linear configuration of the benchmark.
        _linear("ffn_in_w4_4096rows", rows=4096, n=12288, k=3072, bits=4, epilogue="gelu"),
        # Gate / up projection with SwiGLU on a ragged token count (two images of 1.0 MP, odd caption), 8-bit codes.
        _linear("swiglu_w8_2x4213rows", batch=2, rows=4213, n=20480, k=3840, bits=8, epilogue="swiglu", bias=False),
        # Output projection of a single-stream block with a rank-16 adapter and the gated residual on the float32
        # stream: how a fine-tuned style runs.
        _linear("lora_out_w4_4608rows", rows=4608, n=3072, k=15360, bits=4, epilogue="gate_residual", lora=16),
        # Joint attention of one 1024x1024 image: 4096 image + 512 text tokens, 24 heads.
        {"name": "attention_24x4608", "kind": "attention", "batch": 1, "seq_q": 4608, "seq_kv": 4608, "heads": 24,
         "kv_heads": 24, "mask": False},
        # Quantizing one feed-forward weight at load time and decoding it again.
        {"name": "quantize_w4_12288x3072", "kind": "quantize", "n": 12288, "k": 3072, "bits": 4, "dtype": "bf16"},
        # One image at 512x768 on the 8-bit single-stream model: a few hundred short launches.
        {"name": "zimage_w8_1x512x768", "kind": "zimage", "batch": 1, "height": 512, "width": 768, "text": 77,
         "bits": 8, "cfg": False, "graph": False},
        # One image at 1024x1024 on the 4-bit dual / single-stream model: the usual interactive call.
        {"name": "flux_w4_1x1024x1024", "kind": "flux", "batch": 1, "height": 1024, "width": 1024, "text": 512,
         "bits": 4, "guided": True, "graph": False},
        # A guidance pair with prompts of different lengths (so with a key-padding mask) at 1328x1328, replayed from
        # a CUDA graph.
        {"name": "qwen_w4_pair_1328x1328", "kind": "qwen", "height": 1328, "width": 1328, "text": 203,
         "negative_text": 37, "bits": 4, "graph": True},
        # Sixteen images at 1024x1024: the throughput configuration of the benchmark.
        {"name": "flux_w4_16x1024x1024", "kind": "flux", "batch": 16, "height": 1024, "width": 1024, "text": 512,
         "bits": 4, "guided": True, "graph": False},
    ]


def draw(rng) -> dict:
    """Another case of the same ranges: sizes spread over their logarithm, odd row and token counts among them."""
    kind = rng.choice(["linear"] * 5 + ["attention"] * 3 + ["quantize", "flux", "zimage", "qwen"])
    bits = rng.choice([4, 4, 8, 8, 3, 5, 6])
    if kind == "linear":
        k = rng.choice([256, 768, 2560, 3072, 3584, 3840, 4096, 10240, 12288, 15360, 64 * rng.randint(4, 240)])
        n = rng.choice([3072, 3840, 9216, 11520, 12288, 15360, 18432, 20480, 16 * rng.randint(4, 1200)])
        rows, batch = _log_int(rng, 1, 16384), rng.choice([1, 1, 1, 2, 3])
        epilogue = rng.choice(["none", "none", "gelu", "gelu_approx", "silu", "gate_residual", "swiglu"])
        lora = rng.choice([0, 0, 0, 4, 16, 64])
        if bits not in (4, 8):  # adapters come with 4- and 8-bit models
            lora = 0
        if rows <= 16:          # conditioning vectors: [images, K], no gate
            batch, lora, epilogue = 1, 0, rng.choice(["none", "silu"])
        return _linear(None, batch=batch, rows=rows, n=n, k=k, bits=bits, epilogue=epilogue,
                       bias=rng.random() < 0.7, lora=lora)
    if kind == "attention":
        heads = rng.choice([6, 12, 24, 30])
        seq = _log_int(rng, 64, 8192)
        return {"kind": "attention", "batch": rng.choice([1, 1, 2, 4]), "seq_q": seq,
                "seq_kv": seq + rng.choice([0, 0, 0, _log_int(rng, 32, 4096)]), "heads": heads,
                "kv_heads": rng.choice([heads, heads, heads // 3]), "mask": rng.random() < 0.3}
    if kind == "quantize":
        return {"kind": "quantize", "n": _log_int(rng, 256, 20480) // 8 * 8, "k": 64 * _log_int(rng, 4, 240),
                "bits": bits, "dtype": rng.choice(["bf16", "f32"])}
    side = lambda lo, hi: 16 * _log_int(rng, lo // 16, hi // 16)  # noqa: E731
    bits = rng.choice([4, 8])
    if kind == "flux":
        return {"kind": "flux", "batch": rng.choice([1, 1, 2, 4]), "height": side(256, 1536), "width": side(256, 1536),
                "text": rng.choice([256, 512]), "bits": bits, "guided": rng.random() < 0.5, "graph": rng.random() < 0.3}
    if kind == "zimage":
        return {"kind": "zimage", "batch": rng.choice([1, 1, 2, 4]), "height": side(256, 1536),
                "width": side(256, 1536), "text": _log_int(rng, 16, 512), "bits": bits, "cfg": rng.random() < 0.3,
                "graph": rng.random() < 0.3}
    return {"kind": "qwen", "height": side(512, 1328), "width": side(512, 1328), "text": _log_int(rng, 16, 512),
            "negative_text": _log_int(rng, 16, 512), "bits": bits, "graph": rng.random() < 0.5}


def prepare(case: dict, seed: int):
    return _PREPARE[case["kind"]](case, torch.Generator(device=DEVICE).manual_seed(seed), seed)


def run(state):
    return state["run"]()


def work(case: dict) -> dict:
    """Bytes and tensor operations one pass cannot do without: every input (weights packed) read once, every output
    written once; 2 M N K per linear, 4 H Sq Skv 128 per attention."""
    return dict(zip(("bytes", "flops"), _WORK[case["kind"]](case)))


def tolerance(case: dict):
    """Codes, scales and decoded values are exact. The others were measured on a B200 against the same computation
    in float64 on the same packed weights (linear, attention), or between two kernels that order their sums
    differently (model steps, whose bf16 activations carry the roundings of all blocks); about four times that."""
    if case["kind"] == "quantize":
        return "exact"
    return {"rel": _REL[case["kind"]]}


# measured: linear 2.2e-3 to 2.9e-3, attention 2.3e-3, flux 5.5e-3 to 6.6e-3 (the predicted noise), zimage latents
# 1.1e-3 (2.8e-3 with guidance 4, which multiplies the difference of the two branches), qwen latents 8.7e-3 (likewise)
_REL = {"linear": 1e-2, "attention": 1e-2, "flux": 2.5e-2, "zimage": 1e-2, "qwen": 3e-2}


# ---------------------------------------------------------------------------------------------- helpers
def _linear(name, *, rows, n, k, bits, batch=1, epilogue="none", bias=True, lora=0) -> dict:
    case = {"kind": "linear", "batch": batch, "rows": rows, "n": n, "k": k, "bits": bits, "epilogue": epilogue,
            "bias": bias, "lora": lora}
    return {"name": name, **case} if name else case


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _randn(gen, *shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device=DEVICE, generator=gen) * scale).to(dtype)


def _make_linear(gen, n, k, bias, dtype=torch.bfloat16):
    lin = nn.Linear(k, n, bias=bias, device=DEVICE, dtype=dtype)
    lin.weight.data.copy_(_randn(gen, n, k, scale=0.02, dtype=dtype))
    if bias:
        lin.bias.data.copy_(_randn(gen, n, scale=0.02, dtype=dtype))
    return lin


# ---------------------------------------------------------------------------------------------- one linear
def _prepare_linear(case, gen, seed):
    n, k, rows, batch = case["n"], case["k"], case["rows"], case["batch"]
    layer = _make_linear(gen, n, k, case["bias"]).to_quantized(group_size=64, bits=case["bits"])
    layer.prepared()
    if case["lora"]:
        wrapped = LoRALinear.from_linear(layer, r=case["lora"], scale=0.8)
        wrapped.lora_A.data.copy_(_randn(gen, k, case["lora"], scale=k ** -0.5))
        wrapped.lora_B.data.copy_(_randn(gen, case["lora"], n, scale=0.02))
        layer = wrapped
    lead = (rows,) if batch == 1 and rows <= 16 else (batch, rows)
    x = _randn(gen, *lead, k)
    kw = {}
    if case["epilogue"] != "none":
        kw["epilogue"] = case["epilogue"]
    if case["epilogue"] == "gate_residual":
        kw["gate"] = _randn(gen, batch, n)
        kw["residual"] = _randn(gen, batch, rows, n, dtype=torch.float32)
    return {"run": lambda: layer(x, **kw)}


def _work_linear(case):
    n, k, r = case["n"], case["k"], case["lora"]
    m = case["batch"] * case["rows"]
    out = {"swiglu": m * n, "gate_residual": 8 * m * n + 2 * case["batch"] * n}.get(case["epilogue"], 2 * m * n)
    nbytes = n * k * case["bits"] / 8 + 4 * n * k / 64 + 2 * m * k + out + 2 * n * case["bias"] + 2 * r * (n + k)
    return nbytes, 2.0 * m * n * k + 2.0 * m * r * (n + k)


# ---------------------------------------------------------------------------------------------- one attention call
def _prepare_attention(case, gen, seed):
    b, sq, skv, h, hk = (case[f] for f in ("batch", "seq_q", "seq_kv", "heads", "kv_heads"))
    bias = None
    if case["mask"]:    # the last eighth of the keys is padding, one more here and there
        bias = torch.zeros(b, skv, device=DEVICE)
        for i in range(b):
            bias[i, skv - (skv // 4 + i) // 2:] = -1e9
    if sq == skv and hk == h:      # the fused projection buffer of a self-attention block
        qkv = _randn(gen, b, sq, 3 * h * 128)
        return {"run": lambda: ops.fmha(qkv, h, key_bias=bias)}
    q, kv = _randn(gen, b, sq, h * 128), _randn(gen, b, skv, 2 * hk * 128)
    k, v = kv[..., :hk * 128], kv[..., hk * 128:]
    return {"run": lambda: ops.fmha_ex(q, k, v, h, hk, key_bias=bias)}


def _work_attention(case):
    b, sq, skv, h, hk = (case[f] for f in ("batch", "seq_q", "seq_kv", "heads", "kv_heads"))
    nbytes = 2 * 128 * b * (2 * sq * h + 2 * skv * hk) + (4 * b * skv if case["mask"] else 0)
    return nbytes, 4.0 * b * h * sq * skv * 128


# ---------------------------------------------------------------------------------------------- quantize / dequantize
def _prepare_quantize(case, gen, seed):
    dtype = {"bf16": torch.bfloat16, "f32": torch.float32}[case["dtype"]]
    lin = _make_linear(gen, case["n"], case["k"], False, dtype)

    def call():
        q = lin.to_quantized(group_size=64, bits=case["bits"])
        return {"weight": q.weight.data.view(torch.int32), "scales": q.scales.data, "biases": q.biases.data,
                "decoded": q.dequantize()}

    return {"run": call}


def _work_quantize(case):
    es = 4 if case["dtype"] == "f32" else 2
    elems = case["n"] * case["k"]
    packed = elems * case["bits"] / 8 + 2 * es * elems / 64
    return 2 * (es * elems + packed), 0.0


# ---------------------------------------------------------------------------------------------- model steps
STEP, STEPS = 1, 4      # which step of how long a schedule: the second of four


def _prepare_flux(case, gen, seed):
    cfg = FluxConfig(supports_guidance=case["guided"])
    model = Flux1(quantize=case["bits"], model_config=cfg, device=DEVICE, seed=seed, cuda_graph=case["graph"])
    b, h, w = case["batch"], case["height"], case["width"]
    lat = _randn(gen, b, (h // 16) * (w // 16), cfg.in_channels, dtype=torch.float32)
    ctx, pooled = _randn(gen, b, case["text"], cfg.context_dim), _randn(gen, b, cfg.pooled_dim)
    sched = LinearScheduler(STEPS, w, h, cfg.requires_sigma_shift)
    guidance = torch.full((b,), 3.5 * cfg.num_train_steps, device=DEVICE) if case["guided"] else None

    def call():
        ts = torch.full((b,), float(sched.sigmas[STEP]) * cfg.num_train_steps, device=DEVICE)
        noise = model.predict_noise(lat, ctx, pooled, ts, guidance, h, w)
        return {"noise": noise, "latents": ops.euler_step(lat, noise, sched.dt(STEP))}

    return {"run": call}


def _prepare_zimage(case, gen, seed):
    cfg = ZImageConfig(supports_guidance=case["cfg"])
    model = ZImage(quantize=case["bits"], model_config=cfg, device=DEVICE, seed=seed, cuda_graph=case["graph"])
    b, h, w = case["batch"], case["height"], case["width"]
    lat = _randn(gen, b, cfg.in_channels, 1, h // 8, w // 8, dtype=torch.float32)
    cap = _randn(gen, b, case["text"], cfg.cap_feat_dim)
    neg = _randn(gen, b, case["text"], cfg.cap_feat_dim) if case["cfg"] else None
    sched = model.make_scheduler(STEPS, w, h)
    sigma, dt = float(sched.sigmas[STEP]), sched.dt(STEP)
    return {"run": lambda: model.denoise_step(lat, cap, neg, sigma, dt, 4.0 if case["cfg"] else 0.0)}


def _prepare_qwen(case, gen, seed):
    cfg = QwenConfig()
    model = QwenImage(quantize=case["bits"], model_config=cfg, device=DEVICE, seed=seed, cuda_graph=case["graph"])
    h, w = case["height"], case["width"]
    lat = _randn(gen, 1, (h // 16) * (w // 16), cfg.in_channels, dtype=torch.float32)
    pos = _randn(gen, 1, case["text"], cfg.joint_attention_dim)
    neg = _randn(gen, 1, case["negative_text"], cfg.joint_attention_dim)
    sched = cfg.scheduler(STEPS, w, h)
    sigma, dt = float(sched.sigmas[STEP]), sched.dt(STEP)
    return {"run": lambda: model.denoise_step(lat, pos, neg, sigma, dt, 4.0, h, w)}


def _packed(params, bits):
    return params * (bits / 8 + 4 / 64)


def _work_flux(case):
    cfg = FluxConfig(supports_guidance=case["guided"])
    b, d, r, st = case["batch"], cfg.hidden, cfg.mlp_ratio, case["text"]
    si = (case["height"] // 16) * (case["width"] // 16)
    s = si + st
    stream = (4 + 2 * r) * d * d                           # q, k, v, out and the feed-forward pair
    single = (4 + 2 * r) * d * d                           # q, k, v, mlp in and the joint output projection
    embed = (256 + d) * d * (2 if case["guided"] else 1) + (cfg.pooled_dim + d) * d
    rows_si = cfg.num_joint * stream + 2 * cfg.in_channels * d
    rows_st = cfg.num_joint * stream + cfg.context_dim * d
    rows_1 = cfg.num_joint * 12 * d * d + cfg.num_single * 3 * d * d + 2 * d * d + embed
    rows_s = cfg.num_single * single
    flops = 2.0 * b * (si * rows_si + st * rows_st + s * rows_s + rows_1)
    flops += (cfg.num_joint + cfg.num_single) * 4.0 * b * cfg.heads * s * s * 128
    nbytes = _packed(rows_si + rows_st + rows_s + rows_1, case["bits"])
    return nbytes + b * (si * cfg.in_channels * 10 + st * cfg.context_dim * 2), flops


def _work_zimage(case):
    cfg = ZImageConfig()
    d, f = cfg.dim, cfg.ffn_hidden
    b = case["batch"] * (2 if case["cfg"] else 1)
    si = (case["height"] // 16) * (case["width"] // 16)
    sc = case["text"]
    s = si + sc
    block = 4 * d * d + 3 * d * f
    mods = (cfg.n_layers + cfg.n_refiner_layers) * 4 * d * 256 + 256 * d + 256 * 1024 * 2
    flops = 2.0 * b * (cfg.n_layers * s * block + cfg.n_refiner_layers * s * block + mods)
    flops += 2.0 * b * (2 * si * cfg.embed_dim * d + sc * cfg.cap_feat_dim * d)
    flops += 4.0 * b * cfg.n_heads * 128 * (cfg.n_layers * s * s + cfg.n_refiner_layers * (si * si + sc * sc))
    params = (cfg.n_layers + 2 * cfg.n_refiner_layers) * block + mods + (2 * cfg.embed_dim + cfg.cap_feat_dim) * d
    nbytes = _packed(params, case["bits"]) + case["batch"] * si * cfg.embed_dim * 8 + b * sc * cfg.cap_feat_dim * 2
    return nbytes, flops


def _work_qwen(case):
    cfg = QwenConfig()
    d = cfg.hidden
    si = (case["height"] // 16) * (case["width"] // 16)
    texts = (case["text"], case["negative_text"])
    block = (4 + 2 * cfg.mlp_ratio) * d * d
    flops, mods = 0.0, cfg.num_layers * 12 * d * d + 2 * d * d + (256 + d) * d
    for st in texts:
        flops += 2.0 * (cfg.num_layers * (si + st) * block + mods + 2 * si * cfg.in_channels * d
                        + st * cfg.joint_attention_dim * d)
        flops += cfg.num_layers * 4.0 * cfg.heads * (si + st) ** 2 * 128
    params = 2 * cfg.num_layers * block + mods + (2 * cfg.in_channels + cfg.joint_attention_dim) * d
    return _packed(params, case["bits"]) + si * cfg.in_channels * 8 + sum(texts) * cfg.joint_attention_dim * 2, flops


_PREPARE = {"linear": _prepare_linear, "attention": _prepare_attention, "quantize": _prepare_quantize,
            "flux": _prepare_flux, "zimage": _prepare_zimage, "qwen": _prepare_qwen}
_WORK = {"linear": _work_linear, "attention": _work_attention, "quantize": _work_quantize, "flux": _work_flux,
         "zimage": _work_zimage, "qwen": _work_qwen}
