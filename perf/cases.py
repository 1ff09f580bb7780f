"""The calls a user of this package makes, as cases to measure: the quantized linear layer on device and on host buffers,
the weight-only layer, the fp16 output head, a whole prompt and a decode step of the synthetic Qwen3 model, and the
offline weight quantizer.

A case names a `kind` and its sizes; inputs are drawn on the GPU from the seed with the value distributions of the
benchmark configurations (activations ~ N(0, 1), nibbles uniform, block scales ~ U(0.002, 0.02), block minima
~ U(-0.1, 0), both rounded to fp16, head weights ~ N(0, 0.02)).  Layer shapes are Qwen3-8B's in the listed cases and
anything the layers accept (rows a multiple of 8, K a multiple of 64) in the drawn ones.
"""
import math

import torch

from __graft_entry__ import load_package

pkg = load_package()

SCHEMES = {"A81W41": pkg.A81W41, "A80W40": pkg.A80W40, "A80W4Z": pkg.A80W4Z}
VOCAB, HIDDEN = 151936, 4096     # Qwen3-8B's output head
LAYERS = 36                      # ... and decoder depth
MAX_POS = 512

_context = None


def context():
    """One context for the process, as a serving program keeps it."""
    global _context
    if _context is None:
        _context = pkg.Context(0, torch.cuda.current_stream().cuda_stream)
    return _context


def listed():
    return [
        # one token through an attention block's q, k, v and o projections: the smallest calls, all latency
        {"name": "attention linears m1", "kind": "attention", "scheme": "A81W41", "scales": "f16", "m": 1, "hidden": 4096, "heads": 32,
         "kv_heads": 8},
        # one token through the down projection, symmetric weights: the long-row decode call
        {"name": "linear m1 4096x12288", "kind": "linear", "scheme": "A80W40", "scales": "f16", "m": 1, "n": 4096, "k": 12288},
        # five sequences decoded together through the fused gate_up projection
        {"name": "linear m5 24576x4096", "kind": "linear", "scheme": "A81W41", "scales": "f16", "m": 5, "n": 24576, "k": 4096},
        # a short chat turn through the down projection, zero-point weights
        {"name": "linear m77 4096x12288", "kind": "linear", "scheme": "A80W4Z", "scales": "f16", "m": 77, "n": 4096, "k": 12288},
        # the reference's benchmark prompt (322 tokens) through gate_proj, fp32 scales: the headline shape
        {"name": "linear m322 12288x4096", "kind": "linear", "scheme": "A81W41", "scales": "f32", "m": 322, "n": 12288, "k": 4096},
        # a long prompt through the same layer, symmetric weights
        {"name": "linear m2048 12288x4096", "kind": "linear", "scheme": "A80W40", "scales": "f16", "m": 2048, "n": 12288, "k": 4096},
        # the drop-in use from the reference's C++ class: activations and result in (page-locked) host memory
        {"name": "host m322 12288x4096", "kind": "host", "scheme": "A81W41", "scales": "f32", "m": 322, "n": 12288, "k": 4096},
        # the weight-only layer on the same prompt
        {"name": "w41 m322 12288x4096", "kind": "w41", "m": 322, "n": 12288, "k": 4096},
        # the output head for eight sequences decoded together
        {"name": "head m8 151936x4096", "kind": "head", "m": 8, "n": VOCAB, "k": HIDDEN, "fp16_act": False},
        # the whole model on the benchmark prompt: pp322
        {"name": "model prompt 322", "kind": "prompt", "tokens": 322, "layers": LAYERS},
        # one decode step after that prompt, as a captured graph: tg
        {"name": "model decode at 322", "kind": "decode", "context": 322, "layers": LAYERS},
        # converting one layer's fp32 weights to the 4-bit format
        {"name": "convert 12288x4096", "kind": "convert", "format": 1, "n": 12288, "k": 4096},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _layer(rng, n_max=24576):
    """A layer's (n, k): any multiples of 8 and 64 of the range, no larger than the listed layers."""
    k = 64 * _log_int(rng, 1024 // 64, 12288 // 64)
    n = 8 * _log_int(rng, 512 // 8, min(n_max, 12288 * 4096 * 2 // k) // 8)
    return n, k


def draw(rng):
    kind = rng.choices(["attention", "linear1", "linear", "host", "w41", "head", "prompt", "decode", "convert"], [1, 1, 7, 2, 3, 2, 1, 1, 1])[0]
    if kind == "attention":
        kv = rng.choice([2, 4, 8])
        return {"kind": "attention", "scheme": rng.choice(list(SCHEMES)), "scales": rng.choice(["f16", "f32"]), "m": _log_int(rng, 1, 16),
                "hidden": 64 * _log_int(rng, 1024 // 64, 5120 // 64), "heads": kv * rng.choice([2, 4]), "kv_heads": kv}
    if kind == "linear1":     # one token through a feed-forward layer
        f, h = 64 * _log_int(rng, 9216 // 64, 24576 // 64), 4096
        n, k = (f, h) if rng.random() < 0.6 else (h, min(f, 12288))
        return {"kind": "linear", "scheme": rng.choice(list(SCHEMES)), "scales": rng.choice(["f16", "f32"]), "m": 1, "n": n, "k": k}
    if kind in ("linear", "host"):
        m = _log_int(rng, 2, 2048) if kind == "linear" else _log_int(rng, 1, 512)
        n, k = _layer(rng, 12288 if m > 64 else 24576)
        return {"kind": "host" if kind == "host" else "linear", "scheme": rng.choice(list(SCHEMES)), "scales": rng.choice(["f16", "f32"]),
                "m": m, "n": n, "k": k}
    if kind == "w41":
        m = _log_int(rng, 1, 2048)
        n, k = _layer(rng, 12288)
        return {"kind": "w41", "m": m, "n": n, "k": k}
    if kind == "head":
        n = 8 * _log_int(rng, 16384 // 8, VOCAB // 8)
        return {"kind": "head", "m": _log_int(rng, 1, 64), "n": n, "k": rng.choice([2048, 2560, HIDDEN]), "fp16_act": rng.random() < 0.3}
    if kind == "prompt":
        return {"kind": "prompt", "tokens": _log_int(rng, 8, 322), "layers": LAYERS}
    if kind == "decode":
        return {"kind": "decode", "context": _log_int(rng, 8, MAX_POS - 16), "layers": LAYERS}
    n, k = _layer(rng, 12288)
    return {"kind": "convert", "format": rng.choice([0, 1]), "n": n, "k": k}


def _logical_weights(g, n, k):
    """A layer in the on-disk format, on the GPU: nibbles, scales, minima, zero points."""
    nib = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    d = (torch.rand((n, k // 32), device="cuda", generator=g) * 0.018 + 0.002).half().float()
    m = (torch.rand((n, k // 32), device="cuda", generator=g) * -0.1).half().float()
    zp = torch.randint(0, 16, (n, k // 32), dtype=torch.uint8, device="cuda", generator=g)
    return nib, d, m, zp


def _weight(g, scheme, scale_mode, n, k):
    nib, d, m, zp = _logical_weights(g, n, k)
    w = context().weight_dev(scheme, scale_mode, n, k, nib, d, m if scheme in (pkg.A81W41, pkg.W41) else None,
                             zp if scheme == pkg.A80W4Z else None)
    context().synchronize()      # the logical arrays are read by the re-tiling kernel
    return w


def _model(seed, layers):
    return pkg.qwen3_forward.Qwen3Synthetic(pkg, context(), pkg.qwen3_forward.Qwen3Config(layers=layers, max_pos=MAX_POS), seed=seed)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    kind = case["kind"]
    s = dict(case)
    if kind == "attention":
        m, h = case["m"], case["hidden"]
        for name, n, k in _projections(case):
            w = _weight(g, SCHEMES[case["scheme"]], pkg.SCALES_F16 if case["scales"] == "f16" else pkg.SCALES_F32, n, k)
            s[name] = (w, n, torch.zeros((m, n), device="cuda"))
        s["x"] = torch.randn((m, h), device="cuda", generator=g)
        s["attn"] = torch.randn((m, case["heads"] * 128), device="cuda", generator=g)
    elif kind in ("linear", "host"):
        m, n, k = case["m"], case["n"], case["k"]
        s["w"] = _weight(g, SCHEMES[case["scheme"]], pkg.SCALES_F16 if case["scales"] == "f16" else pkg.SCALES_F32, n, k)
        s["x"] = torch.randn((m, k), device="cuda", generator=g)
        if kind == "host":
            s["x"] = s["x"].cpu().pin_memory()
            s["c"] = torch.zeros((m, n), pin_memory=True)
        else:
            s["c"] = torch.zeros((m, n), device="cuda")
    elif kind == "w41":
        m, n, k = case["m"], case["n"], case["k"]
        s["w"] = _weight(g, pkg.W41, pkg.SCALES_F16, n, k)
        s["x"] = torch.randn((m, k), device="cuda", generator=g).half()
        s["c"] = torch.zeros((m, n), device="cuda")
    elif kind == "head":
        m, n, k = case["m"], case["n"], case["k"]
        w16 = (torch.randn((n, k), device="cuda", generator=g) * 0.02).half()
        s["w"] = context().f16w_dev(w16, n, k)
        context().synchronize()
        s["x"] = torch.randn((m, k), device="cuda", generator=g)
        s["c"] = torch.zeros((m, n), device="cuda")
    elif kind == "prompt":
        s["model"] = _model(seed, case["layers"])
        s["prompt"] = torch.randint(0, VOCAB, (case["tokens"],), dtype=torch.int32, device="cuda", generator=g)
    elif kind == "decode":
        # a program that generates: prompt, one eager step (every scratch buffer exists), one step captured as a graph
        model = _model(seed, case["layers"])
        model.prefill(torch.randint(0, VOCAB, (case["context"],), dtype=torch.int32, device="cuda", generator=g))
        model.decode_step()
        model.capture_decode()
        s["model"] = model
        s["token"] = torch.randint(0, VOCAB, (1,), dtype=torch.int32, device="cuda", generator=g)
    elif kind == "convert":
        s["x"] = torch.randn((case["n"], case["k"]), device="cuda", generator=g) * 0.02
    else:
        raise ValueError(kind)
    return s


def run(s):
    ctx, kind = context(), s["kind"]
    if kind == "attention":
        for name in ("q", "k", "v", "o"):
            w, n, c = s[name]
            ctx.linear(w, s["attn" if name == "o" else "x"], s["m"], c, n)
        return [s[name][2] for name in ("q", "k", "v", "o")]
    if kind == "linear":
        ctx.linear(s["w"], s["x"], s["m"], s["c"], s["n"])
        return s["c"]
    if kind == "host":
        ctx.linear_host(s["w"], s["x"], s["m"], s["c"], s["n"])
        return s["c"]
    if kind == "w41":
        ctx.gemm_w41_f16act(s["x"], s["m"], s["w"], s["c"], s["n"])
        return s["c"]
    if kind == "head":
        ctx.f16w_matmul_prec(s["w"], s["x"], s["m"], s["c"], s["n"], 1 if s["fp16_act"] else 0)
        return s["c"]
    if kind == "prompt":
        model = s["model"]
        model.reset()
        logits = model.prefill(s["prompt"])
        last = model.layers[-1]
        return {"logits": logits, "k": last["k_cache"], "v": last["v_cache"]}
    if kind == "decode":
        model = s["model"]
        model.pos.fill_(s["context"])
        model.token.copy_(s["token"])
        model.graph.replay()
        last = model.layers[-1]
        return {"logits": model.bufs[1]["logits"], "k": last["k_cache"], "v": last["v_cache"]}
    nib, d, m, zp = ctx.quantize_weights(s["format"], s["x"])
    return {"nib": nib, "d": d, "m": m, "zp": zp}


def _block_bytes(scheme, scales):
    """Bytes of scales (minima, zero points) of one 32-element weight block."""
    if scheme == "A81W41":
        return 8 if scales == "f32" else 4
    return (4 if scales == "f32" else 2) + (0.5 if scheme == "A80W4Z" else 0)


def _projections(case):
    """(name, n, k) of an attention block's linears, heads of 128."""
    h, q, kv = case["hidden"], case["heads"] * 128, case["kv_heads"] * 128
    return [("q", q, h), ("k", kv, h), ("v", kv, h), ("o", h, q)]


def _model_linears(layers):
    """Quantized weights of the model's linears."""
    return layers * (6144 * 4096 + 4096 * 4096 + 24576 * 4096 + 4096 * 12288)


def work(case):
    kind = case["kind"]
    if kind == "attention":
        m, nk = case["m"], _projections(case)
        weights = sum(n * k for _, n, k in nk)
        values = case["hidden"] + case["heads"] * 128 + sum(n for _, n, _ in nk)
        return {"bytes": weights / 2 + weights / 32 * _block_bytes(case["scheme"], case["scales"]) + m * values * 4, "flops": 2.0 * m * weights}
    if kind in ("linear", "host", "w41"):
        m, n, k = case["m"], case["n"], case["k"]
        per_block = 4 if kind == "w41" else _block_bytes(case["scheme"], case["scales"])
        act = 2 if kind == "w41" else 4
        return {"bytes": n * k / 2 + n * (k // 32) * per_block + m * k * act + m * n * 4, "flops": 2.0 * m * n * k}
    if kind == "head":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": n * k * 2 + m * k * 4 + m * n * 4, "flops": 2.0 * m * n * k}
    if kind == "convert":
        n, k = case["n"], case["k"]
        return {"bytes": n * k * 4 + n * k / 2 + n * (k // 32) * 9, "flops": 4.0 * n * k}
    t = case["tokens"] if kind == "prompt" else 1
    past = 0 if kind == "prompt" else case["context"]
    params = _model_linears(case["layers"])
    scores = t * past + t * (t + 1) / 2                       # query x key pairs of one head
    cache = case["layers"] * 2 * 8 * 128 * 2 * (past + t)     # keys and values of the context, fp16
    return {"bytes": params * 0.625 + VOCAB * HIDDEN * 2 + cache + VOCAB * 4,
            "flops": 2.0 * t * params + 2.0 * VOCAB * HIDDEN + case["layers"] * 32 * 4.0 * 128 * scores}


def tolerance(case):
    kind = case["kind"]
    if kind in ("attention", "linear", "host"):
        return {"rel": 1e-5, "max": 4e-4}                     # exact block dots, fp32 sums of K / 32 scaled terms
    if kind == "w41":
        return {"rel": 1e-5, "max": 4e-4}                     # fp16 products, fp32 sums
    if kind == "head":
        # fp32-grade activations; as fp16 values each activation is rounded to 11 bits
        return {"rel": 1e-3, "max": 1e-2} if case["fp16_act"] else {"rel": 5e-5, "max": 4e-4}
    if kind == "convert":
        return "exact"
    # Every layer rounds its activations to int8: another summation order in front of a rounding moves single codes by
    # one, and 36 layers carry that on.
    return {"rel": 2e-2, "max": 0.3}
