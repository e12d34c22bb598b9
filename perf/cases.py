"""Performance cases of the W8A8 linear route: what a program that serves packed int8 linears has the
library do, through the calls it makes (volvoxai_b200.w8a8), over the range of sizes it makes them at.

``listed()`` names twelve cases, ``draw(rng)`` gives more of the same ranges, ``prepare(case, seed)`` makes
the inputs and the weights a program holds before the call, ``run(state)`` is one pass, ``work(case)`` the
bytes and operations no implementation can do without, ``tolerance(case)`` how far another correct
implementation's outputs may lie and ``exact(case, seed)`` the floating outputs of ``run`` in 64 bits.

Kinds of a case:
  f32      one linear, fp32 in and fp32 out (dynamic per-token quantization, dequantization, bias)
  i8       one linear, fp32 in and requantized int8 out (the next layer is W8A8 too)
  layer    the four linears of one decoder layer with their fused heads and tails: RMSNorm + q/k/v,
           o + residual, RMSNorm + gate/up + SiLU*Mul, down + residual
  island   a static W8A8 island: QuantizeLinear, QLinear, RequantizeLinear, QLinear, DequantizeLinear
  grouped  one linear over PackedLinear storage with a scale per K group (8- or 4-bit words), fp32 out
  host     one linear on pinned host buffers, the whole call (upload, kernels, download, wait)
"""
from __future__ import annotations

import math

import torch

from volvoxai_b200 import w8a8

# Weights are drawn as the codes that per-channel quantization of N(0, 0.02) gives: the channel's largest
# magnitude is about 4.2 sigma.
_SIGMA = 0.02
_PEAK = 4.2
# Activations are N(0, 1) with one channel in a hundred scaled by 20 (outlier channels): mean square 4.99.
_OUTLIER_SHARE, _OUTLIER_GAIN = 0.01, 20.0
_EPS = 1e-6


def listed():
    return [
        # one token through a small model's gate projection: pure launch and call latency
        {"name": "decode_one_token_small", "kind": "f32", "rows": 1, "k": 576, "n": 1536, "bias": True},
        # a decode batch of eight against an 8B-sized projection: the weights are streamed once from HBM
        {"name": "decode_batch8_wide", "kind": "f32", "rows": 8, "k": 4096, "n": 14336, "bias": False},
        # one layer of a 0.6B decoder in a decode step at batch 64: chains of launches of a few microseconds each
        {"name": "decode_layer_batch64", "kind": "layer", "rows": 64, "hidden": 1024, "attn": 2048, "kv": 1024, "inter": 3072},
        # one layer of a 135M decoder in prefill of 8 x 512 tokens: short K, bound by its fp32 outputs
        {"name": "prefill_layer_8x512", "kind": "layer", "rows": 4096, "hidden": 576, "attn": 576, "kv": 192, "inter": 1536},
        # prefill of one prompt of 512 tokens through a square projection: fewer tiles than the chip has SMs
        {"name": "prefill_512_square", "kind": "f32", "rows": 512, "k": 4096, "n": 4096, "bias": True},
        # no size a multiple of anything: odd K, ragged rows and columns, bias and zero point in the requantization
        {"name": "requant_ragged", "kind": "i8", "rows": 777, "k": 1283, "n": 2050, "bias": True, "zero": 3},
        # the benchmark's headline linear: a large prefill batch, requantized for the next layer
        {"name": "requant_8192x4096x14336", "kind": "i8", "rows": 8192, "k": 4096, "n": 14336, "bias": False, "zero": 0},
        # a static package's feed-forward island between float operators, 4096 tokens
        {"name": "static_island_4096", "kind": "island", "rows": 4096, "k": 576, "inter": 1536, "unsigned": True},
        # the exporter's default storage (a scale per 128 weights) in prefill
        {"name": "grouped_w8_prefill", "kind": "grouped", "bits": 8, "group": 128, "rows": 2048, "k": 4096, "n": 4096, "bias": True},
        # the same storage in batched decode
        {"name": "grouped_w8_batch8", "kind": "grouped", "bits": 8, "group": 128, "rows": 8, "k": 4096, "n": 14336, "bias": False},
        # 4-bit storage, one token: half the weight bytes
        {"name": "grouped_w4_one_token", "kind": "grouped", "bits": 4, "group": 128, "rows": 1, "k": 4096, "n": 14336, "bias": False},
        # an application that holds host tensors: 2048 rows up, computed, and down
        {"name": "host_2048x4096x14336", "kind": "host", "rows": 2048, "k": 4096, "n": 14336, "bias": False, "zero": 0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng, lo, hi):
    """A layer width: most are multiples of 64, some of 8, some of nothing."""
    v = _log_int(rng, lo, hi)
    p = rng.random()
    if p < 0.5:
        v = max(64, v // 64 * 64)
    elif p < 0.75:
        v = max(8, v // 8 * 8)
    return v


def draw(rng):
    kind = rng.choice(["f32", "f32", "f32", "i8", "i8", "layer", "layer", "island", "grouped", "grouped", "grouped", "host"])
    most = 2.0 * 8192 * 4096 * 14336            # operations of the largest listed case
    while True:
        if kind == "layer":
            heads = rng.randint(4, 24)
            head = rng.choice([64, 128])
            kv = max(1, heads // rng.choice([1, 2, 3, 4]))
            case = {"kind": kind, "rows": _log_int(rng, 1, 4096), "hidden": 64 * rng.randint(6, 32), "attn": heads * head,
                    "kv": kv * head, "inter": 64 * rng.randint(12, 88)}
        elif kind == "island":
            case = {"kind": kind, "rows": _log_int(rng, 1, 8192), "k": _width(rng, 128, 4096), "inter": _width(rng, 256, 8192),
                    "unsigned": rng.random() < 0.5}
        elif kind == "grouped":
            case = {"kind": kind, "bits": rng.choice([8, 4]), "group": rng.choice([32, 64, 128, 128, 256]),
                    "rows": rng.choice([1, 1, _log_int(rng, 2, 64), _log_int(rng, 64, 2048)]), "k": _width(rng, 256, 14336),
                    "n": _width(rng, 256, 14336), "bias": rng.random() < 0.5}
        elif kind == "host":
            case = {"kind": kind, "rows": _log_int(rng, 1, 4096), "k": _width(rng, 256, 8192), "n": _width(rng, 256, 14336),
                    "bias": rng.random() < 0.5, "zero": rng.choice([0, 0, -7])}
        else:
            case = {"kind": kind, "rows": _log_int(rng, 1, 8192), "k": _width(rng, 256, 14336), "n": _width(rng, 192, 16384),
                    "bias": rng.random() < 0.5}
            if kind == "i8":
                case["zero"] = rng.choice([0, 0, 5])
        w = work(case)
        if w["flops"] <= most and w["bytes"] <= 4e8:
            return case


# ---- inputs and weights -----------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(g, rows, k):
    x = torch.randn((rows, k), generator=g, device="cuda")
    loud = torch.randperm(k, generator=g, device="cuda")[:max(1, int(k * _OUTLIER_SHARE))]
    x[:, loud] *= _OUTLIER_GAIN
    return x


def _codes(g, n, k, top=127):
    w = torch.randn((n, k), generator=g, device="cuda").mul_(top / _PEAK).round_().clamp_(-top, top)
    return w.to(torch.int8)


def _scales(g, n, top=127):
    return (_SIGMA * _PEAK / top) * (0.9 + 0.2 * torch.rand(n, generator=g, device="cuda"))


def _drawn(g, n, k, bias=False, bias_i32=False):
    w, ws = _codes(g, n, k), _scales(g, n)
    bf = torch.randn(n, generator=g, device="cuda") * 0.01 if bias else None
    bi = torch.randint(-2000, 2001, (n,), generator=g, device="cuda", dtype=torch.int32) if bias_i32 else None
    return w, ws, bf, bi


def _weight(ctx, g, n, k, bias=False, bias_i32=False):
    host = [None if t is None else t.cpu().numpy() for t in _drawn(g, n, k, bias, bias_i32)]
    return w8a8.Weight.from_i8(ctx, *host)


def _pack_words(codes, bits):
    """Offset-binary storage words, earlier K in lower bits; the last word is padded with the encoded zero."""
    n, k = codes.shape
    per, zero = 32 // bits, 1 << (bits - 1)
    padded = torch.full((n, (k + per - 1) // per * per), zero, dtype=torch.int64, device=codes.device)
    padded[:, :k] = codes.to(torch.int64) + zero
    shifts = torch.arange(per, device=codes.device, dtype=torch.int64) * bits
    words = (padded.view(n, -1, per) << shifts).sum(dim=2)
    return torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32)


def _grouped_drawn(g, case):
    n, k, bits, group = case["n"], case["k"], case["bits"], case["group"]
    top = 127 if bits == 8 else 7
    codes = torch.cat([_codes(g, min(2048, n - lo), k, top) for lo in range(0, n, 2048)])
    scales = _scales(g, n * ((k + group - 1) // group), top).view(n, -1)
    return codes, scales, torch.randn(n, generator=g, device="cuda") * 0.01 if case["bias"] else None


def _grouped_weight(ctx, g, case):
    n, bits = case["n"], case["bits"]
    codes, scales, bias = _grouped_drawn(g, case)
    words = torch.cat([_pack_words(codes[lo:lo + 2048], bits) for lo in range(0, n, 2048)])
    make = w8a8.Weight.from_w8_words if bits == 8 else w8a8.Weight.from_w4_words
    return make(ctx, words.cpu().numpy(), scales.cpu().numpy(), case["k"], case["group"],
                None if bias is None else bias.cpu().numpy())


def _layer_inputs(g, case):
    rows, hidden = case["rows"], case["hidden"]
    x = torch.randn((rows, hidden), generator=g, device="cuda")
    attn = torch.randn((rows, case["attn"]), generator=g, device="cuda") * 0.5
    norms = [1.0 + 0.1 * torch.randn(hidden, generator=g, device="cuda") for _ in range(2)]
    return x, attn, *norms


def _out_scale(k):
    """The 99.9th percentile of |y| over 127, for activations and weights drawn as above."""
    mean_square = 1.0 + _OUTLIER_SHARE * (_OUTLIER_GAIN ** 2 - 1.0)
    return 3.29 * _SIGMA * math.sqrt(k * mean_square) / 127.0


def prepare(case, seed):
    g = _gen(seed)
    ctx = w8a8.Context(0)
    ctx.use_torch_stream()
    kind, rows = case["kind"], case["rows"]
    s = {"kind": kind, "ctx": ctx}
    if kind == "layer":
        hidden, attn, kv, inter = case["hidden"], case["attn"], case["kv"], case["inter"]
        s["x"], s["attn"], s["norm1"], s["norm2"] = _layer_inputs(g, case)
        s["qkv"] = _weight(ctx, g, attn + 2 * kv, hidden)
        s["o"] = _weight(ctx, g, hidden, attn)
        s["gate_up"] = _weight(ctx, g, 2 * inter, hidden)       # channels interleaved (gate_0, up_0, gate_1, ...)
        s["down"] = _weight(ctx, g, hidden, inter)
    elif kind == "island":
        k, inter = case["k"], case["inter"]
        s["x"] = torch.randn((rows, k), generator=g, device="cuda")
        s["up"] = _weight(ctx, g, inter, k, bias_i32=True)
        s["down"] = _weight(ctx, g, k, inter, bias_i32=True)
        s["unsigned"] = bool(case["unsigned"])
        zero = 128 if case["unsigned"] else 0
        s["in"] = (4.0 / 127.0, zero)                           # activation domains: (scale, zero point)
        hidden_scale = 3.29 * _SIGMA * math.sqrt(k) / 127.0
        s["mid"] = (hidden_scale, zero)
        s["mid2"] = (hidden_scale * 1.25, 0)
        s["out"] = (3.29 * _SIGMA * math.sqrt(inter) * hidden_scale * 127.0 / 3.29 / 127.0, 0)
    elif kind == "grouped":
        s["w"] = _grouped_weight(ctx, g, case)
        s["x"] = _activations(g, rows, case["k"])
    else:
        s["w"] = _weight(ctx, g, case["n"], case["k"], bias=case["bias"] and kind == "f32", bias_i32=case["bias"] and kind != "f32")
        x = _activations(g, rows, case["k"])
        if kind != "f32":
            s["out_scale"], s["zero"] = _out_scale(case["k"]), case["zero"]
        if kind == "host":
            s["x"] = torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(x)
            s["y"] = torch.empty((rows, case["n"]), dtype=torch.int8, pin_memory=True)
        else:
            s["x"] = x
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind in ("f32", "grouped"):
        return ctx.linear_f32(s["w"], s["x"])
    if kind == "i8":
        return ctx.linear_i8(s["w"], s["x"], s["out_scale"], s["zero"])
    if kind == "host":
        ctx.linear_host(s["w"], s["x"], s["y"], requant=True, out_scale=s["out_scale"], out_zero=s["zero"])
        return s["y"]
    if kind == "layer":
        x = s["x"]
        qkv = ctx.rmsnorm_linear_f32_fused(s["qkv"], x, s["norm1"], _EPS)
        h = ctx.linear_f32_fused(s["o"], s["attn"], residual=x)
        act = ctx.rmsnorm_linear_f32_fused(s["gate_up"], h, s["norm2"], _EPS, silu_mul=True)
        y = ctx.linear_f32_fused(s["down"], act, residual=h)
        return {"qkv": qkv, "h": h, "act": act, "y": y}
    # island
    q = ctx.quantize_linear(s["x"], *s["in"], unsigned=s["unsigned"])
    mid = ctx.qlinear_device(s["up"], q, *s["in"], *s["mid"], out_unsigned=s["unsigned"])
    mid2 = ctx.requantize_linear(mid, *s["mid"], *s["mid2"])
    out = ctx.qlinear_device(s["down"], mid2, *s["mid2"], *s["out"])
    return {"mid": mid, "q": out, "y": ctx.dequantize_linear(out, *s["out"])}


# ---- the floating outputs in 64 bits --------------------------------------------------------------

def _quantized(x):
    """The row's code and scale are defined in 32 bits (x and scale are fp32, the quotient is rounded to fp32, then
    to the nearest even whole number); a quotient taken in 64 bits and rounded to 32 is that fp32 quotient."""
    scale = (x.abs().amax(dim=1, keepdim=True).double() / 127.0).float()
    scale = torch.where(scale == 0, torch.ones_like(scale), scale)
    return (x.double() / scale.double()).float().round().clamp(-127, 127).double(), scale.double()


def _linear64(x, w, ws, bias=None):
    q, scale = _quantized(x)
    y = (q @ w.double().T) * scale * ws.double()
    return y if bias is None else y + bias.double()


def _norm64(x, weight):
    x = x.double()
    return (x / (x.square().mean(dim=1, keepdim=True) + _EPS).sqrt() * weight.double()).float()


def exact(case, seed):
    """What ``run`` returns in 64 bits, from the codes that the storage holds.  A linear's input is fp32, so a layer's
    outputs are rounded where the next linear takes them up.  None where outputs are codes: those are exact."""
    g, kind, rows = _gen(seed), case["kind"], case["rows"]
    if kind == "f32":
        w, ws, bias, _ = _drawn(g, case["n"], case["k"], bias=case["bias"])
        return _linear64(_activations(g, rows, case["k"]), w, ws, bias)
    if kind == "grouped":
        codes, scales, bias = _grouped_drawn(g, case)
        q, scale = _quantized(_activations(g, rows, case["k"]))
        k, group = case["k"], case["group"]
        y = torch.zeros((rows, case["n"]), dtype=torch.float64, device="cuda")
        for i, lo in enumerate(range(0, k, group)):
            hi = min(k, lo + group)
            y += (q[:, lo:hi] @ codes[:, lo:hi].double().T) * scales[:, i].double()
        y *= scale
        return y if bias is None else y + bias.double()
    if kind == "layer":
        hidden, attn, kv, inter = case["hidden"], case["attn"], case["kv"], case["inter"]
        x, a, norm1, norm2 = _layer_inputs(g, case)
        weights = [_drawn(g, n, k)[:2] for n, k in ((attn + 2 * kv, hidden), (hidden, attn), (2 * inter, hidden), (hidden, inter))]
        qkv = _linear64(_norm64(x, norm1), *weights[0])
        h = _linear64(a, *weights[1]) + x.double()
        gate_up = _linear64(_norm64(h.float(), norm2), *weights[2])
        act = torch.nn.functional.silu(gate_up[:, 0::2]) * gate_up[:, 1::2]
        y = _linear64(act.float(), *weights[3]) + h
        return {"qkv": qkv, "h": h, "act": act, "y": y}
    return None


# ---- what one pass cannot do without ------------------------------------------------------------

def _linear(rows, k, n, in_bytes, out_bytes, weight_bytes=None):
    return (rows * k * in_bytes + (n * k if weight_bytes is None else weight_bytes) + 4 * n + rows * n * out_bytes, 2.0 * rows * k * n)


def work(case):
    kind, rows = case["kind"], case["rows"]
    if kind == "layer":
        hidden, attn, kv, inter = case["hidden"], case["attn"], case["kv"], case["inter"]
        parts = [_linear(rows, hidden, attn + 2 * kv, 4, 4), _linear(rows, attn, hidden, 4, 4),
                 _linear(rows, hidden, 2 * inter, 4, 2), _linear(rows, inter, hidden, 4, 4)]
        extra = 2 * 4 * rows * hidden + 2 * 4 * hidden          # the two residuals and the norm weights
        return {"bytes": sum(p[0] for p in parts) + extra, "flops": sum(p[1] for p in parts)}
    if kind == "island":
        k, inter = case["k"], case["inter"]
        up, down = _linear(rows, k, inter, 4, 1), _linear(rows, inter, k, 0, 1)
        # fp32 in, the requantized hidden bytes out, the int8 result and its fp32 form out
        return {"bytes": up[0] + down[0] + 4 * (k + inter) + 4 * rows * k, "flops": up[1] + down[1]}
    k, n = case["k"], case["n"]
    if kind == "grouped":
        groups = (k + case["group"] - 1) // case["group"]
        b, f = _linear(rows, k, n, 4, 4, weight_bytes=n * ((k * case["bits"] + 31) // 32) * 4 + 4 * n * (groups - 1))
    else:
        b, f = _linear(rows, k, n, 4, 4 if kind == "f32" else 1)
    return {"bytes": b + (4 * n if case["bias"] else 0), "flops": f}


def tolerance(case):
    return _TOLERANCE[case["kind"]]


# Integer results are exact by contract.  The others are four times what the path showed against the same
# arithmetic in 64 bits over the listed and some drawn cases: rel 5e-8 / max 2.5e-7 for one linear (the roundings of
# its epilogue), 1.2e-7 / 9.4e-7 with group scales (the running sum over the groups), 4.6e-5 / 7.7e-3 for a layer,
# where an ulp of a normalized row or of the SiLU moves a code by one on a tie in about one element of two million.
_TOLERANCE = {
    "f32": {"rel": 2e-7, "max": 1e-6},
    "grouped": {"rel": 5e-7, "max": 4e-6},
    "i8": "exact",
    "host": "exact",
    "island": "exact",
    "layer": {"rel": 2e-4, "max": 3e-2},
}
