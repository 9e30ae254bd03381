"""Performance cases of cachalot_b200: the calls a decode or prefill loop makes, over the sizes it makes them at.

A case names one family of calls and its sizes.  `listed()` is the fixed set, `draw()` gives more of the same families
and ranges.  The two bank shapes that appear by themselves, 4096 x 2880 and 5120 x 2304, are the ones this
repository's configurations and defaults use; drawn cases take other multiples of 128 and 64.

    layer    one decode token through stacked MoE layers: routing tail + routed experts (moe_layer_decode)
    block    the whole MoE block of one token: gate, routing, routed experts, shared FP8 expert (moe_layer_forward)
    batch    routed experts of a few concurrent tokens with their slots already known (moe_forward)
    prefill  routed experts of a prompt chunk, expert by expert (moe_prefill_grouped)
    trunk    the FP8 projections around attention for a few tokens: act_quant + GEMV (fp8_linear)
    shared   the shared FP8 expert over a prompt chunk (shared_expert_forward_batched)
    head     the bf16 output head (bf16_gemv_f32)
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cachalot_b200 as cb
from cachalot_b200 import ops

DEV = "cuda"
FULL_SIZE = 4096 * 2880  # weights of one projection of the largest experts (5120 x 2304 is the same)


def _case(name, kind, **sizes):
    return {"name": name, "kind": kind, **sizes}


def listed():
    return [
        # the steady state of a single-user session: one token, the bank that fits one GPU, one launch per layer
        _case("layer-2bit-1", "layer", bank="2bit", hidden=4096, inter=2880, experts=384, topk=6, layers=4, router="sigmoid"),
        # the same token through the reference's keyword-for-keyword layer entry: router GEMV, experts, shared expert
        _case("block-fp4-1", "block", bank="fp4", hidden=5120, inter=2304, experts=384, topk=6, rule="e8m0"),
        # a handful of concurrent sessions, or the drafted tokens of speculative decoding
        _case("batch-2bit-8", "batch", bank="2bit", hidden=4096, inter=2880, experts=384, topk=6, tokens=8),
        _case("batch-fp4-8", "batch", bank="fp4", hidden=4096, inter=2880, experts=384, topk=6, tokens=8),
        # a serving batch
        _case("batch-fp4-64", "batch", bank="fp4", hidden=4096, inter=2880, experts=384, topk=6, tokens=64),
        # a full prompt chunk with MXFP4 activations
        _case("prefill-fp4-4096", "prefill", bank="fp4", hidden=4096, inter=2880, experts=384, topk=6, tokens=4096, act="mxfp4", skew=1.1),
        # the ragged last chunk of a prompt, bf16 activations (the entry's default)
        _case("prefill-fp4-bf16-777", "prefill", bank="fp4", hidden=5120, inter=2304, experts=384, topk=6, tokens=777, act="bf16", skew=1.1),
        # a prompt chunk on the machine that holds the 2-bit bank
        _case("prefill-2bit-2048", "prefill", bank="2bit", hidden=4096, inter=2880, experts=384, topk=6, tokens=2048, act="bf16", skew=1.1),
        # the trunk's projections of one token, and of a batch of them
        _case("trunk-fp8-1", "trunk", n1=12288, k1=4096, n2=4096, k2=8192, rows=1, rule="f32"),
        _case("trunk-fp8-32", "trunk", n1=12288, k1=4096, n2=4096, k2=8192, rows=32, rule="f32"),
        # the shared expert of a ragged prompt chunk
        _case("shared-fp8-1000", "shared", hidden=5120, inter=2304, rows=1000, rule="e8m0"),
        # logits of one token
        _case("head-bf16-1", "head", vocab=129280, hidden=5120, rows=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer", "block", "batch", "batch", "prefill", "prefill", "trunk", "shared", "head"])
    c = {"kind": kind}
    if kind in ("layer", "block", "batch", "prefill"):
        c["bank"] = rng.choice(["fp4", "2bit"])
        hidden = 128 * rng.randint(16, 40)
        other = (hidden, 64 * rng.randint(12, min(44, FULL_SIZE // hidden // 64)))
        c["hidden"], c["inter"] = rng.choice([(4096, 2880), (5120, 2304), other, other])
        c["experts"] = rng.choice([64, 128, 160, 256, 384])
        c["topk"] = rng.choice([4, 6, 6, 8])
    if kind == "layer":
        c["layers"] = rng.randint(2, 4)
        c["router"] = rng.choice(["sigmoid", "sqrt_softplus"])
    if kind == "batch":
        c["tokens"] = _log_int(rng, 2, 64)
    if kind == "prefill":
        c["act"] = rng.choice(["mxfp4", "bf16"]) if c["bank"] == "fp4" else "bf16"
        most = (4096 if c["bank"] == "fp4" else 2048) * 6 // c["topk"]
        c["tokens"] = _log_int(rng, 65, min(most, 4096))
        c["skew"] = rng.choice([0.0, 1.1])
    if kind == "trunk":
        c["n1"], c["k1"] = 128 * rng.randint(8, 96), 128 * rng.randint(12, 64)
        c["n2"], c["k2"] = 128 * rng.randint(8, 40), 128 * rng.randint(12, 64)
        c["rows"] = _log_int(rng, 1, 64)
    if kind == "shared":
        c["hidden"], c["inter"] = 128 * rng.randint(16, 40), 128 * rng.randint(8, 24)
        c["rows"] = _log_int(rng, 65, 1000)
    if kind == "head":
        c["vocab"], c["hidden"] = rng.randint(32000, 129280), 64 * rng.randint(32, 80)
        c["rows"] = rng.randint(1, 4)
    if kind in ("block", "trunk", "shared"):
        c["rule"] = rng.choice(["e8m0", "f32"]) if c.get("inter", 0) % 128 == 0 else "e8m0"  # f32 scales: blocks of 128
    return c


# ---- inputs ---------------------------------------------------------------------------------------

def _bank(c, gen, layers=1):
    fmt = cb.FP4_FORMAT if c["bank"] == "fp4" else cb.affine_format(c["hidden"], c["inter"])
    bank = cb.SlabBank(fmt, c["hidden"], c["inter"], layers * c["experts"], layers=layers, n_experts=c["experts"])
    bank.fill_random(gen)
    return bank


def _x(gen, *shape):
    return torch.randn(shape, device=DEV, generator=gen).to(torch.bfloat16)


def _fp8_matrix(gen, n, k, rule):
    """E4M3 codes of a Gaussian matrix and block scales that keep x . w of order one."""
    codes = (torch.randn((n, k), device=DEV, generator=gen) * 64).to(torch.float8_e4m3fn).view(torch.uint8)
    block = 32 if rule == "e8m0" else 128
    shape = (-(-n // block), k // block)
    if rule == "e8m0":
        scales = torch.randint(0, 3, shape, device=DEV, generator=gen) + (126 - round(math.log2(64 * math.sqrt(k))))
        return codes, scales.to(torch.uint8)
    return codes, (torch.rand(shape, device=DEV, generator=gen) + 0.5) / (64 * math.sqrt(k))


def _popularity(c):
    """Chance of every expert to be the one a route slot asks for: Zipf with exponent `skew` (0: uniform)."""
    p = np.arange(1, c["experts"] + 1, dtype=np.float64) ** -c.get("skew", 0.0)
    return p / p.sum()


def _routes(c, gen, rows):
    """top-k distinct experts per row by the case's popularity, and weights that sum to one."""
    p = torch.tensor(_popularity(c), device=DEV, dtype=torch.float32)
    p = p[torch.randperm(c["experts"], device=DEV, generator=gen)]
    race = torch.empty((rows, c["experts"]), device=DEV).exponential_(generator=gen) / p
    ids = race.topk(c["topk"], dim=1, largest=False).indices.to(torch.int32)
    w = torch.rand((rows, c["topk"]), device=DEV, generator=gen) + 0.1
    return ids, w / w.sum(1, keepdim=True)


def prepare(c, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind = c["kind"]
    s = {"case": c}
    if kind == "layer":
        s["bank"] = _bank(c, gen, c["layers"])
        s["x"] = [_x(gen, c["hidden"]) for _ in range(c["layers"])]
        s["logits"] = [torch.randn(c["experts"], device=DEV, generator=gen) for _ in range(c["layers"])]
        s["bias"] = torch.randn(c["experts"], device=DEV, generator=gen) * 0.05
    elif kind == "block":
        s["bank"], s["x"] = _bank(c, gen), _x(gen, c["hidden"])
        s["gate"] = (torch.randn((c["experts"], c["hidden"]), device=DEV, generator=gen) / math.sqrt(c["hidden"])).to(torch.bfloat16)
        s["bias"] = torch.randn(c["experts"], device=DEV, generator=gen) * 0.05
    elif kind == "batch":
        s["bank"], s["x"] = _bank(c, gen), _x(gen, c["tokens"], c["hidden"])
        s["slots"], s["w"] = _routes(c, gen, c["tokens"])
    elif kind == "prefill":
        s["bank"], s["x"] = _bank(c, gen), _x(gen, c["tokens"], c["hidden"])
        s["ids"], s["w"] = _routes(c, gen, c["tokens"])
    elif kind == "trunk":
        s["x1"], s["x2"] = (_x(gen, c["rows"], c[k]) if c["rows"] > 1 else _x(gen, c[k]) for k in ("k1", "k2"))
        s["w1"], s["w2"] = _fp8_matrix(gen, c["n1"], c["k1"], c["rule"]), _fp8_matrix(gen, c["n2"], c["k2"], c["rule"])
    elif kind == "shared":
        s["x"] = _x(gen, c["rows"], c["hidden"])
    else:
        s["x"] = torch.randn((c["rows"], c["hidden"]) if c["rows"] > 1 else c["hidden"], device=DEV, generator=gen)
        s["w"] = (torch.randn((c["vocab"], c["hidden"]), device=DEV, generator=gen) / math.sqrt(c["hidden"])).to(torch.bfloat16)
    if kind in ("block", "shared"):
        for name, n, k in (("1", c["inter"], c["hidden"]), ("2", c["hidden"], c["inter"]), ("3", c["inter"], c["hidden"])):
            s["s" + name] = _fp8_matrix(gen, n, k, c["rule"])
    return s


# ---- one pass -------------------------------------------------------------------------------------

def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "layer":
        return [cb.moe_layer_decode(x, logits, s["bank"], layer=i, topk=c["topk"], bias=s["bias"], router=c["router"])
                for i, (x, logits) in enumerate(zip(s["x"], s["logits"]))]
    if kind == "block":
        out, r = cb.moe_layer_forward(s["x"], layer_id=0, gate_weight=s["gate"], gate_bias=s["bias"], expert_store=s["bank"],
                                      shared_w1=s["s1"][0], shared_w1_scales=s["s1"][1], shared_w2=s["s2"][0],
                                      shared_w2_scales=s["s2"][1], shared_w3=s["s3"][0], shared_w3_scales=s["s3"][1], topk=c["topk"])
        return [out, r.indices, r.weights, r.scores]
    if kind == "batch":
        return cb.moe_forward(s["x"], s["slots"], s["w"], s["bank"])
    if kind == "prefill":
        return cb.moe_prefill_grouped(s["x"], s["ids"], s["w"], s["bank"], mxfp4_act=c["act"] == "mxfp4")
    if kind == "trunk":
        return [cb.fp8_linear(s["x1"], *s["w1"]), cb.fp8_linear(s["x2"], *s["w2"])]
    if kind == "shared":
        return ops.shared_expert_forward_batched(s["x"], w1=s["s1"][0], w1_scales=s["s1"][1], w2=s["s2"][0], w2_scales=s["s2"][1],
                                                 w3=s["s3"][0], w3_scales=s["s3"][1])
    return ops.bf16_gemv_f32(s["x"], s["w"])


# ---- what a pass cannot do without ----------------------------------------------------------------

def _distinct(c, rows):
    """Expected number of distinct experts that `rows` tokens route to."""
    if rows == 1:
        return c["topk"]
    p, lo, hi = _popularity(c), 0.0, 1e9
    for _ in range(200):  # chance of a token to take expert e: 1 - exp(-z p_e), with z such that they sum to k
        z = (lo + hi) / 2
        lo, hi = (z, hi) if (1 - np.exp(-z * p)).sum() < c["topk"] else (lo, z)
    return float((1 - np.exp(-z * p * rows)).sum())


def _fp8_bytes(n, k, rule):
    return n * k + (-(-n // 32) * (k // 32) if rule == "e8m0" else -(-n // 128) * (k // 128) * 4)


def work(c):
    kind = c["kind"]
    if kind in ("layer", "block", "batch", "prefill"):
        h, i = c["hidden"], c["inter"]
        expert = 3 * h * i * 17 // 32 if c["bank"] == "fp4" else 3 * h * i * 9 // 32
        rows, layers = c.get("tokens", 1), c.get("layers", 1)
        n_bytes = layers * (_distinct(c, rows) * expert + rows * (h * 2 + h * 4 + c["topk"] * 8))
        flops = layers * 6 * rows * c["topk"] * h * i
        if kind == "layer":
            n_bytes += layers * c["experts"] * 12
        if kind == "block":
            n_bytes += c["experts"] * (h * 2 + 12) - h * 2 + 2 * _fp8_bytes(i, h, c["rule"]) + _fp8_bytes(h, i, c["rule"])
            flops += 6 * h * i + 2 * c["experts"] * h
        return {"bytes": n_bytes, "flops": flops}
    if kind == "trunk":
        mats = ((c["n1"], c["k1"]), (c["n2"], c["k2"]))
        return {"bytes": sum(_fp8_bytes(n, k, c["rule"]) + c["rows"] * 2 * (n + k) for n, k in mats), "flops": sum(2 * c["rows"] * n * k for n, k in mats)}
    if kind == "shared":
        h, i = c["hidden"], c["inter"]
        return {"bytes": 2 * _fp8_bytes(i, h, c["rule"]) + _fp8_bytes(h, i, c["rule"]) + c["rows"] * 4 * h, "flops": 6 * c["rows"] * h * i}
    return {"bytes": c["vocab"] * c["hidden"] * 2 + c["rows"] * 4 * (c["hidden"] + c["vocab"]), "flops": 2 * c["rows"] * c["vocab"] * c["hidden"]}


def tolerance(c):
    kind = c["kind"]
    if kind == "head":
        return {"rel": 1e-5}  # fp32 sums
    if kind == "trunk":
        return {"rel": 5e-3}  # bf16 results
    if kind in ("block", "shared"):
        return {"rel": 1e-2}  # a hidden value that rounds the other way in bf16 can move one FP8 step
    if kind == "prefill" and c["act"] == "mxfp4":
        return {"rel": 1e-2}  # ... or one FP4 step
    if c["bank"] == "fp4" and kind in ("layer", "batch"):
        return {"rel": 1e-3}  # fp32 results of hidden values that enter the second product with at least 11 bits
    return {"rel": 5e-3}      # every expert's projections and output are rounded to bf16
