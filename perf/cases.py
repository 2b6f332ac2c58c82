"""The work that a user of this library has it do, as measurable cases.

Each case is one pass through the public entry points, the way a serving or a training program calls
them: the attention side of a decode step, decode attention over a large paged cache, prefill over packed
and over cached sequences, a mixture-of-experts block, the routers and the activation on their own.
`listed()` holds the sizes that stand for them; `draw()` spreads over the same ranges.

Lengths of a batch are spread evenly over their range and shuffled by the seed, so that a case's work does
not depend on the seed while its inputs do.
"""
from __future__ import annotations

import math

import torch

import dlcompiler_b200 as dl

DEVICE = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}


def listed():
    return [
        # One decode step of an attention layer for four running requests: norm with residual, rotary, cache
        # update, attention.  The smallest calls a server makes; latency and launches count.
        {"name": "decode_step_small", "kind": "decode_step", "batch": 4, "lo": 100, "hi": 1000, "page": 16,
         "hq": 32, "hkv": 8, "dim": 128, "dtype": "fp16", "window": 0},
        # Decode attention of a full server: 64 requests of 1k to 32k tokens, 64-token pages.
        {"name": "decode_large", "kind": "decode", "batch": 64, "lo": 1024, "hi": 32768, "page": 64,
         "hq": 32, "hkv": 8, "dim": 128, "dtype": "bf16", "window": 0, "softcap": 0.0},
        # Decode attention over a token-granular cache (request -> token table).
        {"name": "token_decode", "kind": "token_decode", "batch": 16, "lo": 1024, "hi": 32768,
         "hq": 32, "hkv": 8, "dim": 128, "dtype": "bf16"},
        # Prefill of a packed batch of ordinary prompts of odd lengths.
        {"name": "prefill_short", "kind": "prefill", "batch": 13, "lo": 17, "hi": 901,
         "hq": 32, "hkv": 8, "dim": 128, "dtype": "bf16", "causal": True},
        # Prefill of four long prompts, with the log-sum-exp a later merge needs.
        {"name": "prefill_long", "kind": "prefill", "batch": 4, "lo": 8192, "hi": 8192,
         "hq": 32, "hkv": 8, "dim": 128, "dtype": "bf16", "causal": True},
        # Chunked prefill: new tokens of running prompts join the paged cache (keys rotated on the way in)
        # and attend to what is cached already.
        {"name": "prefill_chunked", "kind": "chunked", "batch": 4, "lo": 256, "hi": 768, "past": 8000, "page": 64,
         "hq": 32, "hkv": 8, "dim": 128, "dtype": "bf16", "window": 0},
        # A mixture-of-experts block during decode: 32 tokens, every expert's weights are read.
        {"name": "moe_decode", "kind": "moe", "tokens": 32, "hidden": 4096, "inter": 14336, "experts": 8, "topk": 2,
         "router": "softmax", "dtype": "bf16"},
        # The same block during prefill.
        {"name": "moe_prefill", "kind": "moe", "tokens": 4096, "hidden": 4096, "inter": 14336, "experts": 8,
         "topk": 2, "router": "softmax", "dtype": "bf16"},
        # Many small experts behind the group-limited router: each expert gets a few dozen rows.
        {"name": "moe_many_experts", "kind": "moe", "tokens": 2000, "hidden": 2048, "inter": 1024, "experts": 256,
         "topk": 8, "router": "grouped", "dtype": "bf16"},
        # The group-limited router over a prefill batch.
        {"name": "router", "kind": "router", "tokens": 16384, "experts": 256, "groups": 8, "keep": 4, "topk": 8},
        # Training step of the capacity-limited gate: forward and backward through weights and auxiliary loss.
        {"name": "gate_training", "kind": "gate", "tokens": 4096, "experts": 64, "topk": 8, "factor": 1.0,
         "full_grad": True, "dtype": "fp32"},
        # The gated activation of a dense MLP.
        {"name": "silu_and_mul", "kind": "silu", "tokens": 4096, "inter": 11008, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode_step", "decode", "token_decode", "prefill", "prefill", "chunked", "moe", "moe", "moe",
                       "router", "gate", "silu"])
    hq, hkv = rng.choice([(32, 8), (32, 8), (16, 16), (24, 8), (64, 8), (28, 4)])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "decode_step":
        batch = _log(rng, 1, 64)
        hi = _log(rng, 64, 8192)
        return {"kind": kind, "batch": batch, "lo": max(hi // 10, 1), "hi": hi, "page": rng.choice([16, 64]),
                "hq": hq, "hkv": hkv, "dim": rng.choice([64, 128]), "dtype": dtype,
                "window": rng.choice([0, 0, 0, 1024])}
    if kind == "decode":
        hi = _log(rng, 256, 32768)
        batch = min(_log(rng, 1, 64), (1 << 20) // hi)
        return {"kind": kind, "batch": batch, "lo": max(hi // rng.choice([2, 30]), 1), "hi": hi,
                "page": rng.choice([16, 64]), "hq": 32, "hkv": 8, "dim": rng.choice([64, 96, 128, 128]),
                "dtype": dtype, "window": rng.choice([0, 0, 0, 4096]), "softcap": rng.choice([0.0, 0.0, 0.0, 30.0])}
    if kind == "token_decode":
        hi = _log(rng, 256, 32768)
        return {"kind": kind, "batch": _log(rng, 1, 32), "lo": max(hi // 30, 1), "hi": hi, "hq": 32, "hkv": 8,
                "dim": rng.choice([64, 128, 128]), "dtype": dtype}
    if kind == "prefill":
        causal = rng.random() < 0.85
        hi = _log(rng, 16, 8192 if causal else 4096)
        batch = max(1, min(_log(rng, 1, 16), 32768 // hi))
        return {"kind": kind, "batch": batch, "lo": max(hi // rng.choice([1, 4, 40]), 1), "hi": hi,
                "hq": min(hq, 32), "hkv": hkv, "dim": rng.choice([64, 80, 96, 128, 128, 128]), "dtype": dtype,
                "causal": causal}
    if kind == "chunked":
        hi = _log(rng, 16, 2048)
        return {"kind": kind, "batch": _log(rng, 1, 8), "lo": max(hi // 3, 1), "hi": hi, "past": rng.choice([0, 1]) *
                _log(rng, 64, 16000), "page": rng.choice([16, 64]), "hq": min(hq, 32), "hkv": hkv,
                "dim": rng.choice([64, 128, 128]), "dtype": dtype, "window": rng.choice([0, 0, 0, 1024])}
    if kind == "moe":
        hidden, inter, experts, topk, router = rng.choice(
            [(4096, 14336, 8, 2, "softmax"), (4096, 14336, 8, 2, "softmax"), (2048, 1024, 256, 8, "grouped"),
             (2048, 1408, 64, 6, "softmax"), (1024, 2816, 32, 4, "softmax")])
        return {"kind": kind, "tokens": _log(rng, 1, 4096), "hidden": hidden, "inter": inter, "experts": experts,
                "topk": topk, "router": router, "dtype": dtype}
    if kind == "router":
        experts, groups, keep, topk = rng.choice([(256, 8, 4, 8), (256, 8, 4, 8), (64, 1, 1, 6), (128, 4, 2, 8)])
        return {"kind": kind, "tokens": _log(rng, 16, 32768), "experts": experts, "groups": groups, "keep": keep,
                "topk": topk}
    if kind == "gate":
        experts, topk = rng.choice([8, 16, 64, 128]), rng.choice([1, 2, 4, 8])
        # a capacity above the number of tokens has no list to fill it with
        factor = rng.choice([f for f in (1.0, 1.25, 2.0) if f * topk <= experts])
        return {"kind": kind, "tokens": _log(rng, 256, 16384), "experts": experts, "topk": topk, "factor": factor,
                "full_grad": rng.random() < 0.6, "dtype": "fp32"}
    return {"kind": "silu", "tokens": _log(rng, 1, 8192), "inter": rng.choice([_log(rng, 500, 14336), 4096, 11008]),
            "dtype": rng.choice(["bf16", "bf16", "fp16", "fp32"])}


# ------------------------------------------------------------------------------------------------- inputs
def _lengths(case):
    """The batch's lengths: evenly spread over [lo, hi], both ends included."""
    n, lo, hi = case["batch"], case["lo"], case["hi"]
    return [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _past(case):
    """Tokens already cached per sequence of a chunked prefill: spread over [past / 8, past]."""
    n, hi = case["batch"], case["past"]
    return [hi] if n == 1 else [hi // 8 + (hi - hi // 8) * i // (n - 1) for i in range(n)]


class _Inputs:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE)
        self.g.manual_seed(seed)

    def normal(self, *shape, dtype, std=1.0):
        x = torch.randn(shape, generator=self.g, device=DEVICE, dtype=dtype)
        return x if std == 1.0 else x.mul_(std)

    def shuffled(self, values):
        order = torch.randperm(len(values), generator=self.g, device=DEVICE).tolist()
        return [values[i] for i in order]

    def pages(self, lens, page):
        """(block table int32 [batch, most pages], number of pages): a random permutation of the pool."""
        need = [(n + page - 1) // page for n in lens]
        pool = torch.randperm(sum(need), generator=self.g, device=DEVICE).to(torch.int32)
        table = torch.zeros(len(lens), max(need), dtype=torch.int32, device=DEVICE)
        at = 0
        for b, n in enumerate(need):
            table[b, :n] = pool[at:at + n]
            at += n
        return table, at


def _rotary(positions, dim, dtype):
    """cos / sin rows of the usual rotary embedding (base 10000, both halves alike) at integer positions."""
    inv = 10000.0 ** (-torch.arange(0, dim, 2, device=DEVICE, dtype=torch.float64) / dim)
    a = positions.to(torch.float64)[:, None] * inv
    a = torch.cat([a, a], dim=-1)
    return a.cos().to(dtype), a.sin().to(dtype)


def _ints(values, dtype=torch.int32):
    return torch.tensor(values, dtype=dtype, device=DEVICE)


def _starts(lens):
    at, out = 0, []
    for n in lens:
        out.append(at)
        at += n
    return out


def prepare(case, seed):
    kind, rnd = case["kind"], _Inputs(seed)
    dtype = DTYPES[case.get("dtype", "fp32")]
    s = {"case": case}
    if kind in ("decode_step", "decode", "token_decode", "prefill", "chunked"):
        hq, hkv, d = case["hq"], case["hkv"], case["dim"]
        s["scale"] = d ** -0.5

    if kind == "decode_step":
        lens, n = rnd.shuffled(_lengths(case)), case["batch"]
        hidden = hq * d
        s["x"], s["residual"] = rnd.normal(n, hidden, dtype=dtype), rnd.normal(n, hidden, dtype=dtype)
        s["norm_weight"] = rnd.normal(hidden, dtype=dtype, std=0.1).add_(1.0)
        # q, k and v as a fused projection leaves them: views of one buffer
        qkv = rnd.normal(n, (hq + 2 * hkv) * d, dtype=dtype)
        s["q"], s["k"], s["v"] = (t.view(n, -1, d) for t in qkv.split([hq * d, hkv * d, hkv * d], dim=-1))
        s["cos"], s["sin"] = _rotary(_ints(lens) - 1, d, dtype)
        s["table"], pages = rnd.pages(lens, case["page"])
        s["k_cache"] = rnd.normal(pages, case["page"], hkv, d, dtype=dtype)
        s["v_cache"] = rnd.normal(pages, case["page"], hkv, d, dtype=dtype)
        s["start"], s["one"], s["lens"] = _ints(list(range(n))), _ints([1] * n), _ints(lens)
        s["most"] = max(lens)
    elif kind in ("decode", "token_decode"):
        lens, n = rnd.shuffled(_lengths(case)), case["batch"]
        s["q"] = rnd.normal(n, hq, d, dtype=dtype)
        s["o"] = torch.empty_like(s["q"])
        s["table"], pages = rnd.pages(lens, case.get("page", 1))
        shape = (pages, case["page"], hkv, d) if kind == "decode" else (pages, hkv, d)
        s["k_cache"], s["v_cache"] = rnd.normal(*shape, dtype=dtype), rnd.normal(*shape, dtype=dtype)
        s["start"], s["one"], s["lens"] = _ints(list(range(n))), _ints([1] * n), _ints(lens)
        s["most"] = max(lens)
    elif kind == "prefill":
        lens = rnd.shuffled(_lengths(case))
        total = sum(lens)
        s["q"] = rnd.normal(total, hq, d, dtype=dtype)
        s["k"], s["v"] = rnd.normal(total, hkv, d, dtype=dtype), rnd.normal(total, hkv, d, dtype=dtype)
        s["o"] = torch.empty_like(s["q"])
        s["lse"] = torch.empty(hq, total, dtype=torch.float32, device=DEVICE)
        s["start"], s["lens"], s["most"] = _ints(_starts(lens)), _ints(lens), max(lens)
    elif kind == "chunked":
        lens, past = rnd.shuffled(_lengths(case)), rnd.shuffled(_past(case))
        total, full = sum(lens), [a + b for a, b in zip(lens, past)]
        s["q"] = rnd.normal(total, hq, d, dtype=dtype)
        s["k"], s["v"] = rnd.normal(total, hkv, d, dtype=dtype), rnd.normal(total, hkv, d, dtype=dtype)
        s["o"] = torch.empty_like(s["q"])
        s["cos"], s["sin"] = _rotary(torch.cat([torch.arange(p, p + n, device=DEVICE) for n, p in zip(lens, past)]),
                                     d, dtype)
        s["table"], pages = rnd.pages(full, case["page"])
        s["k_cache"] = rnd.normal(pages, case["page"], hkv, d, dtype=dtype)
        s["v_cache"] = rnd.normal(pages, case["page"], hkv, d, dtype=dtype)
        s["start"], s["lens"], s["full"], s["most"] = _ints(_starts(lens)), _ints(lens), _ints(full), max(lens)
    elif kind == "moe":
        t, h, i, e = case["tokens"], case["hidden"], case["inter"], case["experts"]
        s["x"], s["residual"] = rnd.normal(t, h, dtype=dtype), rnd.normal(t, h, dtype=dtype)
        s["norm_weight"] = rnd.normal(h, dtype=dtype, std=0.1).add_(1.0)
        # trained routers load their experts unevenly: a spread between experts beside the one between tokens
        s["logits"] = rnd.normal(t, e, dtype=torch.float32) + rnd.normal(e, dtype=torch.float32, std=0.3)
        s["bias"] = rnd.normal(e, dtype=torch.float32, std=0.01)
        s["w1"] = rnd.normal(e, 2 * i, h, dtype=dtype, std=0.02)
        s["w2"] = rnd.normal(e, h, i, dtype=dtype, std=0.02)
    elif kind == "router":
        s["logits"] = rnd.normal(case["tokens"], case["experts"], dtype=torch.float32)
        s["bias"] = rnd.normal(case["experts"], dtype=torch.float32, std=0.01)
    elif kind == "gate":
        t, e, k = case["tokens"], case["experts"], case["topk"]
        s["logits"] = rnd.normal(t, e, dtype=dtype).requires_grad_()
        s["grad_aux"] = rnd.normal(1, dtype=dtype).reshape(())
        s["grad_weights"] = rnd.normal(k * t, dtype=dtype)
    else:
        s["x"] = rnd.normal(case["tokens"], 2 * case["inter"], dtype=dtype)
    return s


# ------------------------------------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode_step":
        x, residual = dl.rms_norm(s["x"], s["norm_weight"], 1e-6, residual=s["residual"])
        q, k = dl.apply_rotary_pos_emb(s["q"], s["k"], s["cos"], s["sin"])
        dl.fill_kv_cache(k, s["v"], s["k_cache"], s["v_cache"], s["start"], s["one"], s["lens"], 1, s["table"])
        o = torch.empty_like(q)
        dl.paged_attention_fwd(q, s["k_cache"], s["v_cache"], o, s["table"], s["start"], s["one"], s["lens"],
                               s["most"], window_size=case["window"] or None, sm_scale=s["scale"])
        return {"x": x, "residual": residual, "q": q, "k": k, "o": o, "k_cache": s["k_cache"],
                "v_cache": s["v_cache"]}
    if kind == "decode":
        dl.paged_attention_fwd(s["q"], s["k_cache"], s["v_cache"], s["o"], s["table"], s["start"], s["one"],
                               s["lens"], s["most"], window_size=case["window"] or None, sm_scale=s["scale"],
                               logit_softcapping=case["softcap"] or None)
        return s["o"]
    if kind == "token_decode":
        dl.decode_attention_fwd(s["q"], s["k_cache"], s["v_cache"], s["o"], s["table"], s["start"], None, s["lens"],
                                None, s["most"], s["scale"])
        return s["o"]
    if kind == "prefill":
        dl.context_attention_fwd(s["q"], s["k"], s["v"], s["o"], s["start"], s["lens"], s["most"], lse=s["lse"],
                                 causal=case["causal"])
        return s["o"], s["lse"]
    if kind == "chunked":
        dl.fill_kv_cache(s["k"], s["v"], s["k_cache"], s["v_cache"], s["start"], s["lens"], s["full"], s["most"],
                         s["table"], cos=s["cos"], sin=s["sin"])
        dl.paged_attention_fwd(s["q"], s["k_cache"], s["v_cache"], s["o"], s["table"], s["start"], s["lens"],
                               s["full"], s["most"], window_size=case["window"] or None, sm_scale=s["scale"],
                               q_cos=s["cos"], q_sin=s["sin"])
        return s["o"], s["k_cache"], s["v_cache"]
    if kind == "moe":
        x, residual = dl.rms_norm(s["x"], s["norm_weight"], 1e-6, residual=s["residual"])
        if case["router"] == "grouped":
            ids, weights = dl.grouped_topk_gating(s["logits"], s["bias"], case["topk"], 8, 4, 2.5)
        else:
            weights, ids = dl.softmax_topk(s["logits"], case["topk"], renormalize=True)
        y = dl.fused_moe(x, s["w1"], s["w2"], weights, ids, case["topk"])
        return {"x": x, "residual": residual, "ids": ids, "weights": weights, "y": y}
    if kind == "router":
        return dl.grouped_topk_gating(s["logits"], s["bias"], case["topk"], case["groups"], case["keep"], 2.5)
    if kind == "gate":
        aux, slots, weights, select = dl.topk_gating(s["logits"], case["topk"], case["factor"], 2, case["full_grad"])
        outs, grads = (aux, weights), (s["grad_aux"], s["grad_weights"])
        if not case["full_grad"]:
            outs, grads = outs[:1], grads[:1]
        grad, = torch.autograd.grad(outs, s["logits"], grads)
        return {"aux": aux, "slots": slots, "weights": weights, "select": select, "grad": grad}
    return dl.silu_and_mul(s["x"])


# ------------------------------------------------------------------------------------------------- its work
def work(case):
    kind, es = case["kind"], SIZE[case.get("dtype", "fp32")]
    if kind in ("decode_step", "decode", "token_decode"):
        window = case.get("window") or 0
        seen = sum(min(n, window + 1) if window else n for n in _lengths(case))
        rows = case["batch"] * case["hq"] * case["dim"] * es
        nbytes = 2 * seen * case["hkv"] * case["dim"] * es + 2 * rows
        if kind == "decode_step":
            kv = case["batch"] * case["hkv"] * case["dim"] * es
            nbytes += 4 * rows + rows // case["batch"]      # x, residual and their sums; the norm's weight
            nbytes += 5 * kv + 2 * rows // case["hq"]       # k and v read, k and both cache rows written; cos, sin
            nbytes += rows                                  # q before its rotation
        return {"bytes": nbytes, "flops": 4 * seen * case["hq"] * case["dim"]}
    if kind == "prefill":
        lens = _lengths(case)
        pairs = sum(n * (n + 1) // 2 if case["causal"] else n * n for n in lens)
        nbytes = 2 * sum(lens) * (case["hq"] + case["hkv"]) * case["dim"] * es + sum(lens) * case["hq"] * 4
        return {"bytes": nbytes, "flops": 4 * pairs * case["hq"] * case["dim"]}
    if kind == "chunked":
        lens, past, w = _lengths(case), _past(case), case["window"]
        pairs = sum((min(p + i + 1, w + 1) if w else p + i + 1) for n, p in zip(lens, past) for i in range(n))
        total = sum(lens)
        cached = sum((min(p, w) if w else p) for p in past)
        nbytes = 2 * total * case["hq"] * case["dim"] * es + (4 * total + 2 * cached) * case["hkv"] * case["dim"] * es
        nbytes += 2 * total * case["dim"] * es
        return {"bytes": nbytes, "flops": 4 * pairs * case["hq"] * case["dim"]}
    if kind == "moe":
        t, h, i, e, k = (case[n] for n in ("tokens", "hidden", "inter", "experts", "topk"))
        touched = e * (1.0 - (1.0 - k / e) ** t)            # experts that some token is expected to choose
        return {"bytes": touched * 3 * h * i * es + 5 * t * h * es + t * e * 4 + 2 * t * k * 4,
                "flops": 2 * t * k * 3 * h * i}
    if kind == "router":
        return {"bytes": case["tokens"] * (case["experts"] * 4 + case["topk"] * 8) + case["experts"] * 4, "flops": 0}
    if kind == "gate":
        t, e, k = case["tokens"], case["experts"], case["topk"]
        capacity = math.ceil(t / e * k * case["factor"])
        return {"bytes": 2 * t * e * 4 + t * k * 12 + e * capacity * 8, "flops": 0}
    return {"bytes": 3 * case["tokens"] * case["inter"] * es, "flops": 0}


# Four times the relative error (2-norm) of each path against itself in 64 bits: measured 2.1e-3 for bf16 attention
# outputs (2.7e-4 for fp16), 3.4e-3 where q and k are rotated in their own type first (4.2e-4), 4.3e-3 for the
# mixture-of-experts block (5.3e-4), 1.7e-3 for one rounding (2.1e-4), 1e-7 at most for 32-bit results.  The largest
# single difference was 6 to 14 times that.
REL = {"decode_step": 8e-3, "decode": 8e-3, "token_decode": 8e-3, "prefill": 8e-3, "chunked": 1.4e-2, "moe": 1.7e-2,
       "silu": 6.6e-3}


def tolerance(case):
    """Whole numbers (expert ids, slots, token lists) are the same; floating results within what the types give."""
    dtype = case.get("dtype", "fp32")
    rel = 1e-6 if dtype == "fp32" else REL[case["kind"]] / (8 if dtype == "fp16" else 1)
    return {"rel": rel, "max": 16 * rel, "differ": 0.0}
