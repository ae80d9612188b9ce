"""What this framework's users have it do, as a list of cases with sizes: decode steps of one
engine, of a whole model's layer stack and of a serving batch, attention over one very long
sequence, grouped queries, and prompts that enter the cache in bulk.  Sizes are those of the
benchmark, the tests and their neighbourhood; every cache is used through the public Python
classes with CUDA tensors.

Caches are rings.  The decode cases run at a full ring (capacity = context), the steady state of
a long generation: every step evicts one token and attends to `context` tokens, so a case costs
the same however often it is run.
"""
from __future__ import annotations

import math

import torch

import adaptq_b200

SEED_MASK = 2**64 - 1


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # One Engine with upstream's defaults (sparse V at 0.95), one token: the smallest call there is.
        {"name": "engine_defaults_4x2048", "kind": "engine", "heads": 4, "dim": 64, "k_bits": 4, "v_bits": 2, "context": 2048,
         "dense": False, "dist": "normal"},
        # The first tokens of a conversation: Engine defaults attend to the FP32 window (up to 512 tokens).
        {"name": "engine_window_8x300", "kind": "window", "heads": 8, "dim": 128, "k_bits": 4, "v_bits": 4, "context": 300,
         "dist": "normal"},
        # Batch-1 decode of a small model, all layers in one call; layer 0 keeps FP32 keys.
        {"name": "stack_24x14_k4v2_1024", "kind": "stack", "layers": 24, "heads": 14, "dim": 64, "k_bits": 4, "v_bits": 2,
         "context": 1024, "dist": "student4"},
        {"name": "stack_22x4_k3v2_2048", "kind": "stack", "layers": 22, "heads": 4, "dim": 64, "k_bits": 3, "v_bits": 2,
         "context": 2048, "dist": "lognormal"},
        # A serving batch in lockstep: 32 sequences x 32 layers x 8 KV heads, 8192 tokens each (the benchmark's shape, an eighth of it).
        {"name": "batch_8192x8192_k4v2", "kind": "batch", "heads": 8192, "dim": 128, "k_bits": 4, "v_bits": 2, "context": 8192,
         "dist": "outlier"},
        # Odd sizes: a padded head dimension, a context that fills no tile, fewer heads than a whole number of waves.
        {"name": "batch_334x3001_d96_k4v3", "kind": "batch", "heads": 334, "dim": 96, "k_bits": 4, "v_bits": 3, "context": 3001,
         "dist": "normal"},
        # One very long sequence, one layer (the benchmark's long-context shapes).
        {"name": "long_32x131072_k2v2", "kind": "long", "heads": 32, "dim": 128, "k_bits": 2, "v_bits": 2, "context": 131072,
         "dist": "student3"},
        {"name": "long_32x131072_k4v4", "kind": "long", "heads": 32, "dim": 128, "k_bits": 4, "v_bits": 4, "context": 131072,
         "dist": "student3"},
        # Grouped-query serving step from a bf16 model: 64 sequences x 8 KV heads, four queries per KV head.
        {"name": "grouped_512x4096_g4_k4v2", "kind": "grouped", "batch": 64, "heads": 8, "q_per_kv": 4, "dim": 128, "k_bits": 4,
         "v_bits": 2, "context": 4096, "dense": True, "bf16": True, "dist": "normal"},
        # The same module with upstream's defaults (sparse V), one query per head.
        {"name": "grouped_128x2048_sparse", "kind": "grouped", "batch": 16, "heads": 8, "q_per_kv": 1, "dim": 128, "k_bits": 4,
         "v_bits": 4, "context": 2048, "dense": False, "bf16": False, "dist": "normal"},
        # A long prompt enters one layer's cache, then its first query (the benchmark's bulk append).
        {"name": "prefill_32768x8_k4v4", "kind": "prefill", "tokens": 32768, "heads": 8, "dim": 128, "k_bits": 4, "v_bits": 4,
         "dist": "normal"},
        # A short prompt enters all layers of a small model at once, then its first query.
        {"name": "stack_prefill_517_24x14", "kind": "stack_prefill", "tokens": 517, "layers": 24, "heads": 14, "dim": 64,
         "k_bits": 4, "v_bits": 2, "dist": "student4"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["engine", "window", "stack", "batch", "batch", "long", "grouped", "grouped", "prefill", "stack_prefill"])
    kb, vb = rng.choice([2, 3, 4, 4]), rng.choice([2, 2, 3, 4])
    if kind == "engine":
        return {"kind": kind, "heads": _log(rng, 1, 32), "dim": rng.choice([64, 96, 128]), "k_bits": kb, "v_bits": vb,
                "context": _log(rng, 520, 8192), "dense": rng.random() < 0.4, "dist": "normal"}
    if kind == "window":
        return {"kind": kind, "heads": _log(rng, 1, 32), "dim": rng.choice([64, 80, 128]), "k_bits": kb, "v_bits": vb,
                "context": _log(rng, 16, 512), "dist": "normal"}
    if kind == "stack":
        return {"kind": kind, "layers": rng.randint(8, 32), "heads": rng.randint(2, 16), "dim": rng.choice([64, 128]),
                "k_bits": rng.choice([3, 4]), "v_bits": rng.choice([2, 2, 4]), "context": _log(rng, 256, 4096), "dist": "student4"}
    if kind == "batch":
        heads = _log(rng, 128, 8192)
        return {"kind": kind, "heads": heads, "dim": rng.choice([64, 96, 128, 128, 128]), "k_bits": kb, "v_bits": vb,
                "context": min(_log(rng, 500, 8192), 2**25 // heads), "dist": "outlier"}
    if kind == "long":
        return {"kind": kind, "heads": _log(rng, 4, 32), "dim": 128, "k_bits": kb, "v_bits": vb, "context": _log(rng, 16000, 131072),
                "dist": "student3"}
    if kind == "grouped":
        dense = rng.random() < 0.75
        return {"kind": kind, "batch": _log(rng, 1, 64), "heads": rng.choice([4, 8]), "q_per_kv": rng.choice([1, 2, 4, 7, 8]),
                "dim": rng.choice([64, 128, 128]), "k_bits": kb, "v_bits": vb, "context": _log(rng, 520, 8192 if dense else 4096),
                "dense": dense, "bf16": rng.random() < 0.5, "dist": "normal"}
    if kind == "prefill":
        return {"kind": kind, "tokens": _log(rng, 128, 32768), "heads": _log(rng, 4, 16), "dim": rng.choice([64, 96, 128, 128]),
                "k_bits": kb, "v_bits": vb, "dist": "normal"}
    return {"kind": kind, "tokens": _log(rng, 32, 2048), "layers": rng.randint(8, 32), "heads": rng.randint(2, 16),
            "dim": rng.choice([64, 128]), "k_bits": rng.choice([3, 4]), "v_bits": rng.choice([2, 4]), "dist": "student4"}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _values(shape, dist, gen, channel_scale=None):
    """float32 values as the path meets them: plain normal, heavy-tailed (Student-t), 1 % large
    outliers, or a fixed log-normal scale per channel."""
    x = torch.randn(shape, device="cuda", generator=gen)
    if dist in ("student3", "student4"):
        nu = int(dist[-1])
        chi = torch.randn(shape, device="cuda", generator=gen).square_()
        for _ in range(nu - 1):
            chi += torch.randn(shape, device="cuda", generator=gen).square_()
        x *= torch.rsqrt(chi / nu)
    elif dist == "outlier":
        big = torch.rand(shape, device="cuda", generator=gen) < 0.01
        x = torch.where(big, x * 20.0, x)
    elif dist == "lognormal":
        x *= channel_scale
    return x


def _fill(append, tokens, lead, dim, dist, gen):
    """Append `tokens` tokens in chunks of at most 2^26 values, as a prefill does."""
    scale = torch.exp(0.5 * torch.randn(lead + (dim,), device="cuda", generator=gen)) if dist == "lognormal" else None
    step = max(1, 2**26 // (math.prod(lead) * dim))
    for t in range(0, tokens, step):
        shape = (min(step, tokens - t),) + lead + (dim,)
        append(_values(shape, dist, gen, scale), _values(shape, dist, gen, scale))
    return scale


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) & (2**63 - 1))
    kind, dist, dim = c["kind"], c["dist"], c["dim"]
    s = {"kind": kind}
    if kind in ("engine", "window"):
        kw = dict(v_mass=0.0, hybrid_thresh=0) if c.get("dense") else {}
        cap = c["context"] if kind == "engine" else 4096
        e = adaptq_b200.Engine(dim, c["heads"], c["k_bits"], c["v_bits"], cap, 42, **kw)
        _fill(e.append_many, c["context"], (c["heads"],), dim, dist, gen)
        s["engine"] = e
        s["k"], s["v"], s["q"] = (_values((c["heads"], dim), dist, gen) for _ in range(3))
    elif kind in ("stack", "stack_prefill"):
        lead = (c["layers"], c["heads"])
        kb = [16] + [c["k_bits"]] * (c["layers"] - 1)  # layer 0 keeps FP32 keys
        n = c["context"] if kind == "stack" else c["tokens"]
        s["stack"] = adaptq_b200.LayerStack(c["layers"], c["heads"], dim, k_bits=kb, v_bits=c["v_bits"], capacity=n, seed=42,
                                            v_mass=0.0, hybrid_thresh=0)
        if kind == "stack":
            scale = _fill(s["stack"].append, n, lead, dim, dist, gen)
            s["k"], s["v"] = (_values(lead + (dim,), dist, gen, scale) for _ in range(2))
        else:
            s["k"], s["v"] = (_values((n,) + lead + (dim,), dist, gen) for _ in range(2))
        s["q"] = torch.randn(lead + (dim,), device="cuda", generator=gen)
        s["out"] = torch.empty_like(s["q"])
    elif kind in ("batch", "long"):
        heads, n = c["heads"], c["context"]
        kw = {"seed": 42}
        if kind == "batch":  # engines of many layers and sequences behind one handle: seed 42 ^ layer, 8 heads per layer
            kw = {"seeds": [((42 ^ (i // 8 % 32)) ^ (i % 8 * 0xDEADBEEFCAFE)) & SEED_MASK for i in range(heads)]}
        ctx = adaptq_b200.MHAContext(heads, dim, c["k_bits"], c["v_bits"], n, v_mass=0.0, hybrid_thresh=0, **kw)
        _fill(ctx.append_all, n, (heads,), dim, dist, gen)
        s["ctx"] = ctx
        s["k"], s["v"] = (_values((heads, dim), dist, gen) for _ in range(2))
        s["q"] = torch.randn((heads, dim), device="cuda", generator=gen)
        s["out"] = torch.empty_like(s["q"])
    elif kind == "grouped":
        b, h, g = c["batch"], c["heads"], c["q_per_kv"]
        kw = dict(v_mass=0.0, hybrid_thresh=0) if c["dense"] else {}
        m = adaptq_b200.BatchedAdaptQAttention(dim, h, b, c["k_bits"], c["v_bits"], c["context"], 42, q_per_kv=g, **kw)
        step = max(1, 2**26 // (b * h * dim))
        for t in range(0, c["context"], step):
            shape = (b, min(step, c["context"] - t), h, dim)
            m.prefill(_values(shape, dist, gen), _values(shape, dist, gen))
        s["module"] = m
        dt = torch.bfloat16 if c["bf16"] else torch.float32
        s["k"], s["v"] = (_values((b, h, dim), dist, gen).to(dt) for _ in range(2))
        s["q"] = torch.randn((b, h * g, dim), device="cuda", generator=gen).to(dt)
    else:  # prefill
        heads, n = c["heads"], c["tokens"]
        s["engine"] = adaptq_b200.Engine(dim, heads, c["k_bits"], c["v_bits"], n, 42, v_mass=0.0, hybrid_thresh=0)
        s["k"], s["v"] = (_values((n, heads, dim), dist, gen) for _ in range(2))
        s["q"] = torch.randn((heads, dim), device="cuda", generator=gen)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    """One call as a user's loop makes it.  The packed rows live inside the library's handle; what
    they hold comes back through the attention over all of them."""
    kind = s["kind"]
    if kind == "engine":
        return s["engine"].step(s["k"], s["v"], s["q"])
    if kind == "window":
        return s["engine"].compute(s["q"])
    if kind == "stack":
        return s["stack"].step(s["k"], s["v"], s["q"], out=s["out"])
    if kind == "batch":
        return s["ctx"].decode_step(s["k"], s["v"], s["q"], out=s["out"])
    if kind == "long":
        return s["ctx"].compute_all(s["q"], out=s["out"])
    if kind == "grouped":
        return s["module"](s["q"], s["k"], s["v"])
    if kind == "stack_prefill":
        s["stack"].append(s["k"], s["v"])
        return s["stack"].compute(s["q"], out=s["out"])
    s["engine"].append_many(s["k"], s["v"])
    return s["engine"].compute(s["q"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _padded(dim):
    return 1 << (dim - 1).bit_length()


def _row(dim, bits):
    return 4 * _padded(dim) if bits == 16 else _padded(dim) * bits // 8


def work(case):
    """Bytes: the cache rows and scales of every head once (grouped queries share them), each input
    vector once, each output and each packed row written once.  Flops: 2*dim per token and query
    for the scores and again for the values, and the butterflies of each appended vector."""
    c, dim = case, case["dim"]
    kind = c["kind"]
    fwht = _padded(dim) * (_padded(dim).bit_length() - 1)
    layers = c.get("layers", 1)
    inst = c["heads"] * layers * c.get("batch", 1)                   # head instances
    g = c.get("q_per_kv", 1)
    io = 2 if c.get("bf16") else 4
    n = c.get("context", c.get("tokens"))
    row = _row(dim, c["k_bits"]) + _row(dim, c["v_bits"]) + 8        # packed K and V row with their scales
    extra = 0                                                       # FP32 keys of a stack's first layer
    if kind in ("stack", "stack_prefill"):
        extra = c["heads"] * (_row(dim, 16) - _row(dim, c["k_bits"]))
    if kind == "window":
        row = 8 * dim                                               # the FP32 window
    bytes_ = n * (inst * row + extra) + 2 * io * inst * g * dim      # cache read, q read, out written
    flops = 4.0 * n * dim * inst * g
    if kind in ("engine", "stack", "batch", "grouped"):
        bytes_ += inst * (2 * io * dim + row) + extra                # one token in
        flops += 2.0 * inst * fwht
    if kind in ("prefill", "stack_prefill"):
        bytes_ += n * (inst * (8 * dim + row) + extra)               # the prompt in, its rows written
        flops += 2.0 * n * inst * fwht
    return {"bytes": float(bytes_), "flops": flops}


def tolerance(case):
    """Measured between the specialised and the general kernels, which sum in different orders
    (largest over the listed and 24 drawn cases), times about four."""
    if not case.get("dense", True):
        # Sparse V stops at a running mass of weights: the last bits of the weights can move one head's
        # cut by a block of four tokens.  Moving it in a float64 model of one head of 520 tokens changes
        # the output by 2.2e-2, falling with the root of the tokens and of the heads beside it.
        inst = case["heads"] * case.get("batch", 1)
        return {"rel": max(3e-3, 0.025 * math.sqrt(520 / (case["context"] * inst))), "max": 0.1}
    if case.get("bf16"):
        return {"rel": 3e-4, "max": 0.02}  # outputs rounded to bf16: 5.7e-5 and 7.1e-3 (one bf16 step) measured
    if case["dist"] in ("student3", "student4", "outlier"):
        return {"rel": 4e-6, "max": 2e-4}  # 8.3e-7 and 3.7e-5 measured: some logits are in the hundreds
    return {"rel": 4e-6, "max": 4e-5}      # 8.5e-7 and 3.8e-6 measured
