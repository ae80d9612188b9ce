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

import numpy as np
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


def _draw_inputs(case, seed, append):
    """Everything a case is given, in one order: the tokens already in the cache go to `append`
    as (tokens, ..., dim) chunks; the token, prompt and queries of the pass come back."""
    c, kind, dist, dim = case, case["kind"], case["dist"], case["dim"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed) & (2**63 - 1))
    lead = {"stack": (c.get("layers"), c["heads"]), "stack_prefill": (c.get("layers"), c["heads"]),
            "grouped": (c.get("batch"), c["heads"])}.get(kind, (c["heads"],))
    if kind in ("prefill", "stack_prefill"):
        k, v = (_values((c["tokens"],) + lead + (dim,), dist, gen) for _ in range(2))
    else:
        scale = _fill(append, c["context"], lead, dim, dist, gen)
        k, v = (_values(lead + (dim,), dist, gen, scale) for _ in range(2))
    if kind in ("engine", "window"):
        return k, v, _values(lead + (dim,), dist, gen)
    q = torch.randn(lead[:-1] + (lead[-1] * c.get("q_per_kv", 1), dim), device="cuda", generator=gen)
    if c.get("bf16"):
        k, v, q = (t.to(torch.bfloat16) for t in (k, v, q))
    return k, v, q


def _batch_seeds(heads):
    """Engines of many layers and sequences behind one handle: seed 42 ^ layer, 8 heads per layer."""
    return [((42 ^ (i // 8 % 32)) ^ (i % 8 * 0xDEADBEEFCAFE)) & SEED_MASK for i in range(heads)]


def _k_bits(case):
    """Key bits per layer: a stack's layer 0 keeps FP32 keys."""
    return [16] + [case["k_bits"]] * (case["layers"] - 1)


def prepare(case, seed):
    c, kind, dim = dict(case), case["kind"], case["dim"]
    s = {"kind": kind}
    if kind in ("engine", "window", "prefill"):
        kw = dict(v_mass=0.0, hybrid_thresh=0) if c.get("dense", kind == "prefill") else {}
        cap = {"engine": c.get("context"), "window": 4096, "prefill": c.get("tokens")}[kind]
        s["engine"] = adaptq_b200.Engine(dim, c["heads"], c["k_bits"], c["v_bits"], cap, 42, **kw)
        append = s["engine"].append_many
    elif kind in ("stack", "stack_prefill"):
        s["stack"] = adaptq_b200.LayerStack(c["layers"], c["heads"], dim, k_bits=_k_bits(c), v_bits=c["v_bits"],
                                            capacity=c["context"] if kind == "stack" else c["tokens"], seed=42, v_mass=0.0,
                                            hybrid_thresh=0)
        append = s["stack"].append
    elif kind in ("batch", "long"):
        kw = {"seeds": _batch_seeds(c["heads"])} if kind == "batch" else {"seed": 42}
        s["ctx"] = adaptq_b200.MHAContext(c["heads"], dim, c["k_bits"], c["v_bits"], c["context"], v_mass=0.0, hybrid_thresh=0, **kw)
        append = s["ctx"].append_all
    else:  # grouped
        kw = dict(v_mass=0.0, hybrid_thresh=0) if c["dense"] else {}
        m = s["module"] = adaptq_b200.BatchedAdaptQAttention(dim, c["heads"], c["batch"], c["k_bits"], c["v_bits"], c["context"], 42,
                                                             q_per_kv=c["q_per_kv"], **kw)
        append = lambda k, v: m.prefill(k.transpose(0, 1), v.transpose(0, 1))  # noqa: E731
    s["k"], s["v"], s["q"] = _draw_inputs(c, seed, append)
    s["out"] = torch.empty_like(s["q"])
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


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
# Lloyd-Max centroids of N(0, 1) for 2, 3 and 4 bits (upper halves; the codebooks are odd)
_CENTROIDS = {2: [0.4528, 1.5104], 3: [0.2451, 0.7560, 1.3439, 2.1529],
              4: [0.1258, 0.3795, 0.6402, 0.9138, 1.2016, 1.5105, 1.8944, 2.4008]}


def _signs(seeds, padded):
    """Rademacher signs of each seed: one xorshift64 step per coordinate, +1 where the low bit is set."""
    s = np.array([x if x else 0xDEADBEEFCAFE1234 for x in seeds], dtype=np.uint64)
    out = np.empty((len(seeds), padded), dtype=np.float32)
    for j in range(padded):
        s ^= s << np.uint64(13)
        s ^= s >> np.uint64(7)
        s ^= s << np.uint64(17)
        out[:, j] = np.where(s & np.uint64(1), 1.0, -1.0)
    return torch.from_numpy(out).cuda()


def _hadamard(x):
    """Unnormalised Walsh-Hadamard butterflies over the last axis, stage by stage."""
    shape, p, h = x.shape, x.shape[-1], 1
    while h < p:
        y = x.reshape(-1, p // (2 * h), 2, h)
        x = torch.stack((y[:, :, 0] + y[:, :, 1], y[:, :, 0] - y[:, :, 1]), 2).reshape(shape)
        h *= 2
    return x


def _pad(x, padded):
    return torch.nn.functional.pad(x, (0, padded - x.shape[-1]))


def _quantise(x, signs, bits):
    """Rows as the cache holds them: levels and scale.  What is stored is defined in 32-bit steps
    (norm summed in order, scale, signs, butterflies, two scalings, thresholds), so this part is 32 bits."""
    total = torch.zeros_like(x[..., 0])
    for j in range(x.shape[-1]):
        total = total + x[..., j] * x[..., j]
    norm = torch.sqrt(total + 1e-12)
    padded = signs.shape[-1]
    root = np.sqrt(np.float32(padded))
    y = _hadamard(_pad(x * (torch.ones_like(norm) / norm)[..., None], padded) * signs)
    y = (y * float(np.float32(1) / root)) * float(root)
    half = np.array(_CENTROIDS[bits], dtype=np.float32)
    cb = np.concatenate((-half[::-1], half))
    thr = torch.from_numpy((cb[:-1] + cb[1:]) * np.float32(0.5)).cuda()
    return torch.bucketize(y, thr, right=True).to(torch.uint8), norm, torch.from_numpy(cb.astype(np.float64)).cuda()


def _attend(q, keys, v_levels, v_scale, v_cb, signs, dim):
    """softmax(q . keys / sqrt(dim)) over (head, token) rows, values decoded; all in 64 bits.
    q (heads, g, p); keys (heads, tokens, p)."""
    p = signs.shape[-1]
    w = torch.softmax(q @ keys.transpose(1, 2) / math.sqrt(dim), dim=-1)
    acc = (w * v_scale.double()[:, None]) @ v_cb[v_levels.long()]
    return (_hadamard(acc) / p * signs[:, None].double())[..., :dim]


def exact(case, seed):
    """Attention over the stored rows in 64 bits; the rows themselves are what 32-bit quantisation
    defines.  None for sparse V (where its running 32-bit sum stops decides what is summed) and for the largest cache."""
    c, kind, dim = case, case["kind"], case["dim"]
    n = c.get("context", c.get("tokens"))
    layers, g = c.get("layers", 1), c.get("q_per_kv", 1)
    inst = c["heads"] * layers * c.get("batch", 1)
    if not c.get("dense", True) or inst * n * dim > 2**31:
        return None
    parts = []
    k, v, q = _draw_inputs(c, seed, lambda kk, vv: parts.append((kk.reshape(-1, inst, dim), vv.reshape(-1, inst, dim))))
    if kind in ("prefill", "stack_prefill"):
        parts = [(k.reshape(-1, inst, dim), v.reshape(-1, inst, dim))]
    q = q.reshape(inst, g, dim).double()
    if kind == "window":  # up to 512 tokens are attended to as they came
        ks, vs = (torch.cat([x[i] for x in parts]).double().transpose(0, 1) for i in range(2))
        w = torch.softmax(q @ ks.transpose(1, 2) / math.sqrt(dim), dim=-1)
        return (w @ vs).reshape(c["heads"], dim)
    if kind in ("engine", "stack", "batch", "grouped"):  # the ring is full: the new token takes the oldest one's place
        parts[0] = tuple(x[1:] for x in parts[0])
        parts.append((k.float().reshape(1, inst, dim), v.float().reshape(1, inst, dim)))
    heads = c["heads"]
    seeds = _batch_seeds(heads) if kind == "batch" else [
        ((42 ^ l) ^ (i * 0xDEADBEEFCAFE)) & SEED_MASK for l in range(layers) for i in range(heads)] * c.get("batch", 1)
    padded = _padded(dim)
    signs = _signs(seeds, padded)
    bits = [b for b in (_k_bits(c) if kind in ("stack", "stack_prefill") else [c["k_bits"]]) for _ in range(heads)]
    out = torch.empty((inst, g, dim), dtype=torch.float64, device="cuda")
    step = max(1, 2**24 // (n * padded))
    for a in range(0, inst, step):
        b = min(inst, a + step)
        ks, vs = (torch.cat([x[i][:, a:b] for x in parts]).transpose(0, 1) for i in range(2))
        sg = signs[a:b]
        vl, vsc, vcb = _quantise(vs, sg[:, None], c["v_bits"])
        kb = [bits[i] if len(bits) > heads else bits[0] for i in range(a, b)]
        for fp32 in (True, False):
            rows = [i for i, x in enumerate(kb) if (x == 16) == fp32]
            if not rows:
                continue
            r = torch.tensor(rows, device="cuda")
            qq = q[a:b][r]
            if fp32:
                keys = ks[r].double()
            else:
                kl, ksc, kcb = _quantise(ks[r], sg[r][:, None], c["k_bits"])
                keys = kcb[kl.long()] * (ksc.double() / padded)[..., None]
                qq = _hadamard(_pad(qq, padded) * sg[r][:, None].double())
            out[a:b][r] = _attend(qq, keys, vl[r], vsc[r], vcb, sg[r], dim)
    shape = {"stack": (layers, heads, dim), "stack_prefill": (layers, heads, dim),
             "grouped": (c.get("batch"), heads * g, dim)}.get(kind, (heads, dim))
    return out.reshape(shape)
