"""The work a user of this library has it do, as measurable cases.

Seven families, each through the public Python API: training steps over dense and packed batches (forward and
backward), dense and packed forward passes without gradients, prefill chunks against a paged KV cache, decode steps
against dense and paged KV caches (one or several new tokens), and decode steps against an int8 latent cache.
`listed` names a case or two of each, `draw` makes more of the same ranges.  A case is a dict of plain values; ragged
lengths come from the case's own `lens_seed`, so that the work of a case does not depend on the seed of its inputs.
"""
import math
import os
import random
import sys

import torch

# the process runs in the root of the tree it measures
_PKG = os.path.join(os.getcwd(), "flash-attention-npu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import flash_attn_npu as fa2  # noqa: E402
import flash_attn_npu_3 as fa3  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # One attention layer of a long-context training step: the benchmark's forward + backward workload.
        {"name": "train_dense_4k", "family": "train_dense", "dtype": "bf16", "b": 4, "sq": 4096, "sk": 4096, "hq": 32,
         "hkv": 32, "d": 128, "causal": True, "left": -1, "softcap": 0.0, "api": 2},
        # A training step of a small model: the whole call is a few tens of microseconds of kernels, so launches and host
        # work show.  Shape of the reference's own backward tests.
        {"name": "train_dense_small", "family": "train_dense", "dtype": "fp16", "b": 5, "sq": 1024, "sk": 1024, "hq": 4,
         "hkv": 4, "d": 128, "causal": True, "left": -1, "softcap": 0.0, "api": 2},
        # A training step at head dim 256 under a query group, as models with few wide heads have it.
        {"name": "train_dense_d256", "family": "train_dense", "dtype": "bf16", "b": 2, "sq": 2048, "sk": 2048, "hq": 8,
         "hkv": 4, "d": 256, "causal": True, "left": -1, "softcap": 0.0, "api": 2},
        # Fine-tuning on packed documents of mixed lengths, grouped-query attention, through the second API version.
        {"name": "train_packed", "family": "train_packed", "dtype": "bf16", "b": 12, "lo": 128, "hi": 4096, "lens_seed": 7,
         "hq": 16, "hkv": 4, "d": 128, "causal": True, "left": -1, "api": 3},
        # A bidirectional encoder over an odd number of tokens, head dim 64, inference only.
        {"name": "encode_d64", "family": "forward_dense", "dtype": "fp16", "b": 16, "sq": 1025, "sk": 1025, "hq": 16,
         "hkv": 16, "d": 64, "causal": False, "left": -1, "softcap": 0.0, "api": 2},
        # A layer with a sliding window and capped scores (the softcap of the reference's tests), long context.
        {"name": "forward_window_softcap", "family": "forward_dense", "dtype": "bf16", "b": 1, "sq": 8192, "sk": 8192,
         "hq": 16, "hkv": 8, "d": 128, "causal": True, "left": 1024, "softcap": 30.0, "api": 2},
        # Prefill of a batch of prompts of mixed lengths, packed: the benchmark's packed forward workload.
        {"name": "prefill_packed", "family": "forward_packed", "dtype": "bf16", "b": 16, "lo": 256, "hi": 8192,
         "lens_seed": 1234, "hq": 32, "hkv": 8, "d": 128, "causal": True, "left": -1, "api": 2},
        # Chunked prefill in a serving loop: 512 new tokens a sequence, appended with rotary to paged caches of mixed
        # lengths.
        {"name": "prefill_chunk", "family": "cache", "dtype": "bf16", "b": 4, "sq": 512, "lo": 1000, "hi": 16000,
         "lens_seed": 3, "hq": 32, "hkv": 8, "d": 128, "page": 256, "append": True, "rotary": True, "api": 2},
        # The smallest call: one token a sequence for a handful of short sequences with a dense cache, append + rotary.
        {"name": "decode_small", "family": "cache", "dtype": "bf16", "b": 4, "sq": 1, "lo": 300, "hi": 2000,
         "lens_seed": 5, "hq": 32, "hkv": 8, "d": 128, "page": 0, "append": True, "rotary": True, "api": 2},
        # Large-batch serving decode against paged caches of mixed lengths: the benchmark's paged-decode workload.
        {"name": "decode_paged", "family": "cache", "dtype": "bf16", "b": 128, "sq": 1, "lo": 1024, "hi": 32768,
         "lens_seed": 1234, "hq": 32, "hkv": 8, "d": 128, "page": 256, "append": True, "rotary": True, "api": 2},
        # Speculative decoding: four new tokens a step, already appended, under a query group of 8.
        {"name": "decode_multi", "family": "cache", "dtype": "bf16", "b": 16, "sq": 4, "lo": 1024, "hi": 32768,
         "lens_seed": 11, "hq": 64, "hkv": 8, "d": 128, "page": 256, "append": False, "rotary": False, "api": 3},
        # Latent (MLA) decode against an int8 cache: the benchmark's latent-decode workload.
        {"name": "decode_latent", "family": "latent", "b": 64, "lo": 4096, "hi": 131072, "lens_seed": 1234, "hq": 128,
         "page": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _heads(rng, most=32):
    hkv = rng.choice([1, 2, 4, 8, 8, 16])
    g = rng.choice([1, 1, 2, 4, 4, 8])
    while hkv * g > most:
        g = max(1, g // 2)
        hkv = hkv if hkv * g <= most else hkv // 2
    return hkv * g, hkv


def _draw_one(rng):
    family = rng.choice(["train_dense", "train_dense", "train_packed", "forward_dense", "forward_packed", "cache", "cache",
                         "cache", "cache", "latent"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    d = rng.choice([64, 128, 128, 128])
    api = rng.choice([2, 2, 3])
    if family == "train_dense":
        d = rng.choice([64, 96, 128, 128, 128, 256])
        hq, hkv = _heads(rng)
        s = _log(rng, 200, 8192)
        return {"family": family, "dtype": dtype, "b": _log(rng, 1, 8), "sq": s, "sk": s, "hq": hq, "hkv": hkv, "d": d,
                "causal": rng.random() < 0.75, "left": _log(rng, 128, 2048) if rng.random() < 0.15 else -1,
                "softcap": 0.0, "api": api}
    if family == "train_packed":
        d = rng.choice([64, 96, 128, 128, 128])
        hq, hkv = _heads(rng)
        return {"family": family, "dtype": dtype, "b": _log(rng, 2, 24), "lo": 64, "hi": _log(rng, 256, 6000),
                "lens_seed": rng.randrange(1 << 20), "hq": hq, "hkv": hkv, "d": d, "causal": True, "left": -1, "api": api}
    if family == "forward_dense":
        d = rng.choice([64, 96, 128, 128, 192, 256])
        hq, hkv = _heads(rng)
        s = _log(rng, 200, 12000)
        causal = rng.random() < 0.6
        return {"family": family, "dtype": dtype, "b": _log(rng, 1, 16), "sq": s, "sk": s, "hq": hq, "hkv": hkv, "d": d,
                "causal": causal, "left": _log(rng, 256, 4096) if causal and rng.random() < 0.3 else -1,
                "softcap": 30.0 if rng.random() < 0.2 else 0.0, "api": api}
    if family == "forward_packed":
        d = rng.choice([64, 128, 128, 128, 256])
        hq, hkv = _heads(rng)
        return {"family": family, "dtype": dtype, "b": _log(rng, 2, 32), "lo": 32, "hi": _log(rng, 256, 8192),
                "lens_seed": rng.randrange(1 << 20), "hq": hq, "hkv": hkv, "d": d, "causal": True,
                "left": -1, "api": api}
    if family == "cache":
        hq, hkv = _heads(rng, 64)
        sq = rng.choice([1, 1, 1, 1, _log(rng, 2, 8), _log(rng, 64, 2048)])
        append = rng.random() < 0.7
        hi = _log(rng, 300, 32768)
        return {"family": family, "dtype": dtype, "b": _log(rng, 1, 128) if sq < 64 else _log(rng, 1, 8), "sq": sq,
                "lo": max(16, hi // rng.choice([2, 8, 32])), "hi": hi, "lens_seed": rng.randrange(1 << 20), "hq": hq,
                "hkv": hkv, "d": rng.choice([64, 128, 128, 128, 256]), "page": rng.choice([0, 64, 128, 256, 256]),
                "append": append, "rotary": append and rng.random() < 0.7, "api": api}
    hi = _log(rng, 512, 131072)
    return {"family": "latent", "b": _log(rng, 1, 64), "lo": max(64, hi // rng.choice([2, 8, 32])), "hi": hi,
            "lens_seed": rng.randrange(1 << 20), "hq": rng.choice([128, 128, 64, 16]), "page": rng.choice([64, 128, 256])}


def draw(rng):
    while True:
        c = _draw_one(rng)
        w = work(c)
        most = 1.6e12 if c.get("d", 0) <= 128 or not c["family"].startswith("train") else 2.0e11
        if w["flops"] <= most and w["bytes"] <= 8e9:
            return c


# ---------------------------------------------------------------------------------------------------------------
def _lens(case):
    r = random.Random(case["lens_seed"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["b"])]


def _visible(sq, sk, causal, left):
    """Visible (query, key) pairs of one sequence under bottom-right aligned causal / left-window masks."""
    i = torch.arange(sq, dtype=torch.int64) + (sk - sq)
    hi = torch.clamp(i, max=sk - 1) if causal else torch.full((sq,), sk - 1, dtype=torch.int64)
    lo = torch.clamp(i - left, min=0) if left >= 0 else torch.zeros(sq, dtype=torch.int64)
    return int(torch.clamp(hi - lo + 1, min=0).sum())


def work(case):
    f = case["family"]
    if f == "latent":
        tokens = sum(_lens(case))
        hq = case["hq"]
        return {"bytes": tokens * (512 + 4 + 128) + case["b"] * hq * (576 + 512) * 2, "flops": 2.0 * (576 + 512) * hq * tokens}
    hq, hkv, d = case["hq"], case["hkv"], case["d"]
    if f == "cache":
        new = case["sq"] if case["append"] else 0
        lens = _lens(case)
        pairs = sum(_visible(case["sq"], n + new, True, -1) for n in lens)
        rows = case["b"] * case["sq"]
        # keys and values in the cache, the new rows (read and appended), q and out
        nbytes = sum(lens) * hkv * d * 4 + case["b"] * new * hkv * d * 8 + rows * hq * d * 4
        return {"bytes": nbytes, "flops": 4.0 * hq * d * pairs}
    if f.endswith("packed"):
        lens = _lens(case)
        pairs = sum(_visible(n, n, case["causal"], case["left"]) for n in lens)
        tq = tk = sum(lens)
    else:
        pairs = case["b"] * _visible(case["sq"], case["sk"], case["causal"], case["left"])
        tq, tk = case["b"] * case["sq"], case["b"] * case["sk"]
    flops = 4.0 * hq * d * pairs
    nbytes = 2 * d * (2 * tq * hq + 2 * tk * hkv)                       # q, out; k, v
    if f.startswith("train"):
        flops *= 3.5
        nbytes += 2 * d * (2 * tq * hq + 2 * tk * hkv)                  # dout, dq; dk, dv
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Outputs are rounded to the input type once, P (and dS in the backward) once before the second product; two correct
    kernels differ by where those roundings fall and by the order of the sums.  Four times what the default kernels and
    the general ones (64-key tiles, no stored exponent base) differ by on these cases and 24 drawn ones: at most 3.0e-3
    / 4.0e-2 (2-norm / single value) in bf16, 3.8e-4 / 3.4e-3 in fp16; latent decode with another split of the keys
    1.5e-3 / 1.0e-2."""
    if case["family"] == "latent":
        return {"rel": 6e-3, "max": 4e-2}
    return {"rel": 1.2e-2, "max": 0.16} if case["dtype"] == "bf16" else {"rel": 1.5e-3, "max": 1.5e-2}


# ---------------------------------------------------------------------------------------------------------------
def _randn(gen, dtype, *shape):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)


def _pages(case, lens, extra, gen):
    """A page table over a pool in random order, as a serving loop that has been running for a while has it."""
    page = case["page"]
    need = [(n + extra + page - 1) // page for n in lens]
    pool = sum(need)
    order = torch.randperm(pool, generator=gen, device="cuda").to(torch.int32)
    table = torch.zeros(len(lens), max(need), dtype=torch.int32, device="cuda")
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
    return pool, table


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f = case["family"]
    s = {"case": case, "family": f}
    if f == "latent":
        lens = _lens(case)
        pool, s["table"] = _pages(case, lens, 0, gen)
        page = case["page"]
        s["latent"] = torch.randint(-127, 128, (pool, page, 512), generator=gen, device="cuda", dtype=torch.int8)
        s["scales"] = torch.rand(pool, page, generator=gen, device="cuda") * 0.02 + 0.001
        s["rope"] = _randn(gen, torch.bfloat16, pool, page, 64)
        s["q_nope"] = _randn(gen, torch.bfloat16, case["b"], 1, case["hq"], 512)
        s["q_rope"] = _randn(gen, torch.bfloat16, case["b"], 1, case["hq"], 64)
        s["lens"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
        return s
    dt, hq, hkv, d = _DTYPES[case["dtype"]], case["hq"], case["hkv"], case["d"]
    s["fa"] = fa2 if case["api"] == 2 else fa3
    if f == "cache":
        lens, b, sq = _lens(case), case["b"], case["sq"]
        new = sq if case["append"] else 0
        if case["page"]:
            pool, s["table"] = _pages(case, lens, new, gen)
            shape = (pool, case["page"], hkv, d)
        else:
            s["table"] = None
            shape = (b, (case["hi"] + new + 127) // 128 * 128, hkv, d)
        s["k_cache"], s["v_cache"] = _randn(gen, dt, *shape), _randn(gen, dt, *shape)
        s["q"] = _randn(gen, dt, b, sq, hq, d)
        s["k"] = s["v"] = s["cos"] = s["sin"] = None
        if new:
            s["k"], s["v"] = _randn(gen, dt, b, sq, hkv, d), _randn(gen, dt, b, sq, hkv, d)
        if case["rotary"]:
            pos = torch.arange(case["hi"] + new + 1, device="cuda", dtype=torch.float32)
            freq = 10000.0 ** (-torch.arange(0, d, 2, device="cuda", dtype=torch.float32) / d)
            ang = pos[:, None] * freq[None, :]
            s["cos"], s["sin"] = ang.cos().to(dt), ang.sin().to(dt)
        # without an append the new tokens are in the cache already
        s["lens"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
        return s
    grad = f.startswith("train")
    if f.endswith("packed"):
        lens = _lens(case)
        total = sum(lens)
        s["max_len"] = max(lens)
        s["cu"] = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
        qs, ks = (total, hq, d), (total, hkv, d)
    else:
        qs, ks = (case["b"], case["sq"], hq, d), (case["b"], case["sk"], hkv, d)
    s["q"], s["k"], s["v"] = _randn(gen, dt, *qs), _randn(gen, dt, *ks), _randn(gen, dt, *ks)
    if grad:
        s["dout"] = _randn(gen, dt, *qs)
        for n in ("q", "k", "v"):
            s[n].requires_grad_(True)
    return s


def run(s):
    case, f = s["case"], s["family"]
    if f == "latent":
        return fa3.flash_attn_mla_with_kvcache(s["q_nope"], s["q_rope"], s["latent"], s["scales"], s["rope"], s["lens"],
                                               s["table"])
    fa = s["fa"]
    if f == "cache":
        table = {"block_table": s["table"]} if case["api"] == 2 else {"page_table": s["table"]}
        out = fa.flash_attn_with_kvcache(s["q"], s["k_cache"], s["v_cache"], s["k"], s["v"], rotary_cos=s["cos"],
                                         rotary_sin=s["sin"], cache_seqlens=s["lens"], causal=True,
                                         rotary_interleaved=False, **table)
        return (out, s["k_cache"], s["v_cache"]) if s["k"] is not None else out
    window = (case["left"], 0 if case["left"] >= 0 else -1)
    if f.endswith("packed"):
        out = fa.flash_attn_varlen_func(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["max_len"], s["max_len"],
                                        causal=case["causal"], window_size=window)
    else:
        out = fa.flash_attn_func(s["q"], s["k"], s["v"], causal=case["causal"], window_size=window,
                                 softcap=case["softcap"])
    if f.startswith("train"):
        return (out,) + torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])
    return out
