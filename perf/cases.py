"""Performance cases of the engine: the calls a user's program makes, over the sizes it makes them with.

`listed()` holds the named cases, `draw(rng)` gives more of the same ranges.  A case is a dict of plain
values; `prepare` makes what a program has in hand before the call, `run` is one pass through the public
entry points, `work` and `tolerance` say what the pass cannot do without and how closely two correct
implementations agree.  All cases run on one GPU (a ring of one).

Keys of a case
  entry     "self": `ring_self_attention` (built-in masks); "general": `ring_attention` with a `ScoreMod`,
            a `bias_fn` callable or no bias
  dtype     "bf16" or "f32"
  b, h, lq, lk, d   batch, heads, query rows, key rows, head dim
  mask      "none" | "causal" | "documents" (causal inside packed documents) | "prefix" (prefix-LM) |
            "alibi+window" (ALiBi and a causal window) | "bias_fn" (a relative-position bias that a
            callable materialises)
  backward  whether the pass is forward + backward (training) or forward only
  pack      seed of the document packing (0 where there are none); the packing belongs to the case, so
            that its visible pairs can be counted
"""
import math

import numpy as np
import torch

import ring_attention_b200 as ra

AXIS = ra.PartitionSpec(None, "sp")
BIAS_RANGE = 128  # the callable's relative positions are clipped to [-BIAS_RANGE, BIAS_RANGE]


def _case(name, **kw):
    c = dict(name=name, entry="self", dtype="bf16", b=1, h=16, lq=1024, lk=1024, d=128, mask="causal", backward=True,
             pack=0, doc_min=0, doc_max=0, window=0)
    c.update(kw)
    return c


def listed():
    return [
        # fp32 training step at the size of the reference's CPU-runnable configuration: latency and launches
        _case("f32_causal_1k", dtype="f32", h=4, lq=1024, lk=1024, d=64),
        # fp32 at the largest size of the test-suite (2048 x 2048, batch 2, 4 heads, no mask), forward + backward:
        # numerics work, gradient checks, small fp32 models
        _case("f32_full_2k", entry="general", dtype="f32", b=2, h=4, lq=2048, lk=2048, d=64, mask="none"),
        # a short-sequence bf16 training step: launch and host latency
        _case("causal_1k", h=16, lq=1024, lk=1024),
        # a training batch whose length is not a multiple of anything (no padding on the user's side)
        _case("causal_ragged_3001", b=2, h=16, lq=3001, lk=3001),
        # the usual pre-training sequence length
        _case("causal_8k", b=2, h=16, lq=8192, lk=8192),
        # the headline configuration: bf16 causal, batch 2, 16 heads, head dim 128, 32768 tokens
        _case("causal_32k", b=2, h=16, lq=32768, lk=32768),
        # long-context training over packed documents of 512 to 16384 tokens
        _case("documents_128k", h=32, lq=131072, lk=131072, mask="documents", doc_min=512, doc_max=16384),
        # long-context prefill with ALiBi and a 4096-token window, head dim 64
        _case("alibi_window_64k", entry="general", b=4, h=16, lq=65536, lk=65536, d=64, mask="alibi+window", window=4096,
              backward=False),
        # head-dim-64 training
        _case("causal_4k_d64", b=4, h=16, lq=4096, lk=4096, d=64),
        # prefix-LM training: the first part of every sequence sees itself in both directions
        _case("prefix_4k", b=2, h=16, lq=4096, lk=4096, mask="prefix"),
        # encoder-decoder cross attention: few queries over a longer, ragged memory
        _case("cross_448_1500", entry="general", b=8, h=16, lq=448, lk=1500, d=64, mask="none"),
        # a user's own bias function (learned relative-position bias), head dim 64
        _case("bias_fn_2k", entry="general", b=2, h=8, lq=2048, lk=2048, d=64, mask="bias_fn"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the same masks, types and directions at sizes spread over 128 to 16384 tokens, half of the
    lengths as they fall (odd ones among them), half rounded to a multiple of 128."""
    while True:
        kind = rng.choice(["causal", "causal", "causal", "documents", "prefix", "alibi+window", "none", "cross", "bias_fn", "f32"])
        d = rng.choice([64, 128])
        c = _case(None, d=d, b=rng.choice([1, 1, 2, 3, 4]), h=rng.choice([4, 8, 12, 16, 32]))
        del c["name"]
        hi = {"bias_fn": 3072, "f32": 2048, "cross": 4096, "documents": 16384}.get(kind, 12288)
        n = _log_int(rng, 128, hi)
        if rng.random() < 0.5:
            n = max(128, (n + 64) // 128 * 128)
        c["lq"] = c["lk"] = n
        c["mask"] = kind
        c["backward"] = rng.random() < 0.75
        if kind == "documents":
            c.update(doc_min=max(16, n // 64), doc_max=max(32, n // 3), pack=rng.randrange(1000))
        elif kind == "alibi+window":
            c.update(entry="general", window=_log_int(rng, 64, 4096))
        elif kind == "none":
            c.update(entry="general")
        elif kind == "cross":
            c.update(entry="general", mask="none", lq=max(1, n // rng.choice([2, 3, 5, 16])))
        elif kind == "bias_fn":
            c.update(entry="general", b=rng.choice([1, 2]), h=rng.choice([4, 8]))
        elif kind == "f32":
            c.update(dtype="f32", mask=rng.choice(["causal", "none", "prefix"]), b=rng.choice([1, 2]), h=rng.choice([2, 4, 8]))
            c["entry"] = "general" if c["mask"] == "none" else "self"
        limit = 0.05e12 if c["dtype"] == "f32" else 4e12
        if work(c)["flops"] <= limit:
            return c


def _doc_lengths(c):
    """Packed documents: lengths uniform in [doc_min, doc_max] until the sequence is full, the last one cut."""
    g = np.random.default_rng(c["pack"])
    out, left = [], c["lq"]
    while left > 0:
        n = min(int(g.integers(c["doc_min"], c["doc_max"] + 1)), left)
        out.append(n)
        left -= n
    return out


def _prefix_len(c):
    return c["lq"] // 4


def _causal_pairs(n):
    return n * (n + 1) // 2


def _pairs(c):
    """Visible (query, key) pairs of one batch element and head."""
    n = c["lq"]
    if c["mask"] == "causal":
        return _causal_pairs(n)
    if c["mask"] == "documents":
        return sum(_causal_pairs(x) for x in _doc_lengths(c))
    if c["mask"] == "prefix":
        p = _prefix_len(c)
        return _causal_pairs(n) + p * (p - 1) // 2
    if c["mask"] == "alibi+window":
        w = min(c["window"], n)
        return _causal_pairs(w) + (n - w) * w
    return n * c["lk"]


def work(c):
    es = 2 if c["dtype"] == "bf16" else 4
    q_b, kv_b = c["b"] * c["lq"] * c["h"] * c["d"] * es, c["b"] * c["lk"] * c["h"] * c["d"] * es
    nbytes = 2 * q_b + 2 * kv_b  # q, k, v in; out
    per_pair = 4 * c["d"]
    if c["backward"]:
        nbytes += 2 * q_b + 2 * kv_b  # dout in; dq, dk, dv out
        per_pair += 10 * c["d"]
    if c["mask"] == "bias_fn":
        nbytes += (2 * BIAS_RANGE + 1) * c["h"] * 4
    if c["mask"] not in ("none",):
        nbytes += c["b"] * (c["lq"] + c["lk"]) * 4
    return {"bytes": nbytes, "flops": c["b"] * c["h"] * _pairs(c) * per_pair}


def tolerance(c):
    # Four times what the path shows against the same attention in 64 bits on the same inputs, over these ranges:
    # f32 rel 9.5e-7, max 1.2e-5 (sums of up to 2048 fp32 atomics); bf16 rel 2.7e-3 (bf16 results, P and dS
    # rounded to bf16 before their products), max 0.13 (gradients of the first, peaked causal rows).
    if c["dtype"] == "f32":
        return {"rel": 4e-6, "max": 5e-5}
    return {"rel": 1e-2, "max": 0.5}


def prepare(c, seed):
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(seed)
    dt = torch.bfloat16 if c["dtype"] == "bf16" else torch.float32
    b, h, lq, lk, d = c["b"], c["h"], c["lq"], c["lk"], c["d"]

    def tensor(n):
        t = torch.empty((b, n, h, d), dtype=dt, device=dev)
        for i in range(b):  # one batch element at a time: the fp32 draw stays small
            t[i] = torch.randn((n, h, d), generator=g, device=dev).to(dt)
        return t

    s = dict(case=c, q=tensor(lq), k=tensor(lk), v=tensor(lk), dout=tensor(lq) if c["backward"] else None)
    if c["backward"]:
        for name in "qkv":
            s[name].requires_grad_(True)
    s["pos"] = torch.arange(lq, dtype=torch.int32, device=dev).expand(b, lq).contiguous()
    s["kpos"] = torch.arange(lk, dtype=torch.int32, device=dev).expand(b, lk).contiguous()
    if c["mask"] == "documents":
        ids = np.repeat(np.arange(len(_doc_lengths(c)), dtype=np.int32), _doc_lengths(c))
        s["seg"] = torch.from_numpy(ids).to(dev).expand(b, lq).contiguous()
    if c["mask"] == "prefix":
        s["prefix"] = (s["pos"] < _prefix_len(c)).contiguous()
    if c["mask"] == "alibi+window":
        slopes = 2.0 ** (-8.0 * torch.arange(1, h + 1, dtype=torch.float32, device=dev) / h)
        s["mod"] = ra.ScoreMod(causal=True, alibi_slopes=slopes, window=c["window"])
    if c["mask"] == "bias_fn":
        table = torch.randn((h, 2 * BIAS_RANGE + 1), generator=g, device=dev) * 0.5

        def bias_fn(q_positions, kv_positions):
            rel = (q_positions[0, :, None] - kv_positions[0, None, :]).clamp(-BIAS_RANGE, BIAS_RANGE) + BIAS_RANGE
            return table[:, rel.long()][None].expand(b, h, lq, lk)

        s["bias_fn"] = bias_fn
    return s


def _forward(s):
    c = s["case"]
    if c["entry"] == "self":
        return ra.ring_self_attention(s["q"], s["k"], s["v"], None, AXIS, causal=c["mask"] in ("causal", "documents"),
                                      segment_ids=s.get("seg"), positions=s["pos"], prefix_mask=s.get("prefix"))
    fn = s.get("bias_fn") or s.get("mod")
    kw = {}
    if fn is not None:
        kw = dict(bias_fn=fn, bias_q_kwargs={"q_positions": s["pos"]}, bias_kv_kwargs={"kv_positions": s["kpos"]})
    return ra.ring_attention(s["q"], s["k"], s["v"], "sp", **kw)


def run(s):
    if not s["case"]["backward"]:
        with torch.no_grad():
            return _forward(s)
    out = _forward(s)
    dq, dk, dv = torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])
    return out, dq, dk, dv
