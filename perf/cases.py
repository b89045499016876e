"""The attention calls whose speed matters, as cases that a timing program can draw, prepare and run.

A case is a dict of plain values.  ``kind`` says which public call it makes:

  prefill  flash_attn_func, forward only
  train    flash_attn_func, forward and backward through autograd
  packed   flash_attn_varlen_func on packed sequences, forward and backward through autograd
  chunk    flash_attn_with_kvcache on several query rows per sequence against a paged cache that already holds
           their keys, queries packed (the FA3-style front end)
  decode   flash_attn_with_kvcache on one or a few query rows per sequence, contiguous or paged cache

The library's package folder is taken from the working folder, so the same cases can be run on another tree.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("flash-attention-npu_b200"))

import flash_attn_npu_v2 as fa2  # noqa: E402
import flash_attn_npu_v3 as fa3  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(kind, b, sq, sk, h, hk, d, dtype="bf16", **more):
    """sq / sk: query rows and keys of the longest sequence; sk_lo (sq_lo): of the shortest one, lengths in between are
    spread evenly.  causal masks are aligned to the last key.  window: keys visible to the left, -1 for all."""
    c = dict(kind=kind, api="v2", b=b, sq=sq, sq_lo=sq, sk=sk, sk_lo=sk, h=h, hk=hk, d=d, dtype=dtype, causal=True, window=-1,
             softcap=0.0, page=0, append=False, rotary=False, plan=False)
    c.update(more)
    return c


def listed():
    return [
        # a unit-test-sized call: nothing but launch latency and host work
        dict(_case("prefill", 2, 128, 128, 4, 4, 64, "fp16"), name="prefill_tiny_b2_s128"),
        # one user's decoding step on a short context: latency again, and too few heads to fill the chip by themselves
        dict(_case("decode", 1, 1, 2048, 32, 8, 128), name="decode_single_L2048"),
        # a serving batch, contiguous cache, new token appended in place with rotary embedding
        dict(_case("decode", 64, 1, 8191, 32, 8, 128, sk_lo=1024, append=True, rotary=True), name="decode_b64_append_rotary"),
        # speculative decoding on a paged cache with a sliding window
        dict(_case("decode", 32, 4, 32768, 64, 8, 128, sk_lo=512, page=256, window=4096), name="decode_b32_paged_window"),
        # long context: 4.3 GB of keys and values for 8 query rows
        dict(_case("decode", 8, 1, 131072, 64, 8, 128), name="decode_long_L131072"),
        # paged decode of wide heads with a plan made ahead of the loop
        dict(_case("decode", 16, 1, 4096, 32, 8, 256, api="v3", sk_lo=300, page=128, plan=True), name="decode_paged_d256_planned"),
        # causal prefill of 4 K tokens, multi-head
        dict(_case("prefill", 4, 4096, 4096, 32, 32, 128), name="prefill_causal_4k"),
        # one scheduler step of chunked prefill: ragged chunks of several requests against their paged caches
        dict(_case("chunk", 4, 2048, 8192, 32, 8, 128, api="v3", sq_lo=301, sk_lo=1777, page=128), name="prefill_chunks_paged"),
        # wide heads, soft-capped scores, grouped heads, an odd length
        dict(_case("prefill", 2, 2047, 2047, 16, 8, 256, softcap=50.0), name="prefill_d256_softcap"),
        # a training step's attention at the prefill shape
        dict(_case("train", 4, 4096, 4096, 32, 32, 128), name="train_causal_4k"),
        # packed documents of odd lengths, grouped heads, fp16
        dict(_case("packed", 12, 2999, 2999, 16, 4, 64, "fp16", sq_lo=37, sk_lo=37), name="train_packed_d64_fp16"),
        # training with wide heads, an odd length
        dict(_case("train", 2, 1777, 1777, 8, 8, 256), name="train_d256_s1777"),
    ]


HEADS = ((4, 4), (8, 8), (16, 16), (32, 32), (8, 1), (16, 4), (16, 8), (32, 8), (64, 8))
MOST_FLOPS = 5.5e11  # of one forward: the 4 K causal prefill
MOST_BYTES = 4.3e9   # the long-context decode


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges that listed() stands for: sizes spread over their logarithm, shrunk until the case costs no
    more than the largest listed one of its kind."""
    kind = rng.choice(("prefill", "train", "packed", "chunk", "decode", "decode"))
    h, hk = rng.choice(HEADS)
    d = rng.choice((64, 96, 128, 128, 128, 192, 256))
    c = _case(kind, 1, 1, 1, h, hk, d, rng.choice(("bf16", "bf16", "fp16")), api=rng.choice(("v2", "v3")))
    c["causal"] = rng.random() < 0.8
    if kind == "decode":
        c["b"], c["sq"], c["sk"] = _log(rng, 1, 128), rng.choice((1, 1, 1, 2, 4)), _log(rng, 256, 131072)
        c["sq_lo"] = c["sq"]
        while c["b"] > 1 and 4.0 * c["b"] * c["sk"] * hk * d > MOST_BYTES:
            c["b"] //= 2
        c["sk_lo"] = max(c["sq"], c["sk"] // rng.choice((1, 2, 8, 32)))
        c["page"] = rng.choice((0, 128, 256))
        c["append"] = rng.random() < 0.4
        c["rotary"] = c["append"] and rng.random() < 0.6
        c["window"] = rng.choice((-1, -1, -1, 1024, 4096))
        c["causal"] = c["causal"] or c["window"] >= 0 or c["rotary"]
        c["plan"] = c["api"] == "v3" and rng.random() < 0.5
        return c
    c["b"], c["sq"] = _log(rng, 1, 8), _log(rng, 100, 8192)
    c["sk"] = c["sq"]
    if kind == "chunk":
        c["api"], c["page"] = "v3", rng.choice((128, 256))
        c["sq"] = min(c["sq"], 4096)
        c["sk"] = _log(rng, c["sq"], 32768)
    elif kind == "packed":
        c["b"] = _log(rng, 1, 32)
    elif rng.random() < 0.2:
        c["softcap"], c["dtype"] = 30.0, "bf16"
    if kind == "prefill" and c["causal"] and rng.random() < 0.2:
        c["window"] = rng.choice((256, 1024))
    c["sq_lo"], c["sk_lo"] = c["sq"], c["sk"]
    if kind in ("chunk", "packed"):
        c["sq_lo"] = max(1, c["sq"] // rng.choice((1, 4, 64)))
        c["sk_lo"] = c["sq_lo"] if kind == "packed" else max(c["sq"], c["sk"] // rng.choice((1, 4)))
    while c["b"] > 1 and 4.0 * d * h * sum(_pairs(c)) > MOST_FLOPS:
        c["b"] //= 2
    while 4.0 * d * h * sum(_pairs(c)) > MOST_FLOPS:
        for n in ("sq", "sq_lo", "sk", "sk_lo"):
            c[n] = max(1, c[n] // 2)
    return c


def _spread(lo, hi, n):
    return [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _lengths(c):
    """(query rows, keys) of every sequence, shortest first; keys include appended ones."""
    more = c["sq"] if c["append"] else 0
    return list(zip(_spread(c["sq_lo"], c["sq"], c["b"]), [n + more for n in _spread(c["sk_lo"], c["sk"], c["b"])]))


def _pairs(c):
    """Visible (query, key) pairs of every sequence."""
    got = []
    for nq, nk in _lengths(c):
        last = np.arange(nq, dtype=np.int64) + nk - nq if c["causal"] else np.full(nq, nk - 1, dtype=np.int64)
        first = np.maximum(0, np.arange(nq, dtype=np.int64) + nk - nq - c["window"]) if c["window"] >= 0 else 0
        got.append(float(np.maximum(0, last + 1 - first).sum()))
    return got


def work(case):
    c = case
    nq = sum(a for a, _ in _lengths(c))
    seen = sum(min(k, c["window"] + q) if c["window"] >= 0 else k for q, k in _lengths(c))  # keys that any query row sees
    q_bytes, kv_bytes, lse = 2.0 * nq * c["h"] * c["d"], 4.0 * seen * c["hk"] * c["d"], 4.0 * nq * c["h"]
    flops = 4.0 * c["d"] * c["h"] * sum(_pairs(c))
    if c["kind"] in ("train", "packed"):
        # forward: q, k, v in, out and lse out; backward: those and dout in, dq, dk, dv out
        return {"bytes": 6 * q_bytes + 3 * kv_bytes + 2 * lse, "flops": 3.5 * flops}
    more = 4.0 * nq * c["hk"] * c["d"] if c["append"] else 0.0  # new keys and values are read from their own tensors and written
    return {"bytes": 2 * q_bytes + kv_bytes + lse + more, "flops": flops}


def tolerance(case):
    """Probabilities and (in the backward) score gradients are rounded to the input type before the second product, and results
    are rounded to it: relative errors of 2^-9 (bf16) or 2^-12 (fp16) each, root mean square, of which a backward adds up
    several."""
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 3e-3}


def _randn(gen, dtype, *shape):
    return torch.randn(shape, generator=gen, device="cuda", dtype=dtype)


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _cu(lengths):
    return _i32([0] + [int(x) for x in np.cumsum(lengths)])


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    host = np.random.RandomState(int(seed) % (1 << 31))
    dt, b, h, hk, d = DTYPES[c["dtype"]], c["b"], c["h"], c["hk"], c["d"]
    lengths = _lengths(c)
    host.shuffle(lengths)
    s = dict(c, window_size=(c["window"], -1), lengths=lengths)
    if c["kind"] in ("prefill", "train"):
        s["q"], s["k"], s["v"] = (_randn(gen, dt, b, n, heads, d) for n, heads in ((c["sq"], h), (c["sk"], hk), (c["sk"], hk)))
    elif c["kind"] == "packed":
        total = sum(a for a, _ in lengths)
        s["q"], s["k"], s["v"] = (_randn(gen, dt, total, heads, d) for heads in (h, hk, hk))
        s["cu"], s["longest"] = _cu([a for a, _ in lengths]), c["sq"]
    if c["kind"] in ("train", "packed"):
        s["dout"] = _randn(gen, dt, *s["q"].shape)
        for n in ("q", "k", "v"):
            s[n].requires_grad_(True)
    if c["kind"] in ("chunk", "decode"):
        _prepare_cache(s, gen, host, dt)
    return s


def _prepare_cache(s, gen, host, dt):
    b, h, hk, d, page = s["b"], s["h"], s["hk"], s["d"], s["page"]
    new = s["sq"] if s["append"] else 0
    room = s["sk"] + new
    if page:
        per = -(-room // page)
        blocks = b * per
        s["table"] = _i32(host.permutation(blocks).reshape(b, per).tolist())
        s["k_cache"], s["v_cache"] = (_randn(gen, dt, blocks, page, hk, d) for _ in range(2))
        room = per * page
    else:
        s["table"] = None
        s["k_cache"], s["v_cache"] = (_randn(gen, dt, b, room, hk, d) for _ in range(2))
    s["lens"] = _i32([k - new for _, k in s["lengths"]])
    if s["kind"] == "chunk":
        s["q"] = _randn(gen, dt, sum(a for a, _ in s["lengths"]), h, d)
        s["cu"] = _cu([a for a, _ in s["lengths"]])
    else:
        s["q"] = _randn(gen, dt, b, s["sq"], h, d)
    s["k_new"], s["v_new"] = (_randn(gen, dt, b, new, hk, d) for _ in range(2)) if new else (None, None)
    s["cos"] = s["sin"] = None
    if s["rotary"]:
        inv = 10000.0 ** (-torch.arange(0, d, 2, dtype=torch.float32, device="cuda") / d)
        angle = torch.arange(room, dtype=torch.float32, device="cuda")[:, None] * inv[None, :]
        s["cos"], s["sin"] = torch.cos(angle).to(dt), torch.sin(angle).to(dt)
    s["metadata"] = None
    if s["plan"]:
        s["metadata"] = fa3.get_scheduler_metadata(
            b, s["sq"], room, h, hk, d, s["lens"], qkv_dtype=dt, page_size=page or None, max_seqlen_k_new=new,
            causal=s["causal"], window_size=s["window_size"])


def run(s):
    kind, v3 = s["kind"], s["api"] == "v3"
    mask = dict(causal=s["causal"], window_size=s["window_size"], softcap=s["softcap"])
    if kind == "prefill":
        return tuple((fa3 if v3 else fa2).flash_attn_func(s["q"], s["k"], s["v"], return_attn_probs=True, **mask)[:2])
    if kind == "train":
        out = (fa3 if v3 else fa2).flash_attn_func(s["q"], s["k"], s["v"], **mask)
        return (out,) + torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])
    if kind == "packed":
        out = (fa3 if v3 else fa2).flash_attn_varlen_func(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["longest"], s["longest"], **mask)
        return (out,) + torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])
    if kind == "chunk":
        return tuple(fa3.flash_attn_with_kvcache(
            s["q"], s["k_cache"], s["v_cache"], cache_seqlens=s["lens"], page_table=s["table"], cu_seqlens_q=s["cu"],
            max_seqlen_q=s["sq"], return_softmax_lse=True, **mask)[:2])
    kw = dict(rotary_cos=s["cos"], rotary_sin=s["sin"], cache_seqlens=s["lens"], rotary_interleaved=False,
              return_softmax_lse=True, **mask)
    if v3:
        out = fa3.flash_attn_with_kvcache(s["q"], s["k_cache"], s["v_cache"], s["k_new"], s["v_new"], page_table=s["table"],
                                          scheduler_metadata=s["metadata"], **kw)[:2]
    else:
        out = fa2.flash_attn_with_kvcache(s["q"], s["k_cache"], s["v_cache"], s["k_new"], s["v_new"], block_table=s["table"], **kw)
    return tuple(out) + ((s["k_cache"], s["v_cache"]) if s["append"] else ())
