"""The work this library is used for, as measurable cases.

Four operations, all through the package's public entry points:

* ``train``   : one layer's training step: ``flash_moba_varlen_func`` forward, autograd backward
  (outputs O, dQ, dK, dV);
* ``prefill`` : the same function without gradients, queries and keys of equal length;
* ``cached``  : serving against a key/value cache whose centroids are kept in a ``CentroidCache``:
  ``CentroidCache.attend`` with one new row per sequence (decode) or with a block of new rows per
  sequence (chunked prefill);
* ``pattern`` : ``flash_topk_varlen_func`` alone (pool, gating, column pattern), for callers that
  build a layer's pattern once and hand it to the attention themselves.

Inputs are independent normal values, as in the benchmark configurations of this repository
(`bench.py`), whose shapes the large cases take; selections are then close to uniform over the chunks.
"""
import math

import numpy as np
import torch

import flash_moba_b200 as F

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(name, op, lens_q, lens_k=None, *, heads, heads_k, d, chunk, topk, causal=True, dtype="bf16", scale=1.0):
    text = lambda xs: ",".join(str(int(x)) for x in xs)  # noqa: E731
    c = {"op": op, "lens_q": text(lens_q), "lens_k": text(lens_q if lens_k is None else lens_k), "heads": heads,
         "heads_k": heads_k, "d": d, "chunk": chunk, "topk": topk, "causal": causal, "dtype": dtype, "scale": scale}
    return c if name is None else dict(c, name=name)


def _ints(text):
    return [int(x) for x in text.split(",")]


# the sixteen ragged lengths of the grouped-query configuration in bench.py
GQA_LENGTHS = [29760, 14720, 26944, 31232, 15872, 3392, 10560, 18816, 17984, 15360, 32192, 27776, 29248, 12032, 17728, 13824]


def listed():
    return [
        # the smallest configuration: two short sequences, small heads; a step is bound by the host and by launches
        _case("train_tiny", "train", [1024, 2048], heads=8, heads_k=8, d=64, chunk=128, topk=4),
        # the headline: one 64K sequence, a full layer of 32 heads
        _case("train_64k", "train", [65536], heads=32, heads_k=32, d=128, chunk=128, topk=8),
        # a usual training batch: packed 8K sequences
        _case("train_8x8k", "train", [8192] * 8, heads=32, heads_k=32, d=128, chunk=128, topk=8),
        # grouped queries, ragged sequences, narrow chunks and long lists; the largest case
        _case("train_gqa_ragged", "train", GQA_LENGTHS, heads=32, heads_k=8, d=128, chunk=64, topk=16),
        # long context with wide chunks: the heads that one of eight GPUs holds
        _case("train_512k_4heads", "train", [524288], heads=4, heads_k=4, d=128, chunk=256, topk=16, scale=0.5),
        # wide heads, half precision, grouped queries, lengths that fit no tile
        _case("train_d256_odd", "train", [9001, 4777, 2611], heads=16, heads_k=4, d=256, chunk=128, topk=8, dtype="fp16"),
        # encoder layer: no causal mask, small heads, narrow chunks, half precision, odd lengths
        _case("train_encoder_d64", "train", [4096, 3001, 1777, 517], heads=12, heads_k=12, d=64, chunk=64, topk=8,
              causal=False, dtype="fp16"),
        # prompt processing of one 32K prompt
        _case("prefill_32k", "prefill", [32768], heads=16, heads_k=16, d=128, chunk=128, topk=8, scale=0.5),
        # chunked prefill: blocks of new rows behind caches of various lengths, one block almost empty
        _case("extend_ragged", "cached", [512, 1000, 37, 2048], [20000, 9111, 32768, 4096], heads=32, heads_k=8, d=128,
              chunk=128, topk=8, dtype="fp16"),
        # decoding: one new row in each of sixteen sequences of various lengths
        _case("decode_16", "cached", [1] * 16, [n - 13 for n in GQA_LENGTHS], heads=32, heads_k=8, d=128, chunk=128, topk=8),
        # decoding a single long sequence: latency alone
        _case("decode_1", "cached", [1], [65001], heads=32, heads_k=8, d=128, chunk=128, topk=8),
        # the pattern of the 32K prompt by itself
        _case("pattern_32k", "pattern", [32768], heads=16, heads_k=16, d=128, chunk=128, topk=8, scale=0.5),
    ]


# A drawn case's (row, chunk) entries in units of 128 keys and 128 values, and its (row, centroid) scores: about half
# of what the largest listed case has
MOST_ENTRIES = 8e7
MOST_SCORES = 1.5e9


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ragged(rng, total, n):
    """n lengths of about `total` in all, mostly odd ones, none empty."""
    shares = [rng.uniform(0.2, 1.0) for _ in range(n)]
    return [max(1, int(total * s / sum(shares))) for s in shares]


def draw(rng):
    op = rng.choice(["train"] * 5 + ["prefill"] * 2 + ["cached"] * 3 + ["pattern"] * 2)
    d = rng.choice([64, 128] if op == "cached" else [64, 64, 96, 128, 128, 128, 128, 256])
    chunk = rng.choice([64, 128, 128, 256])
    topk = rng.choice([4, 8, 8, 12, 16])
    heads_k = rng.choice([1, 2, 4, 8, 16])
    heads = min(32, heads_k * rng.choice([1, 1, 2, 4, 8]))
    causal = op == "cached" or rng.random() < 0.85
    nseq = rng.choice([1, 1, 2, 3, 5, 8, 16])
    if op == "cached":
        nseq = rng.choice([1, 2, 5, 8, 16, 33, 64])
        lens_k = [_log_uniform(rng, 300, 60000) for _ in range(nseq)]
        lens_q = [1] * nseq if rng.random() < 0.6 else [min(n, _log_uniform(rng, 2, 2500)) for n in lens_k]
    else:
        lens_k = lens_q = _ragged(rng, _log_uniform(rng, 900, 260000), nseq)
    while True:
        units = sum(lens_q) * heads * topk * max(1.0, d / 128) * max(1.0, chunk / 128)
        scores = sum(a * b for a, b in zip(lens_q, lens_k)) / chunk * heads
        rows = sum(lens_k) * heads_k * d + sum(lens_q) * heads * d
        if units <= MOST_ENTRIES and scores <= MOST_SCORES and rows <= 1e9:
            break
        lens_q, lens_k = [max(1, n * 2 // 3) for n in lens_q], [max(1, n * 2 // 3) for n in lens_k]
    return _case(None, op, lens_q, lens_k, heads=heads, heads_k=heads_k, d=d, chunk=chunk, topk=topk, causal=causal,
                 dtype=rng.choice(["bf16", "bf16", "fp16"]), scale=rng.choice([0.5, 1.0]))


def _cu(lens):
    return torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device="cuda")


def prepare(case, seed):
    lens_q, lens_k = _ints(case["lens_q"]), _ints(case["lens_k"])
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype, d = DTYPES[case["dtype"]], case["d"]

    def rows(n, heads, scale):
        return torch.randn(n, heads, d, generator=gen, device="cuda", dtype=dtype).mul_(scale)

    s = dict(case=case, q=rows(sum(lens_q), case["heads"], case["scale"]), k=rows(sum(lens_k), case["heads_k"], case["scale"]),
             cu_q=_cu(lens_q), cu_k=_cu(lens_k), max_q=max(lens_q), max_k=max(lens_k))
    if case["op"] != "pattern":
        s["v"] = rows(sum(lens_k), case["heads_k"], case["scale"])
    if case["op"] == "train":
        s["dout"] = rows(sum(lens_q), case["heads"], 1.0)
        for n in ("q", "k", "v"):
            s[n].requires_grad_(True)
    if case["op"] == "cached":
        s["cache"] = F.CentroidCache(len(lens_k), case["heads_k"], d, case["chunk"], max(lens_k), dtype=dtype)
        s["cache"].update(s["k"], [0] + [int(x) for x in np.cumsum(lens_k)], lens_k)
    return s


def run(s):
    c = s["case"]
    if c["op"] == "pattern":
        return F.flash_topk_varlen_func(s["q"], s["k"], s["cu_q"], s["cu_k"], s["max_q"], s["max_k"], c["topk"], c["chunk"],
                                        causal=c["causal"])
    if c["op"] == "cached":
        with torch.no_grad():
            return s["cache"].attend(s["q"], s["k"], s["v"], s["cu_q"], s["cu_k"], s["max_q"], s["max_k"], c["topk"])
    if c["op"] == "prefill":
        with torch.no_grad():
            return F.flash_moba_varlen_func(s["q"], s["k"], s["v"], s["cu_q"], s["cu_k"], s["max_q"], s["max_k"], c["chunk"],
                                            c["topk"], causal=c["causal"])
    out = F.flash_moba_varlen_func(s["q"], s["k"], s["v"], s["cu_q"], s["cu_k"], s["max_q"], s["max_k"], c["chunk"], c["topk"],
                                   causal=c["causal"])
    dq, dk, dv = torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])
    return {"out": out.detach(), "dq": dq, "dk": dk, "dv": dv}


def _counts(case):
    """(selected unmasked (row, key) pairs, selected (row, chunk) entries, (row, centroid) scores), per query head."""
    pairs = entries = scores = 0
    chunk, topk = case["chunk"], case["topk"]
    for lq, lk in zip(_ints(case["lens_q"]), _ints(case["lens_k"])):
        n = -(-lk // chunk)
        if not case["causal"]:
            pairs += lq * min(lk, min(topk, n) * chunk)
            entries += lq * min(topk, n)
            scores += lq * n
            continue
        pos = np.arange(lk - lq, lk, dtype=np.int64)          # bottom-right aligned
        pos = pos[pos >= 0]
        own = pos // chunk
        sel = np.minimum(topk, own + 1)
        pairs += int(((sel - 1) * chunk + pos % chunk + 1).sum())
        entries += int(sel.sum())
        scores += int(own.sum())
    return pairs, entries, scores


def work(case):
    lens_q, lens_k = _ints(case["lens_q"]), _ints(case["lens_k"])
    H, Hk, d = case["heads"], case["heads_k"], case["d"]
    tq, tk, el = sum(lens_q), sum(lens_k), 2
    chunks = sum(-(-n // case["chunk"]) for n in lens_k)
    pairs, entries, scores = _counts(case)
    q_bytes, kv_bytes = tq * H * d * el, tk * Hk * d * el
    gate_flops = 2 * d * scores * H
    if case["op"] == "pattern":
        ncol = -(-max(lens_k) // case["chunk"])
        return {"bytes": q_bytes + kv_bytes + tq * H * case["topk"] * 4 + 12 * len(lens_q) * H * ncol,
                "flops": gate_flops + tk * Hk * d}
    if case["op"] == "cached":
        # the centroids once, and the keys and values of the chunks that any row selects (selections taken as independent)
        used = 0.0
        for lq, lk in zip(lens_q, lens_k):
            n = -(-lk // case["chunk"])
            share = min(1.0, case["topk"] / n)
            used += min(lk, n * (1.0 - (1.0 - share) ** (lq * (H // Hk))) * case["chunk"])
        return {"bytes": 2 * q_bytes + chunks * Hk * d * el + 2 * used * Hk * d * el, "flops": gate_flops + 4 * d * pairs * H}
    if case["op"] == "prefill":
        return {"bytes": 2 * q_bytes + 2 * kv_bytes, "flops": gate_flops + tk * Hk * d + 4 * d * pairs * H}
    # forward and backward: q, k, v, dO read; O, dQ, dK, dV written
    return {"bytes": 4 * q_bytes + 4 * kv_bytes, "flops": gate_flops + tk * Hk * d + 14 * d * pairs * H}


def tolerance(case):
    if case["op"] == "pattern":
        return {"rel": 0.0, "differ": 0.005}      # rows whose k-th and (k+1)-th scores agree to the last bits
    # probabilities, their gradients and each chunk's part of a row are rounded to the inputs' type (8 or 11 bits)
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
