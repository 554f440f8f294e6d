"""Performance cases: what a program that uses this library has it do, through the public API.

Kinds of work:

* ``prefill``: a whole attention pass of one GPU (``Ring.prefill`` with one rank): every layout,
  dense, causal and with a document mask, MHA and GQA, 16-bit and fp32, output and log-sum-exp.
* ``rank``: the compute of one rank of a ring of ``cp`` ranks: a step on its own shard, then one
  per received shard into the same state (``attention_step_ex``), init and finalize fused.
* ``flash``: the stand-alone fp32-in / fp32-out entry points, in fp32 and through fp16.
* ``chunk``: a chunk of new prompt rows against everything a KV cache holds, read in place.
* ``decode``: one query row per sequence against the cache (``run_local_decode_step``); with
  ``tokens`` a whole request: reset, copy the prompt in, then append and decode that often.
"""
import math

import torch

import ring_attention_b200.api as ra

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
LAYOUTS = {"contiguous": 0, "zigzag": 1, "striped": 2}


def case(kind, dtype, batch, heads, kv_heads, seq_q, seq_k, head_dim, causal=True,
         layout="contiguous", n_splits=2, docs=1, cp=1, rank=0, tokens=0, name=None):
    c = {"kind": kind, "dtype": dtype, "batch": batch, "heads": heads, "kv_heads": kv_heads, "seq_q": seq_q,
         "seq_k": seq_k, "head_dim": head_dim, "causal": causal, "layout": layout, "n_splits": n_splits,
         "docs": docs, "cp": cp, "rank": rank, "tokens": tokens}
    return {"name": name, **c} if name else c


def listed():
    return [
        # latency of one token of a chat-sized context, the smallest call a server makes
        case("decode", "fp16", 1, 32, 8, 1, 1061, 128, name="decode_short"),
        # a whole short request of a small batch: prompt into the cache, then token by token
        case("decode", "bf16", 5, 24, 6, 1, 1531, 64, tokens=8, name="generate_ragged_bf16"),
        # the reference's published decode shape: fp32 cache, one sequence, MHA
        case("decode", "fp32", 1, 8, 8, 1, 16384, 128, name="decode_fp32"),
        # the long-context decode workload of the benchmark: the cache is 4.3 GB
        case("decode", "fp16", 4, 32, 8, 1, 262144, 128, name="decode_long"),
        # the reference's unit shape: a short dense fp32 pass
        case("flash", "fp32", 1, 8, 8, 1024, 1024, 64, causal=False, name="flash_fp32_short"),
        # the shape of the reference's command-line benchmark, in fp32
        case("flash", "fp32", 1, 4, 4, 16384, 16384, 128, name="flash_fp32_long"),
        # a small ragged batch, fp32 tensors computed in fp16
        case("flash", "fp16", 2, 12, 12, 1531, 1531, 64, name="flash_half_ragged"),
        # the benchmark's headline workload
        case("prefill", "fp16", 1, 8, 8, 32768, 32768, 64, layout="zigzag", name="prefill_d64"),
        # long-prompt GQA prefill, striped (a quarter of the benchmark's length)
        case("prefill", "fp16", 2, 32, 8, 32768, 32768, 128, layout="striped", name="prefill_gqa"),
        # long packed context: four documents under one mask
        case("prefill", "bf16", 1, 16, 16, 65536, 65536, 128, layout="zigzag", docs=4, name="prefill_docs_bf16"),
        # one rank of four, zig-zag shards of a length that no tile divides
        case("rank", "bf16", 1, 16, 4, 2 * 1021, 8 * 1021, 64, layout="zigzag", cp=4, rank=1, name="rank_zigzag_ragged"),
        # chunked prefill: the next 384 prompt rows against 40000 cached ones
        case("chunk", "fp16", 1, 32, 8, 384, 40384, 128, name="chunk_cached"),
    ]


# ---- work, and draws of the same ranges ----------------------------------------------------


def _positions(c):
    """(query positions, key positions) of a ``prefill`` / ``rank`` case, in storage order: keys
    shard by shard in the order the steps fold them."""
    cp, n = c["cp"], c["n_splits"]
    total = c["seq_k"]

    def shard(r):
        if c["layout"] == "contiguous":
            return torch.arange(total // cp) + r * (total // cp)
        if c["layout"] == "striped":
            return torch.arange(total // cp) * cp + r
        chunk = total // (n * cp)
        parts = []
        for sg in range(n):
            at = (sg // 2 * cp + r) if sg % 2 == 0 else ((n - 1 - sg // 2) * cp + (cp - 1 - r))
            parts.append(torch.arange(chunk) + at * chunk)
        return torch.cat(parts)

    return shard(c["rank"]), [shard((c["rank"] - s) % cp) for s in range(cp)]


def _visible(c):
    """Visible (query, key) pairs of one head."""
    sq, sk = c["seq_q"], c["seq_k"]
    if c["kind"] == "decode":
        return sum(sk + t for t in range(1, c["tokens"] + 1)) if c["tokens"] else sk
    if not c["causal"]:
        return sq * sk // c["docs"]
    if c["kind"] in ("flash", "chunk"):
        return sq * (sk - sq) + sq * (sq + 1) // 2
    q = _positions(c)[0]
    doc = sk // c["docs"]
    return int((q % doc + 1).sum())


def work(c):
    es = 4 if c["dtype"] == "fp32" or c["kind"] == "flash" else 2
    rows_q, heads, kvh, d = c["batch"] * c["heads"] * c["seq_q"], c["heads"], c["kv_heads"], c["head_dim"]
    flops = 4 * c["batch"] * heads * _visible(c) * d
    if c["kind"] == "decode":
        steps = c["tokens"] or 1
        keys = _visible(c)
        if c["tokens"]:  # the prompt is read and written once, every token's row too
            keys += 2 * (c["seq_k"] + steps)
        kv = 2 * c["batch"] * kvh * keys * d * es
        return {"bytes": kv + steps * rows_q * d * (es + 4), "flops": flops}
    kv = 2 * c["batch"] * kvh * c["seq_k"] * d * es
    lse = 0 if c["kind"] == "flash" else 4
    return {"bytes": kv + rows_q * d * (es + 4) + rows_q * lse, "flops": flops}


def _cost(c):
    """A time for the case, from rates its path has (only to bound what draw gives)."""
    w = work(c)
    rate = 1e15 if c["dtype"] != "fp32" else (1.5e14 if c["head_dim"] <= 128 else 1.5e13)
    return max(w["flops"] / rate, w["bytes"] / 3e12)


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["decode", "decode", "decode", "flash", "flash", "prefill", "prefill", "rank", "chunk", "chunk"])
        head_dim = rng.choice([32, 64, 64, 64, 128, 128, 128, 128, 256])
        kv_heads = rng.choice([1, 2, 4, 4, 6, 8, 8, 16])
        heads = kv_heads * rng.choice([1, 1, 2, 3, 4, 4, 8])
        batch = rng.choice([1, 1, 1, 2, 3, 5])
        if heads > 64:
            continue
        if kind == "decode":
            dtype = rng.choice(["fp16", "fp16", "bf16", "fp32"])
            tokens = rng.choice([0, 0, 0, 4, 8])
            seq = span(200, 6000) if tokens else span(200, 262144)
            c = case(kind, dtype, batch, heads, kv_heads, 1, seq, head_dim, tokens=tokens)
        elif kind == "flash":
            sq = span(300, 16384)
            sk = sq if rng.random() < 0.7 else sq + span(100, 8000)
            c = case(kind, rng.choice(["fp32", "fp32", "fp16"]), batch, heads, kv_heads, sq, sk, head_dim,
                     causal=rng.random() < 0.6)
        elif kind == "chunk":
            sq = span(16, 2048)
            c = case(kind, rng.choice(["fp16", "bf16"]), batch, heads, kv_heads, sq, sq + span(1000, 100000), head_dim)
        else:
            cp = 1 if kind == "prefill" else rng.choice([2, 4, 8])
            layout = rng.choice(["contiguous", "zigzag", "zigzag", "striped"])
            n = rng.choice([2, 2, 4]) if layout == "zigzag" else 2
            docs = rng.choice([1, 1, 1, 2, 4])
            unit = cp * n * docs
            total = max(1, span(1000, 65536) // unit) * unit
            dtype = rng.choice(["fp16", "fp16", "bf16", "bf16", "fp32"])
            c = case(kind, dtype, batch, heads, kv_heads, total // cp, total, head_dim, causal=docs > 1 or rng.random() < 0.8,
                     layout=layout, n_splits=n, docs=docs, cp=cp, rank=rng.randrange(cp))
        elements = c["batch"] * (c["heads"] * c["seq_q"] + 2 * c["kv_heads"] * c["seq_k"]) * c["head_dim"]
        if _cost(c) <= most and elements <= 2.2e9:
            return c


# ---- inputs ----------------------------------------------------------------------------------


def _inputs(c, seed):
    """q, k, v (and the new rows of a request) as the seed gives them: N(0, 1), on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float32 if c["kind"] == "flash" else DTYPES[c["dtype"]]
    b, h, kvh, d = c["batch"], c["heads"], c["kv_heads"], c["head_dim"]

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dt)

    if c["kind"] == "decode" and c["tokens"]:
        n = c["tokens"]
        return normal(n, b, h, 1, d), normal(b, kvh, c["seq_k"], d), normal(b, kvh, c["seq_k"], d), \
            normal(n, b, kvh, 1, d), normal(n, b, kvh, 1, d)
    q = normal(b, h, c["seq_q"], d)
    if c["kind"] == "rank":  # one tensor per shard, in the order they arrive
        local = c["seq_k"] // c["cp"]
        return q, [normal(b, kvh, local, d) for _ in range(c["cp"])], [normal(b, kvh, local, d) for _ in range(c["cp"])]
    return q, normal(b, kvh, c["seq_k"], d), normal(b, kvh, c["seq_k"], d)


def prepare(c, seed):
    b, h, kvh, sq, sk, d = (c[k] for k in ("batch", "heads", "kv_heads", "seq_q", "seq_k", "head_dim"))
    s = {"case": c}
    q, k, v, *new = _inputs(c, seed)
    s["q"] = q
    if c["kind"] == "prefill":
        s["k"], s["v"] = k, v
        s["ring"] = ra.Ring()
    elif c["kind"] == "flash":
        s["k"], s["v"] = k, v
        s["shape"] = ra.AttentionShape(b, h, sq, sk, d, kvh)
        s["out"] = torch.empty(b, h, sq, d, device="cuda")
    elif c["kind"] == "rank":
        part = ra.RingPartition(c["cp"], c["rank"], sk, LAYOUTS[c["layout"]], c["n_splits"])
        s["maps"] = [part.step_maps(i) for i in range(c["cp"])]
        s["shape"] = ra.AttentionShape(b, h, sq, sk // c["cp"], d, kvh)
        s["k"], s["v"] = k, v
    else:
        # what a serving program holds: the cache with room to grow, filled with the context
        room = 256
        s["cache"] = ra.DeviceKVCache(b, kvh, sk + room, d, DTYPES[c["dtype"]])
        s["cache"].copy_prefill(k, v, sk)
        if c["kind"] == "chunk":
            s["shape"] = ra.AttentionShape(b, h, sq, sk, d, kvh)
            s["qmap"], s["kmap"] = ra.SegMap.make([sk - sq], sq), ra.SegMap.make([0], sk)
            s["keys"], s["values"] = s["cache"].k_view(), s["cache"].v_view()
        elif new:
            s["k"], s["v"], (s["k_new"], s["v_new"]) = k, v, new
            s["out"] = torch.empty(c["tokens"], b, h, 1, d, device="cuda")
        else:
            s["out"] = torch.empty(b, h, 1, d, device="cuda")
    if c["kind"] in ("rank", "chunk"):
        s["out"] = torch.empty(b, h, sq, d, device="cuda")
        s["m"] = torch.empty(b, h, sq, device="cuda")
        s["l"] = torch.empty(b, h, sq, device="cuda")
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "prefill":
        return s["ring"].prefill(s["q"], s["k"], s["v"], seq=c["seq_k"], causal=c["causal"], layout=LAYOUTS[c["layout"]],
                                 n_splits=c["n_splits"], doc_len=c["seq_k"] // c["docs"] if c["docs"] > 1 else 0,
                                 want_lse=True)
    if c["kind"] == "flash":
        call = ra.launch_flash_attention if c["dtype"] == "fp32" else ra.launch_flash_attention_fp16
        call(s["q"], s["k"], s["v"], s["out"], s["shape"], c["causal"])
        return s["out"]
    if c["kind"] == "rank":
        doc = c["seq_k"] // c["docs"] if c["docs"] > 1 else 0
        for i, (qmap, kmap, stride) in enumerate(s["maps"]):
            ra.attention_step_ex(s["q"], s["k"][i], s["v"][i], s["out"], s["m"], s["l"], s["shape"], qmap, kmap,
                                 pos_stride=stride, causal=c["causal"], fresh=i == 0, finalize=i == c["cp"] - 1,
                                 doc_len=doc)
        return s["out"], ra.attention_lse(s["m"], s["l"])
    if c["kind"] == "chunk":
        ra.attention_step_ex(s["q"], s["keys"], s["values"], s["out"], s["m"], s["l"], s["shape"], s["qmap"], s["kmap"],
                             causal=True, fresh=True, finalize=True, kv_row_stride=s["cache"].s_max())
        return s["out"], ra.attention_lse(s["m"], s["l"])
    cache = s["cache"]
    if not c["tokens"]:
        ra.run_local_decode_step(s["q"], cache, c["heads"], c["seq_k"] - 1, 0, True, s["out"])
        return s["out"]
    cache.reset()
    cache.copy_prefill(s["k"], s["v"], c["seq_k"])
    for t in range(c["tokens"]):
        cache.append(s["k_new"][t], s["v_new"][t])
        ra.run_local_decode_step(s["q"][t], cache, c["heads"], c["seq_k"] + t, 0, True, s["out"][t])
    return s["out"]


# ---- what is right ---------------------------------------------------------------------------


def tolerance(c):
    # about four times the distance from the 64-bit result that the path shows: fp32 sums that a
    # tensor core accumulates (2.6e-5 over 16384 keys) or that a thread does (3e-7), 16-bit
    # probabilities (a relative 2^-11 or 2^-8 each) under fp32 sums, and inputs that the entry
    # point rounds to fp16 first
    if c["dtype"] == "fp32":
        return {"rel": 2e-6 if c["kind"] == "decode" else 1e-4}
    if c["dtype"] == "bf16":
        return {"rel": 6e-3}
    return {"rel": 1.6e-3 if c["kind"] == "flash" else 1e-3}


def _attend(q, k, v, qpos, kpos, causal, doc):
    """softmax(q k^T / sqrt(d)) v and its log-sum-exp in 64 bits, a head and some rows at a time."""
    b, h, sq, d = q.shape
    kvh = k.shape[1]
    out = torch.empty(b, h, sq, d, dtype=torch.float64, device=q.device)
    lse = torch.empty(b, h, sq, dtype=torch.float64, device=q.device)
    step = max(1, min(sq, 2 ** 27 // max(1, k.shape[2])))
    for i in range(b):
        for g in range(kvh):
            kk, vv = k[i, g].double(), v[i, g].double()
            for j in range(g, h, kvh):
                for at in range(0, sq, step):
                    rows = slice(at, min(sq, at + step))
                    s = (q[i, j, rows].double() / math.sqrt(d)) @ kk.T
                    if causal:
                        s.masked_fill_(kpos[None, :] > qpos[rows, None], -math.inf)
                    if doc:
                        s.masked_fill_(kpos[None, :] // doc != qpos[rows, None] // doc, -math.inf)
                    lse[i, j, rows] = s.logsumexp(-1)
                    s.sub_(lse[i, j, rows, None]).exp_()
                    out[i, j, rows] = s @ vv
    return out, lse


def exact(c, seed):
    if c["batch"] * c["heads"] * c["seq_q"] * c["seq_k"] > 8e10:
        return None
    q, k, v, *new = _inputs(c, seed)
    dev = q.device
    if c["kind"] == "decode":
        if not new:
            kpos = torch.arange(c["seq_k"], device=dev)
            return _attend(q, k, v, kpos[-1:], kpos, False, 0)[0]
        outs = []
        for t in range(c["tokens"]):
            k, v = torch.cat([k, new[0][t]], 2), torch.cat([v, new[1][t]], 2)
            kpos = torch.arange(k.shape[2], device=dev)
            outs.append(_attend(q[t], k, v, kpos[-1:], kpos, False, 0)[0])
        return torch.stack(outs)
    if c["kind"] in ("flash", "chunk"):
        kpos = torch.arange(c["seq_k"], device=dev)
        got = _attend(q, k, v, kpos[c["seq_k"] - c["seq_q"]:], kpos, c["causal"], 0)
        return got[0] if c["kind"] == "flash" else got
    qpos, kpos = _positions(c)
    if c["kind"] == "rank":
        k, v = torch.cat(k, 2), torch.cat(v, 2)
    return _attend(q, k, v, qpos.to(dev), torch.cat(kpos).to(dev), c["causal"], c["seq_k"] // c["docs"] if c["docs"] > 1 else 0)
