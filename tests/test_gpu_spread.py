"""The spread form of the 16-bit step kernel: shares of the key tiles, one block each, in a workspace that a second
launch folds. Held against 64 bits on the same rounded inputs (the tolerances of the other step tests: 1e-3 for fp16 and
8e-3 for bf16 P, absolute and relative; log-sum-exps 1e-5), and against the key split, which the same calls take without
a workspace."""
import ctypes as C
import random

import numpy as np
import pytest
import torch

from ring_attention_b200 import api
from ring_attention_b200._lib import RA_BF16, RA_F16, SegMap, lib
from util import assert_close

pytestmark = pytest.mark.gpu

TOL = {torch.float16: 1e-3, torch.bfloat16: 8e-3}
SPREAD = 128
CAUSAL, FRESH, FINALIZE = 1, 2, 4


def in_64_bits(q, k, v, qpos, kpos, causal, doc):
    """(out, log-sum-exp), on the GPU; rows that see nothing give 0 and -inf."""
    group = q.shape[1] // k.shape[1]
    k, v = (x.double().repeat(1, group, 1, 1) for x in (k, v))  # query head h uses KV head h % kv_heads
    s = q.double() @ k.transpose(-1, -2) / np.sqrt(q.shape[-1])
    seen = (kpos[None, :] <= qpos[:, None]) | (not causal)
    if doc:
        seen &= kpos[None, :] // doc == qpos[:, None] // doc
    s.masked_fill_(~seen, -float("inf"))
    lse = s.logsumexp(-1)
    p = torch.exp(s - lse.nan_to_num(neginf=0.0)[..., None])
    return p @ v, lse


def positions(bases, n, stride):
    return torch.cat([torch.arange(n, device="cuda") * stride + b for b in bases])


CASES = {  # B, H, kvH, query bases, rows a segment, key bases, keys a segment, stride, causal, doc_len
    "chunk": (1, 4, 2, [20000], 300, [0], 20300, 1, True, 0),
    "two rows": (2, 4, 4, [19000], 2, [0], 19002, 1, True, 0),
    "odd group, ragged tiles": (2, 3, 1, [21000], 130, [0], 21130, 1, True, 0),
    "segments": (1, 4, 2, [9000, 24000], 150, [0, 8000, 16000], 8000, 1, True, 0),
    "strides": (1, 4, 1, [50001], 140, [0], 20000, 3, True, 0),
    "documents": (1, 3, 1, [20800], 400, [0], 21200, 1, True, 10500),
    "dense": (1, 2, 1, [0], 129, [0], 20000, 1, False, 0),
    "heads of a tile": (1, 8, 2, [20000], 24, [0], 20024, 1, True, 0),
    "some heads left over": (2, 6, 2, [30000], 50, [0], 15000, 2, True, 0),
    "half a tile each": (1, 16, 1, [16000], 64, [0], 16064, 1, True, 0),
    "single rows": (1, 7, 1, [30000], 1, [0], 30001, 1, True, 16000),
    "blocks without keys": (1, 2, 2, [0, 22000], 200, [2000], 20000, 1, True, 0),
}


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64, 128, 256])
@pytest.mark.parametrize("case", list(CASES))
def test_spread_steps_match_64_bits(dtype, D, case):
    B, H, kvH, qb, rows, kb, keys, stride, causal, doc = CASES[case]
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda").to(dtype)
               for h, n in ((H, rows * len(qb)), (kvH, keys * len(kb)), (kvH, keys * len(kb))))
    want, want_lse = in_64_bits(q, k, v, positions(qb, rows, stride), positions(kb, keys, stride), causal, doc)
    shape, qmap, kmap = api.AttentionShape(B, H, rows * len(qb), keys * len(kb), D, kvH), SegMap.make(qb, rows), SegMap.make(kb, keys)
    room = keys * len(kb) + 77  # a cache with room: rows of K and V read in place
    ck, cv = (torch.full((B, kvH, room, D), float("nan"), device="cuda").to(dtype) for _ in range(2))
    ck[:, :, :keys * len(kb)], cv[:, :, :keys * len(kb)] = k, v
    state = [torch.full(s, float("nan"), device="cuda") for s in (q.shape, q.shape[:3], q.shape[:3])]
    api.attention_step_ex(q, ck, cv, *state, shape, qmap, kmap, pos_stride=stride, causal=causal, fresh=True, finalize=True,
                          doc_len=doc, kv_row_stride=room)
    assert lib().ra_debug_step_form() & SPREAD
    lse = api.attention_lse(state[1], state[2])
    seen = torch.isfinite(want_lse)
    assert_close(state[0].cpu().numpy(), want.cpu().numpy(), TOL[dtype], TOL[dtype], "out")
    assert_close(lse[seen].cpu().numpy(), want_lse[seen].cpu().numpy(), 1e-5, 1e-5, "lse")
    assert (state[1][~seen] == -float("inf")).all() and (state[2][~seen] == 0).all()
    # twice the same keys into a state: the same rows, and log-sum-exps log(2) up; a normalised state of rows that see
    # nothing stays what it was
    state = [torch.full(s, x, device="cuda") for s, x in ((q.shape, 0.0), (q.shape[:3], -float("inf")), (q.shape[:3], 0.0))]
    for flags in (0, FINALIZE):
        api.attention_step_ex(q, k, v, *state, shape, qmap, kmap, pos_stride=stride, causal=causal, finalize=flags != 0, doc_len=doc)
        assert lib().ra_debug_step_form() & SPREAD
    lse = api.attention_lse(state[1], state[2])
    assert_close(state[0].cpu().numpy(), want.cpu().numpy(), TOL[dtype], TOL[dtype], "two steps")
    assert_close(lse[seen].cpu().numpy(), want_lse[seen].cpu().numpy() + np.log(2), 1e-5, 1e-5, "lse of two steps")
    assert api.device_status()[0] == 0


def call(entry, q, k, v, state, shape, qmap, kmap, stride, flags, doc, ws=None, ws_bytes=0):
    code = RA_F16 if q.dtype == torch.float16 else RA_BF16
    args = [code, *(api._ptr(t) for t in (q, k, v, *state)), C.byref(shape.c()), C.byref(qmap), C.byref(kmap), stride, flags, doc, 0]
    api.check(lib().ra_attention_step_ex(*args, api._stream()) if entry == "ex" else
              lib().ra_attention_step_ws(*args, ws, ws_bytes, api._stream()))
    return lib().ra_debug_step_form()


def test_random_spread_calls_match_the_key_split():
    # (both round P to 16 bits under reference points that may differ: two roundings of 2^-11 / 2^-8 of every P, which
    # average out over the keys)
    rng, taken = random.Random(5), 0
    for n in range(250):
        kvH = rng.choice([1, 2, 3, 4, 8])
        B, H, D = rng.choice([1, 2]), kvH * rng.choice([1, 2, 3, 4]), rng.choice([32, 64, 128, 256])
        dtype = rng.choice([torch.float16, torch.bfloat16])
        rows, stride = rng.choice([1, 2, 5, 7, 16, 33, 42, 43, 64, 65, 127, 128, 129, 200, 257, 400]), rng.choice([1, 1, 2])
        nq, nk = rng.choice([1, 1, 2, 3]), rng.choice([1, 1, 2])
        keys = rng.randrange(1000, 20000)
        qb = sorted(rng.randrange(0, 30000) for _ in range(nq))
        kb = sorted(rng.randrange(0, 15000) for _ in range(nk))
        if rng.random() < 0.2:
            qb.reverse()
        flags = rng.choice([0, CAUSAL, CAUSAL]) | rng.choice([0, FRESH]) | rng.choice([0, FINALIZE])
        doc = rng.choice([0, 0, 0, 900, 12000])
        shape, qmap, kmap = api.AttentionShape(B, H, nq * rows, nk * keys, D, kvH), SegMap.make(qb, rows), SegMap.make(kb, keys)
        need = lib().ra_attention_step_workspace_bytes(RA_F16, C.byref(shape.c()), C.byref(qmap), C.byref(kmap), stride, flags, doc)
        if need == 0:
            continue
        taken += 1
        g = torch.Generator(device="cuda").manual_seed(n)
        q, k, v = (torch.randn(B, h, s, D, generator=g, device="cuda").to(dtype) for h, s in ((H, nq * rows), (kvH, nk * keys), (kvH, nk * keys)))
        old = [torch.randn(B, H, nq * rows, D, generator=g, device="cuda"), torch.randn(B, H, nq * rows, generator=g, device="cuda"),
               torch.rand(B, H, nq * rows, generator=g, device="cuda") + 0.5]
        a, b = [t.clone() for t in old], [t.clone() for t in old]
        guard = torch.full((need + 256,), 0x5a, dtype=torch.uint8, device="cuda")
        assert not call("ex", q, k, v, a, shape, qmap, kmap, stride, flags, doc) & SPREAD
        assert call("ws", q, k, v, b, shape, qmap, kmap, stride, flags, doc, guard.data_ptr(), need) & SPREAD
        assert (guard[need:] == 0x5a).all()
        what = f"{n}: B{B} H{H}/{kvH} D{D} {rows} x {qb} on {keys} x {kb} stride {stride} flags {flags} doc {doc}"
        lse = [(t[1] + torch.log(t[2])).cpu().numpy() for t in (a, b)]
        assert_close(lse[1][np.isfinite(lse[0])], lse[0][np.isfinite(lse[0])], 1e-5, 1e-5, what)
        assert np.array_equal(np.isfinite(lse[0]), np.isfinite(lse[1])), what
        x, y = ((t[0] if flags & FINALIZE else t[0] / t[2][..., None]).nan_to_num().cpu().numpy() for t in (a, b))
        assert_close(y, x, TOL[dtype], TOL[dtype], what)
    assert taken >= 20 and api.device_status()[0] == 0


def spoil(what, q, k, v):
    last = k.shape[2] - 1 - q.shape[2]  # every row sees the keys up to here
    if what == "scores":
        k[:, :, 777, 1] = float("nan")       # NaN in every row
    elif what == "scores, some heads":
        k[:, 0, 5, 2] = float("inf")         # +inf or -inf by the sign of q
        k[:, 0, last, 0] = float("nan")
    elif what == "values":
        v[:, :, 100, 3] = float("inf")
        v[:, :, last - 70, 0] = float("nan")
        v[:, :, 4000, 5], v[:, :, 4001, 5] = float("inf"), -float("inf")
    elif what == "queries":
        q[:, 1, 0] = float("nan")
        q[:, -1, -1, 3] = float("inf")
        q[:, 0, q.shape[2] // 2] = -float("inf")
    elif what == "hidden key":
        k[:, :, 300] = -float("inf")         # a score of -inf in every row, and nothing else
        q.abs_()
        q[q == 0] = 1


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64, 128, 256])
@pytest.mark.parametrize("H,kvH,rows", [(4, 2, 200), (6, 2, 24), (7, 1, 50), (5, 1, 1)])  # rows of a head, heads that share tiles
@pytest.mark.parametrize("what", ["plain", "scores", "scores, some heads", "values", "queries", "hidden key"])
def test_what_is_not_finite_stays_where_it_belongs(dtype, D, H, kvH, rows, what):
    """Beside the key split, which rounds the same P: the same elements are finite, and they agree. Rows that only fill a tile hold
    what shared memory held, here NaN."""
    keys = 20000 + rows
    g = torch.Generator(device="cuda").manual_seed(rows)
    q, k, v = (torch.randn(1, h, n, D, generator=g, device="cuda").to(dtype) for h, n in ((H, rows), (kvH, keys), (kvH, keys)))
    nan = torch.full((1, 160, 256, D), float("nan"), device="cuda", dtype=dtype)
    junk = [torch.empty(s, device="cuda") for s in (nan.shape, nan.shape[:3], nan.shape[:3])]
    spoil(what, q, k, v)
    shape, qmap, kmap = api.AttentionShape(1, H, rows, keys, D, kvH), SegMap.make([keys - rows], rows), SegMap.make([0], keys)
    need = lib().ra_attention_step_workspace_bytes(RA_F16, C.byref(shape.c()), C.byref(qmap), C.byref(kmap), 1, CAUSAL | FRESH | FINALIZE, 0)
    ws = torch.full((need,), 0xff, dtype=torch.uint8, device="cuda")
    a, b = ([torch.full(s, 7.0, device="cuda") for s in (q.shape, q.shape[:3], q.shape[:3])] for _ in range(2))
    assert not call("ex", q, k, v, a, shape, qmap, kmap, 1, CAUSAL | FRESH | FINALIZE, 0) & SPREAD
    call("ex", nan, nan, nan, junk, api.AttentionShape(1, 160, 256, 256, D, 160), SegMap.make([0], 256), SegMap.make([0], 256), 1, FRESH, 0)
    assert call("ws", q, k, v, b, shape, qmap, kmap, 1, CAUSAL | FRESH | FINALIZE, 0, ws.data_ptr(), need) & SPREAD
    for x, y in zip(a, b):
        assert torch.equal(x.isfinite(), y.isfinite())
    finite = a[0].isfinite()
    assert finite.all() == (what in ("plain", "hidden key"))
    assert finite.any() == (what != "scores" and (what != "scores, some heads" or kvH > 1))
    assert_close(b[0][finite].cpu().numpy(), a[0][finite].cpu().numpy(), TOL[dtype], TOL[dtype], what)
    assert api.device_status()[0] == 0


@pytest.mark.parametrize("D", [64, 256])
def test_other_forms_run_without_a_usable_workspace(D):
    B, H, kvH, rows, keys = 1, 4, 2, 200, 20000
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(B, h, s, D, generator=g, device="cuda").half() for h, s in ((H, rows), (kvH, keys), (kvH, keys)))
    shape, qmap, kmap = api.AttentionShape(B, H, rows, keys, D, kvH), SegMap.make([keys - rows], rows), SegMap.make([0], keys)

    def bytes_for(flags=CAUSAL | FRESH, s=shape, km=kmap):
        return lib().ra_attention_step_workspace_bytes(RA_F16, C.byref(s.c()), C.byref(qmap), C.byref(km), 1, flags, 0)

    need = bytes_for()
    ws = torch.empty(need + 64, dtype=torch.uint8, device="cuda")
    state = [torch.empty(s, device="cuda") for s in (q.shape, q.shape[:3], q.shape[:3])]
    forms = [call("ws", q, k, v, state, shape, qmap, kmap, 1, CAUSAL | FRESH, 0, p, n)
             for p, n in ((None, 0), (None, need), (ws.data_ptr(), need - 1), (ws.data_ptr() + 4, need), (ws.data_ptr(), need))]
    assert [f & SPREAD for f in forms] == [0, 0, 0, 0, SPREAD]
    # asked for another form, too few keys, nothing to do, nonsense
    assert bytes_for(CAUSAL | 3 << 8) == bytes_for(CAUSAL | 16) == bytes_for(CAUSAL | 8) == 0
    assert bytes_for(s=api.AttentionShape(B, H, rows, 2047, D, kvH), km=SegMap.make([0], 2047)) == 0
    assert bytes_for(s=api.AttentionShape(B, H, rows, 0, D, kvH), km=SegMap.make([0], 0)) == 0
    assert bytes_for(s=api.AttentionShape(B, H, rows + 1, keys, D, kvH)) == 0


def test_spread_calls_replay_from_a_graph_and_keep_their_state_behind_one_that_gave_up():
    B, H, kvH, rows, keys, D = 1, 4, 2, 200, 20000, 128
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(B, h, s, D, generator=g, device="cuda").half() for h, s in ((H, rows), (kvH, keys), (kvH, keys)))
    shape, qmap, kmap = api.AttentionShape(B, H, rows, keys, D, kvH), SegMap.make([keys - rows], rows), SegMap.make([0], keys)

    def run(state, **kw):
        api.attention_step_ex(q, k, v, *state, shape, qmap, kmap, causal=True, fresh=True, finalize=True, **kw)

    want, state = ([torch.full(s, 3.0, device="cuda") for s in (q.shape, q.shape[:3], q.shape[:3])] for _ in range(2))
    run(want)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        run(state)
        run(state)
    for t in state:
        t.fill_(0)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(state, want))
    state = [torch.full_like(t, 3.0) for t in want]
    lib().ra_debug_set_wait_limit_ns(5_000_000)
    lib().ra_debug_stall_producer_after(4)  # some shares end, others wait for keys that never come
    try:
        run(state)
        lib().ra_debug_stall_producer_after(-1)
        run(state)  # starts beside the first
        torch.cuda.synchronize()
    finally:
        lib().ra_debug_stall_producer_after(-1)
        lib().ra_debug_set_wait_limit_ns(0)
    assert api.device_status()[0] == 5
    assert all((t == 3.0).all() for t in state)
