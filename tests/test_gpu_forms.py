"""GPU parity of the forms that a call's shape selects: the key-split form of the step kernels (the
blocks of a cluster share a query block's keys), the scaled fp16 splitting of the fp32 step, the two
forms of the decode kernels and the one-launch cache append.

Tolerances are those of the other step and decode tests: 1e-5 for fp32 and 1e-3 / 8e-3 for fp16 /
bf16 P, absolute and relative, against the oracle on the same rounded inputs. Where values are
scaled by 2^e the absolute part scales with V."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
from ring_attention_b200 import api
from ring_attention_b200._lib import RA_BF16, RA_F16, RA_F32, SegMap, lib
from util import assert_close, normal_inputs, round_to

pytestmark = pytest.mark.gpu

TOL = {torch.float32: 1e-5, torch.float16: 1e-3, torch.bfloat16: 8e-3}
CODE = {torch.float32: RA_F32, torch.float16: RA_F16, torch.bfloat16: RA_BF16}
CAUSAL, FRESH, FINALIZE = 1, 2, 4


def dev(x, dtype=torch.float32):
    return torch.from_numpy(np.ascontiguousarray(x)).to("cuda").to(dtype).contiguous()


def step(q, k, v, state, shape, qmap, kmap, flags, split=0, doc_len=0):
    out, m, l = state
    api.check(lib().ra_attention_step_ex(
        CODE[q.dtype], api._ptr(q), api._ptr(k), api._ptr(v), api._ptr(out), api._ptr(m), api._ptr(l),
        C.byref(shape.c()), C.byref(qmap), C.byref(kmap), 1, flags | split << 8, doc_len, 0, api._stream()))


def poisoned(B, H, Sq, D):
    return [torch.full(s, float("nan"), device="cuda") for s in ((B, H, Sq, D), (B, H, Sq), (B, H, Sq))]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D", [32, 64, 128, 256])
@pytest.mark.parametrize("split", [1, 2, 3, 8])
def test_key_split_in_two_steps_matches_the_oracle(dtype, D, split):
    # 300 query rows (a whole block and one of a single short tile), two key chunks of which the
    # second has fewer tiles than blocks; document and causal limits leave some shares empty
    if dtype == torch.float32 and D == 256:
        pytest.skip("head_dim 256 in fp32 runs the SIMT kernel")
    B, H, kvH, Sq, Sk, doc = 1, 4, 2, 300, 1333, 900
    q, k, v = (round_to(x, dtype) for x in normal_inputs(5, B, H, kvH, Sq, Sk, D))
    cut = 1100
    qmap = SegMap.make([Sk - Sq], Sq)
    state = poisoned(B, H, Sq, D)
    dq = dev(q, dtype)
    for lo, hi, flags in ((0, cut, FRESH), (cut, Sk, FINALIZE)):
        step(dq, dev(k[:, :, lo:hi], dtype), dev(v[:, :, lo:hi], dtype), state,
             api.AttentionShape(B, H, Sq, hi - lo, D, kvH), qmap, SegMap.make([lo], hi - lo), flags | CAUSAL, split, doc)
    lse = api.attention_lse(state[1], state[2]).cpu().numpy()
    assert api.device_status()[0] == 0
    w_out, w_m, w_l = oracle.attention_init((B, H, Sq, D), (B, H, Sq))
    oracle.attention_step(q, k, v, w_out, w_m, w_l, [Sk - Sq], [0], causal=True, kv_heads=kvH, doc_len=doc)
    oracle.attention_finalize(w_out, w_l)
    assert_close(state[0].cpu().numpy(), w_out, TOL[dtype], TOL[dtype], "out")
    assert_close(lse, w_m + np.log(w_l), TOL[dtype], TOL[dtype], "lse")


def test_key_split_leaves_rows_without_a_visible_key_alone():
    B, H, Sq, Sk, D = 1, 2, 200, 512, 64
    q, k, v = normal_inputs(6, B, H, H, Sq, Sk, D)
    state = [torch.full((B, H, Sq, D), 3.0, device="cuda"), torch.full((B, H, Sq), 0.5, device="cuda"),
             torch.full((B, H, Sq), 2.0, device="cuda")]
    for dtype in (torch.float16, torch.float32):
        step(dev(q, dtype), dev(k, dtype), dev(v, dtype), state, api.AttentionShape(B, H, Sq, Sk, D),
             SegMap.make([0], Sq), SegMap.make([1000], Sk), CAUSAL, 4)
    assert (state[0] == 3.0).all() and (state[1] == 0.5).all() and (state[2] == 2.0).all()


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("case", ["small", "large", "tiny_keys", "outlier_key", "growing_v", "zero_v_tiles", "shrinking_v"])
def test_fp32_step_holds_its_precision_over_the_range_of_fp32(D, case):
    # magnitudes that fp16 cannot hold have to come through the scaling of Q rows, keys and V tiles
    B, H, Sq, Sk = 1, 2, 140, 400
    q, k, v = normal_inputs(8, B, H, H, Sq, Sk, D)
    if case == "small":
        q, k, v = q * 2.0 ** 20, k * 2.0 ** -20, v * 2.0 ** -30
    elif case == "large":
        q, k, v = q * 2.0 ** -40, k * 2.0 ** 40, v * 2.0 ** 60
    elif case == "tiny_keys":
        k *= 2.0 ** -60
    elif case == "outlier_key":  # hides itself behind a hugely negative score
        q = np.abs(q)
        k[:, :, 37] = -1e9
    elif case == "growing_v":
        v *= 2.0 ** (np.arange(Sk, dtype=np.float32) // 64 * 9)[None, None, :, None]
    elif case == "shrinking_v":
        v *= 2.0 ** -(np.arange(Sk, dtype=np.float32) // 64 * 9)[None, None, :, None]
    else:
        v[:, :, :130] = 0.0
        v[:, :, 256:320] = 0.0
    q, k, v = (x.astype(np.float32) for x in (q, k, v))
    want, want_lse = oracle.cpu_attention(q, k, v, False, want_lse=True)
    state = poisoned(B, H, Sq, D)
    step(dev(q), dev(k), dev(v), state, api.AttentionShape(B, H, Sq, Sk, D), SegMap.make([0], Sq),
         SegMap.make([0], Sk), FRESH | FINALIZE)
    lse = api.attention_lse(state[1], state[2]).cpu().numpy()
    unit = float(np.abs(want).max())  # errors of a weighted sum of V scale with the largest V
    assert_close(state[0].cpu().numpy() / unit, want / unit, 1e-5, 1e-5, "out")
    assert_close(lse, want_lse, 1e-5, 1e-5, "lse")


def _in_64_bits(q, k, v, qpos, kpos, causal, doc):
    """(out, log-sum-exp) with one KV head per query head."""
    seen = (kpos[None, :] <= qpos[:, None]) | (not causal)
    if doc:
        seen = seen & (kpos[None, :] // doc == qpos[:, None] // doc)
    s = np.einsum("bhid,bhjd->bhij", q.astype(np.float64), k.astype(np.float64)) / np.sqrt(q.shape[-1])
    s = np.where(seen, s, -np.inf)
    m = s.max(-1, keepdims=True)
    p = np.exp(s - m)
    out = np.einsum("bhij,bhjd->bhid", p, v.astype(np.float64)) / p.sum(-1, keepdims=True)
    return out, (m + np.log(p.sum(-1, keepdims=True)))[..., 0]


def _wide_inputs(case, D):
    """Finite inputs whose parts differ by powers of two: (q, k, v, causal, doc_len, [(rows, columns)]).
    Every part of the output is held against its own largest value."""
    S, every = 500, slice(None)
    q, k, v = (x.astype(np.float64) for x in normal_inputs(21, 1, 2, 2, S, S, D))
    kind, n = case
    if kind in ("document", "ragged document"):  # inside a query block, on a key tile's edge or not
        at = 192 if kind == "document" else 230
        v[:, :, :at] *= 2.0 ** n
        return q, k, v, True, at, [(slice(0, at), every), (slice(at, 2 * at), every), (slice(2 * at, S), every)]
    if kind in ("future", "ragged future"):
        at = 192 if kind == "future" else 150
        v[:, :, at:] *= 2.0 ** n
        return q, k, v, True, 0, [(slice(0, at), every), (slice(at, S), every)]
    if kind == "column":
        v[..., 5] *= 2.0 ** n
        return q, k, v, False, 0, [(every, slice(0, 5)), (every, slice(5, 6)), (every, slice(6, D))]
    if kind == "element":  # in the first key tile; rows before it do not see it
        v[:, :, 10, 3] = 2.0 ** n
        return q, k, v, True, 0, [(slice(0, 10), every), (slice(10, S), slice(3, 4)), (slice(10, S), slice(4, D))]
    if kind == "key":  # visible, under a weight of e^-40
        q[..., 0], k[..., 0] = 4.0, 0.0
        v[:, :, 100] *= 2.0 ** n
        k[:, :, 100] = 0.0
        k[:, :, 100, 0] = -10.0 * np.sqrt(D)
        return q, k, v, False, 0, [(every, every)]
    if kind == "every other key":  # values 2^n larger under weights about 2^n smaller
        q[..., 0], k[..., 0] = 4.0, 0.0
        v[:, :, ::2] *= 2.0 ** n
        k[:, :, ::2, 0] = -n * np.log(2.0) / 4.0 * np.sqrt(D)
        return q, k, v, False, 0, [(every, every)]
    if kind == "small keys":
        v[:, :, 64:] *= 2.0 ** n
        v[:, :, 70:80] *= 2.0 ** -n
        return q, k, v, True, 0, [(slice(0, 64), every), (slice(64, S), every)]
    if kind in ("first tile", "last tile"):  # values 2^n larger under weights about 2^n smaller
        at = slice(0, 64) if kind == "first tile" else slice(448, S)
        v[:, :, at] *= 2.0 ** n
        q[..., 0], k[..., 0] = 4.0, 0.0
        k[:, :, at] *= 0.1
        k[:, :, at, 0] = -n * np.log(2.0) / 4.0 * np.sqrt(D)
        return q, k, v, False, 0, [(every, every)]
    if kind == "channel":  # one element of every Q row far larger, of every key far smaller
        q[..., 0] *= 2.0 ** n
        k[..., 0] *= 2.0 ** -n
        return q, k, v, False, 0, [(every, every)]
    if kind == "channels apart":  # large elements that do not meet, in some rows and keys
        q[:, :, ::3, 0] = 2.0 ** n
        q[..., 1] = 0.0
        k[..., 0] = 0.0
        k[:, :, 130::7, 1] = 2.0 ** n
        return q, k, v, True, 0, [(every, every)]
    if kind == "V":
        return q, k, v * 2.0 ** n, False, 0, [(every, every)]
    if kind == "Q against K":
        return q * 2.0 ** n, k * 2.0 ** -n, v, False, 0, [(every, every)]
    raise ValueError(kind)


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("split", [1, 3])
@pytest.mark.parametrize("case", [("document", 20), ("document", 34), ("document", 100), ("document", -40), ("future", 40),
                                  ("first tile", 20), ("first tile", 34), ("last tile", 20), ("last tile", 34), ("V", -70), ("V", -90), ("V", -104), ("V", 120),
                                  ("ragged document", 12), ("ragged document", 34), ("ragged document", 100), ("ragged document", -100),
                                  ("ragged future", 40), ("column", 20), ("column", 30), ("column", 100), ("element", 30),
                                  ("element", 100), ("key", 24), ("key", 34), ("every other key", 20), ("every other key", 30),
                                  ("small keys", -40), ("Q against K", 80), ("Q against K", -80), ("channel", 24), ("channel", 40), ("channels apart", 26), ("Q against K", 104), ("Q against K", -96)], ids=str)
def test_fp32_step_holds_the_precision_of_every_part_of_the_output(D, split, case):
    # Values that a row cannot see, or sees under a negligible weight, must not cost it bits, nor may
    # one column cost another. Against 64 bits; 1e-5 of the part's largest value, the fp32 tolerance.
    q, k, v, causal, doc, parts = _wide_inputs(case, D)
    q, k, v = (x.astype(np.float32) for x in (q, k, v))
    B, H, S, _ = q.shape
    want, want_lse = _in_64_bits(q, k, v, np.arange(S), np.arange(S), causal, doc)
    state = poisoned(B, H, S, D)
    step(dev(q), dev(k), dev(v), state, api.AttentionShape(B, H, S, S, D), SegMap.make([0], S), SegMap.make([0], S),
         FRESH | FINALIZE | (CAUSAL if causal else 0), split, doc)
    got, lse = state[0].cpu().numpy(), api.attention_lse(state[1], state[2]).cpu().numpy()
    assert_close(lse, want_lse, 1e-5, 1e-5, "lse")
    for rows, cols in parts:
        unit = np.abs(want[:, :, rows, cols]).max()
        assert_close(got[:, :, rows, cols] / unit, want[:, :, rows, cols] / unit, 1e-5, 0.0, f"rows {rows} columns {cols}")


def test_fp32_step_passes_on_nan_and_infinity_of_visible_values_only():
    B, H, S, D = 1, 1, 200, 64
    q, k, v = normal_inputs(9, B, H, H, S, S, D)
    v[0, 0, 150, 7] = np.inf
    k[0, 0, 190, 3] = np.nan
    state = poisoned(B, H, S, D)
    step(dev(q), dev(k), dev(v), state, api.AttentionShape(B, H, S, S, D), SegMap.make([0], S),
         SegMap.make([0], S), FRESH | FINALIZE | CAUSAL)
    got = state[0].cpu().numpy()[0, 0]
    want = oracle.cpu_attention(q[:, :, :128], k[:, :, :128], v[:, :, :128], True)[0, 0]
    assert_close(got[:128], want, 1e-5, 1e-5, "rows whose key tiles are finite")
    assert not np.isfinite(got[160, 7]) and np.isnan(got[195]).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("D", [32, 128, 256])
@pytest.mark.parametrize("shape", [  # B, H, kvH, Sk: both forms, single stages, ragged ends, several head batches
    (1, 1, 1, 1), (1, 8, 8, 64), (1, 40, 2, 65), (3, 6, 2, 1023), (1, 4, 4, 30011), (2, 34, 1, 9000), (40, 4, 4, 190)])
def test_decode_forms_match_the_oracle_with_and_without_a_state(dtype, D, shape):
    B, H, kvH, Sk = shape
    q, k, v = (round_to(x, dtype) for x in normal_inputs(11, B, H, kvH, 1, Sk, D))
    want, want_lse = oracle.cpu_attention(q, k, v, False, kv_heads=kvH, want_lse=True, threads=8)
    s = api.AttentionShape(B, H, 1, Sk, D, kvH)
    dq, dk, dv = dev(q, dtype), dev(k, dtype), dev(v, dtype)
    out, m, l = poisoned(B, H, 1, D)
    api.launch_attention_init(out, m, l, s)
    # the least workspace that has always been enough (one partial per row) and the full one
    one = B * H * (D + 2) * 4
    spaces = [None, torch.empty(lib().ra_decode_workspace_bytes(C.byref(s.c())), dtype=torch.uint8, device="cuda")]
    if Sk == 1:
        spaces.append(torch.empty(one, dtype=torch.uint8, device="cuda"))
    for ws in spaces:  # folding the same keys again leaves the normalised result as it is
        api.launch_attention_decode_step(dq, dk, dv, out, m, l, s, 0, 0, False, workspace=ws)
    lse = api.attention_lse(m, l).cpu().numpy() - np.log(len(spaces))
    api.launch_attention_finalize(out, l, s)
    assert_close(out.cpu().numpy(), want, TOL[dtype], TOL[dtype], "out")
    assert_close(lse, want_lse, TOL[dtype], TOL[dtype], "lse")


@pytest.mark.parametrize("dtype,D", [(torch.float32, 1), (torch.float16, 3), (torch.bfloat16, 8), (torch.float16, 128)])
def test_cache_append_of_any_row_size_and_alignment(dtype, D):
    B, kvH, s_max = 2, 3, 5
    cache = api.DeviceKVCache(B, kvH, s_max, D, dtype)
    flat = torch.randn(2 * s_max * B * kvH * D + 1, device="cuda").to(dtype)[1:]  # not 16-byte aligned
    rows = flat.view(2, s_max, B, kvH, 1, D)
    for t in range(s_max):
        cache.append(rows[0, t], rows[1, t])
    assert torch.equal(cache.k_view(), rows[0, :, :, :, 0].permute(1, 2, 0, 3))
    assert torch.equal(cache.v_view(), rows[1, :, :, :, 0].permute(1, 2, 0, 3))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("heads,kv_heads,rows,D", [(8, 8, 20000, 128), (16, 2, 6000, 128), (8, 8, 300, 64), (4, 4, 9000, 256)])
def test_decode_and_key_split_replay_from_a_captured_graph(dtype, heads, kv_heads, rows, D):
    # the fold of the decode partials is a programmatic dependent launch, the key split a cluster launch
    g = torch.Generator(device="cuda").manual_seed(3)
    k = torch.randn((1, kv_heads, rows, D), generator=g, device="cuda").to(dtype)
    v = torch.randn((1, kv_heads, rows, D), generator=g, device="cuda").to(dtype)
    cache = api.DeviceKVCache(1, kv_heads, rows + 1, D, dtype)
    cache.copy_prefill(k, v, rows)
    q1 = torch.randn((1, heads, 1, D), generator=g, device="cuda").to(dtype)
    qn = torch.randn((1, heads, 100, D), generator=g, device="cuda").to(dtype)
    o1 = torch.empty((1, heads, 1, D), device="cuda")
    on, m, l = poisoned(1, heads, 100, D)
    shape = api.AttentionShape(1, heads, 100, rows, D, kv_heads)
    maps = SegMap.make([rows - 100], 100), SegMap.make([0], rows)

    def both():
        api.run_local_decode_step(q1, cache, heads, rows - 1, 0, True, o1)
        api.attention_step_ex(qn, k, v, on, m, l, shape, *maps, causal=True, fresh=True, finalize=True)

    both()  # workspaces are made here
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        both()
    q1.copy_(torch.randn(q1.shape, generator=g, device="cuda").to(dtype))
    qn.copy_(torch.randn(qn.shape, generator=g, device="cuda").to(dtype))
    graph.replay()
    torch.cuda.synchronize()
    got1, gotn = o1.clone(), on.clone()
    both()
    torch.cuda.synchronize()
    assert torch.equal(got1, o1) and torch.equal(gotn, on) and api.device_status()[0] == 0


def test_cache_append_on_a_stream_of_its_own_and_from_a_captured_graph():
    cache = api.DeviceKVCache(2, 3, 4, 64, torch.float16)
    rows = torch.randn(4, 2, 2, 3, 1, 64, device="cuda").half()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        cache.append(rows[0, 0], rows[0, 1])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cache.append(rows[1, 0], rows[1, 1])
    rows[1].copy_(rows[2])
    graph.replay()
    torch.cuda.synchronize()
    for i, src in enumerate((0, 2)):
        assert torch.equal(cache.k_view()[:, :, i], rows[src, 0, :, :, 0]) and torch.equal(cache.v_view()[:, :, i], rows[src, 1, :, :, 0])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_decode_calls_in_a_row_fold_their_own_partials(dtype):
    # The fold starts while the split kernel runs and all calls share a workspace: what it reads has to
    # be this call's partials and this call's state, not what it finds there when it starts.
    H, Sk, D, calls = 8, 6000, 128, 12
    shape = api.AttentionShape(1, H, 1, Sk, D, H)
    g = torch.Generator(device="cuda").manual_seed(4)
    k, v, q = (torch.randn((calls, 1, H, n, D), generator=g, device="cuda").to(dtype) for n in (Sk, Sk, 1))
    ws = torch.full((lib().ra_decode_workspace_bytes(C.byref(shape.c())) // 4,), float("nan"), device="cuda")
    alone, chain = [], poisoned(1, H, 1, D)
    for i in range(calls):
        state = poisoned(1, H, 1, D)
        api.launch_attention_init(*state, shape)
        api.launch_attention_decode_step(q[i], k[i], v[i], *state, shape, 0, 0, False, workspace=ws)
        torch.cuda.synchronize()
        ws.fill_(float("nan"))
        alone.append(state)
    api.launch_attention_init(*chain, shape)
    row = [poisoned(1, H, 1, D) for _ in range(calls)]
    for state in row:
        api.launch_attention_init(*state, shape)
    torch.cuda.synchronize()
    for i in range(calls):  # nothing waits between these
        api.launch_attention_decode_step(q[i], k[i], v[i], *row[i], shape, 0, 0, False, workspace=ws)
        api.launch_attention_decode_step(q[i], k[i], v[i], *chain, shape, 0, 0, False, workspace=ws)
    torch.cuda.synchronize()
    for a, b in zip(alone, row):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
    # the chained state is the merge of the single ones
    m = torch.stack([s[1] for s in alone]).double()
    w = (m - m.max(0).values).exp()
    l = (torch.stack([s[2] for s in alone]).double() * w).sum(0)
    o = (torch.stack([s[0] for s in alone]).double() * w[..., None]).sum(0) / l[..., None]
    api.launch_attention_finalize(chain[0], chain[2], shape)
    assert_close(chain[0].cpu().numpy(), o.cpu().numpy(), 1e-5, 1e-5, "chained state")


@pytest.mark.parametrize("dtype,D", [(torch.float32, 64), (torch.float32, 128), (torch.float16, 64), (torch.float16, 128)])
@pytest.mark.parametrize("split", [1, 3])
@pytest.mark.parametrize("finalize", [False, True])
def test_rows_whose_wait_ran_out_keep_their_state(dtype, D, split, finalize):
    # The producer stops after so many ring items that with three blocks to a query block the first one or
    # two finish their share and the last cannot: none of the rows may get a part of the sum.
    L, S = lib(), 1024
    q, k, v = (dev(x, dtype) for x in normal_inputs(13, 1, 2, 2, S, S, D))
    state = [torch.full((1, 2, S, D), 3.0, device="cuda"), torch.full((1, 2, S), 0.5, device="cuda"),
             torch.full((1, 2, S), 2.0, device="cuda")]
    assert api.device_status()[0] == 0
    L.ra_debug_set_wait_limit_ns(5_000_000)
    L.ra_debug_stall_producer_after(10 if dtype == torch.float32 else 4)
    try:
        step(q, k, v, state, api.AttentionShape(1, 2, S, S, D), SegMap.make([0], S), SegMap.make([0], S),
             FINALIZE if finalize else 0, split)
        torch.cuda.synchronize()
    finally:
        L.ra_debug_stall_producer_after(-1)
        L.ra_debug_set_wait_limit_ns(0)
    status = api.device_status()
    assert status[0] == 5 and status[1] > 0, status
    assert (state[0] == 3.0).all() and (state[1] == 0.5).all() and (state[2] == 2.0).all()


@pytest.mark.parametrize("dtype,D", [(torch.float32, 64), (torch.float32, 128), (torch.float16, 32), (torch.float16, 64),
                                     (torch.bfloat16, 128), (torch.float16, 256)])
@pytest.mark.parametrize("split,pair", [(0, False), (1, False), (3, False), (1, True)])
@pytest.mark.parametrize("fresh", [False, True])
def test_steps_behind_one_that_gave_up_leave_their_state(dtype, D, split, pair, fresh):
    # One block waits 20 ms for keys that never come. The blocks of the next step start beside it, before there is
    # anything to see in the status word; neither they nor those of the one after may touch their state.
    if pair and (D not in (128, 256) or dtype == torch.float32):
        pytest.skip("the pair form is built for head_dim 128 and 256")
    L, H, rows, Sk = lib(), 4, 700, 1000
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(1, H, s, D, generator=g, device="cuda").to(dtype) for s in (rows, Sk, Sk))
    first = [torch.full(s, 0.5, device="cuda") for s in ((1, 1, 128, D), (1, 1, 128), (1, 1, 128))]
    states = [[torch.full(s, 3.0, device="cuda") for s in ((1, H, rows, D), (1, H, rows), (1, H, rows))] for _ in range(2)]
    q0, k0, v0 = (x[:, :1, :n].contiguous() for x, n in ((q, 128), (k, Sk), (v, Sk)))
    assert api.device_status()[0] == 0
    L.ra_debug_set_wait_limit_ns(20_000_000)
    L.ra_debug_stall_producer_after(2)
    try:
        step(q0, k0, v0, first, api.AttentionShape(1, 1, 128, Sk, D), SegMap.make([0], 128), SegMap.make([0], Sk), 0, 1)
        L.ra_debug_stall_producer_after(-1)
        for state in states:
            api.attention_step_ex(q, k, v, *state, api.AttentionShape(1, H, rows, Sk, D), SegMap.make([500], rows),
                                  SegMap.make([600], Sk), causal=True, fresh=fresh, finalize=True, key_split=split, cta_pair=pair)
        torch.cuda.synchronize()
    finally:
        L.ra_debug_stall_producer_after(-1)
        L.ra_debug_set_wait_limit_ns(0)
    status = api.device_status()
    assert status[0] == 5 and status[1] > 0, status
    for state in states:
        assert all((t == 3.0).all() for t in state)


@pytest.mark.parametrize("which", [0, 1, 2])
def test_half_flash_call_with_one_unaligned_source(which):
    B, H, kvH, S, D = 1, 4, 2, 300, 64
    x = [dev(t) for t in normal_inputs(14, B, H, kvH, S, S, D)]
    shape, want, got = api.AttentionShape(B, H, S, S, D, kvH), *(torch.empty(B, H, S, D, device="cuda") for _ in range(2))
    api.launch_flash_attention_fp16(*x, want, shape, True)
    flat = torch.empty(x[which].numel() + 1, device="cuda")[1:]
    x[which] = flat.copy_(x[which].flatten()).view(x[which].shape)
    api.launch_flash_attention_fp16(*x, got, shape, True)
    assert torch.equal(got, want)


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("split", [1, 2])
@pytest.mark.parametrize("case", ["plain", "growing scores", "documents", "marked tiles", "growing v"])
def test_fp32_step_over_many_key_tiles_into_a_state(D, split, case):
    # 47 key tiles, 36 of them in one step (18 to a block when two share them): the ring wraps several times, the
    # 16 tile exponents and 8 sets of key exponents are reused, and the second step folds into the first's state
    Sq, Sk, cut, doc = 300, 2950, 700, 0
    q, k, v = (x.astype(np.float64) for x in normal_inputs(17, 1, 2, 2, Sq, Sk, D))
    if case == "growing scores":  # about 1.5 in the exponent from one key tile to the next
        q[..., 0], k[..., 0] = 4.0, np.arange(Sk) / 64.0 * 1.5 / 4.0 * np.sqrt(D)
    elif case == "documents":
        doc = 1100
    elif case == "marked tiles":  # single keys and columns, a channel of some keys
        v[:, :, 100::450] *= 2.0 ** 20
        v[:, :, 1300:1400, 7] *= 2.0 ** 30
        q[..., 1], k[..., 1] = q[..., 1] * 2.0 ** 16, k[..., 1] * 2.0 ** -16
        k[:, :, 2000:2100, 2] = 0.0
        k[:, :, 2050, 2] = -(2.0 ** 16)
        q[..., 2] = np.abs(q[..., 2])
    elif case == "growing v":
        v *= 2.0 ** (np.arange(Sk) // 64)[None, None, :, None]
    q, k, v = (x.astype(np.float32) for x in (q, k, v))
    want, want_lse = _in_64_bits(q, k, v, np.arange(Sq) + Sk - Sq, np.arange(Sk), True, doc)
    state = poisoned(1, 2, Sq, D)
    for lo, hi, flags in ((0, cut, FRESH), (cut, Sk, FINALIZE)):
        step(dev(q), dev(k[:, :, lo:hi]), dev(v[:, :, lo:hi]), state, api.AttentionShape(1, 2, Sq, hi - lo, D),
             SegMap.make([Sk - Sq], Sq), SegMap.make([lo], hi - lo), flags | CAUSAL, split, doc)
    lse = api.attention_lse(state[1], state[2]).cpu().numpy()
    assert api.device_status()[0] == 0
    # fp32 scores of up to 70 (growing scores) carry 4e-6 each: half an ulp of the score before scaling
    assert_close(lse, want_lse, 1e-5, 1e-5, "lse")
    unit = np.abs(want).max()
    assert_close(state[0].cpu().numpy() / unit, want / unit, 2e-5, 0.0, "out")


@pytest.mark.parametrize("dtype,D", [(torch.float16, 64), (torch.float16, 128), (torch.bfloat16, 256), (torch.float32, 64),
                                     (torch.float32, 128)])
@pytest.mark.parametrize("split", [1, 3])
def test_document_mask_and_moving_reference_in_both_forms(dtype, D, split):
    # scores that climb by about 24 in the exponent per 128 keys, and documents that begin inside tiles
    S, Sq, doc = 1024, 256, 600
    rng = np.random.default_rng(12)
    q, k = rng.standard_normal((1, 2, Sq, D)) * 0.3, rng.standard_normal((1, 2, S, D)) * 0.3
    q[..., 0] = 4.0
    k[0, 0, :, 0] = np.arange(S) / 128.0 * 17.0 * np.sqrt(D) / 4.0
    k[0, 1, :, 0] = -k[0, 0, :, 0]
    v = rng.standard_normal((1, 2, S, D))
    q, k, v = (round_to(x.astype(np.float32), dtype) for x in (q, k, v))
    want, want_lse = _in_64_bits(q, k, v, np.arange(Sq) + S - Sq, np.arange(S), True, doc)
    state = poisoned(1, 2, Sq, D)
    step(dev(q, dtype), dev(k, dtype), dev(v, dtype), state, api.AttentionShape(1, 2, Sq, S, D), SegMap.make([S - Sq], Sq),
         SegMap.make([0], S), FRESH | FINALIZE | CAUSAL, split, doc)
    lse = api.attention_lse(state[1], state[2]).cpu().numpy()
    # fp32: raw scores of about 1000, one ulp of which is 1.5e-5 in the exponent after scaling
    tol = 1e-4 if dtype == torch.float32 else TOL[dtype]
    assert_close(state[0].cpu().numpy(), want, tol, tol, "out")
    assert_close(lse, want_lse, tol, tol, "lse")


@pytest.mark.parametrize("dtype,H,kvH,Sk,D", [(torch.float16, 32, 2, 300, 256), (torch.float16, 8, 8, 20000, 128),
                                              (torch.float32, 16, 2, 6000, 256), (torch.float32, 8, 8, 500, 32),
                                              (torch.bfloat16, 48, 1, 9000, 64)])
def test_decode_into_a_state_and_a_workspace_aligned_to_four_bytes(dtype, H, kvH, Sk, D):
    # every form (cluster, equal shares, fixed splits) writes and folds four columns at a time where it can
    q, k, v = (round_to(x, dtype) for x in normal_inputs(15, 1, H, kvH, 1, Sk, D))
    want, want_lse = oracle.cpu_attention(q, k, v, False, kv_heads=kvH, want_lse=True, threads=8)
    s = api.AttentionShape(1, H, 1, Sk, D, kvH)
    out = torch.full((H * D + 1,), float("nan"), device="cuda")[1:].view(1, H, 1, D)
    m, l = (torch.full((1, H, 1), float("nan"), device="cuda") for _ in range(2))
    ws = torch.full((lib().ra_decode_workspace_bytes(C.byref(s.c())) // 4 + 1,), float("nan"), device="cuda")[1:]
    api.launch_attention_init(out, m, l, s)
    for _ in range(2):
        api.launch_attention_decode_step(dev(q, dtype), dev(k, dtype), dev(v, dtype), out, m, l, s, 0, 0, False, workspace=ws)
    lse = api.attention_lse(m, l).cpu().numpy() - np.log(2.0)
    api.launch_attention_finalize(out, l, s)
    assert_close(out.cpu().numpy(), want, TOL[dtype], TOL[dtype], "out")
    assert_close(lse, want_lse, TOL[dtype], TOL[dtype], "lse")


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("split", [1, 2])
def test_marked_tiles_in_a_cache_with_segments_strides_and_grouped_heads(D, split):
    # plain scores read K from memory by segment, batch row, KV head and row stride
    B, H, kvH, Lq, Lk, stride, room = 2, 4, 2, 70, 150, 3, 400
    rng = np.random.default_rng(23)
    q = rng.standard_normal((B, H, 2 * Lq, D))
    k, v = (rng.standard_normal((B, kvH, room, D)) for _ in range(2))
    q[..., 0] *= 2.0 ** 20
    k[..., 0] *= 2.0 ** -20
    k[:, 1, 20:140, 3] = 0.0
    k[:, 1, 30, 3] = -(2.0 ** 12)  # one KV head has larger keys too
    q[..., 3] = np.abs(q[..., 3])
    v[:, :, 40] *= 2.0 ** 15
    q, k, v = (x.astype(np.float32) for x in (q, k, v))
    qmap, kmap = SegMap.make([300, 2000], Lq), SegMap.make([0, 1500], Lk)
    qpos = np.concatenate([b + np.arange(Lq) * stride for b in (300, 2000)])
    kpos = np.concatenate([b + np.arange(Lk) * stride for b in (0, 1500)])
    heads = [h % kvH for h in range(H)]
    want, want_lse = _in_64_bits(q, k[:, heads, :2 * Lk], v[:, heads, :2 * Lk], qpos, kpos, True, 0)
    out, m, l = poisoned(B, H, 2 * Lq, D)
    shape = api.AttentionShape(B, H, 2 * Lq, 2 * Lk, D, kvH)
    api.attention_step_ex(dev(q), dev(k), dev(v), out, m, l, shape, qmap, kmap, pos_stride=stride, causal=True, fresh=True,
                          finalize=True, kv_row_stride=room, key_split=split)
    lse = api.attention_lse(m, l).cpu().numpy()
    assert api.device_status()[0] == 0
    assert_close(lse, want_lse, 1e-5, 1e-5, "lse")
    unit = np.abs(want).max()
    assert_close(out.cpu().numpy() / unit, want / unit, 1e-5, 0.0, "out")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("heads,rows,qbases,kbases,seg_k,stride", [
    (36, 1000, [0], [0], 1000, 1),                    # eight tiles, the last one short
    (28, 1100, [0], [0], 1100, 1),                    # nine: the middle one alone
    (16, 1021, [1021, 6126], [1021, 6126], 1021, 1),  # a zig-zag rank's own shard
    (48, 600, [200], [0], 800, 1),                    # rows behind a cache
    (40, 700, [0], [350], 700, 1),                    # the first tiles see no key
    (32, 1000, [1], [0], 1000, 2),                    # striped
])
def test_light_and_heavy_query_tiles_share_a_block(dtype, D, heads, rows, qbases, kbases, seg_k, stride):
    # causal calls of one wave pair a head's tiles light with heavy; asking for an unsplit call gives
    # neighbours. Every row folds the same tiles in the same order, so the results are the same bits.
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    Sq, Sk, kvH = rows * len(qbases), seg_k * len(kbases), heads // 2
    q, k, v = (torch.randn(1, h, s, D, generator=g, device="cuda").to(dtype) for h, s in ((heads, Sq), (kvH, Sk), (kvH, Sk)))
    shape = api.AttentionShape(1, heads, Sq, Sk, D, kvH)
    results = []
    for split in (0, 1):
        state = poisoned(1, heads, Sq, D)
        for i, qi in enumerate((q, -q)):
            api.attention_step_ex(qi, k, v, *state, shape, SegMap.make(qbases, rows), SegMap.make(kbases, seg_k),
                                  pos_stride=stride, causal=True, fresh=i == 0, finalize=i == 1, key_split=split)
            assert lib().ra_debug_step_form() == (1 if split else 1 | 16)
        results.append(state)
    torch.cuda.synchronize()
    assert api.device_status()[0] == 0
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("heads,rows,qbases,kbases,seg_k,stride", [
    (28, 1100, [0], [0], 1100, 1), (16, 1021, [1021, 6126], [1021, 6126], 1021, 1), (32, 1000, [1], [0], 1000, 2)])
def test_folded_calls_match_64_bits(dtype, D, heads, rows, qbases, kbases, seg_k, stride):
    kvH = heads // 2
    Sq, Sk = rows * len(qbases), seg_k * len(kbases)
    q, k, v = (round_to(x, dtype) for x in normal_inputs(23, 1, heads, kvH, Sq, Sk, D))
    state = poisoned(1, heads, Sq, D)
    api.attention_step_ex(dev(q, dtype), dev(k, dtype), dev(v, dtype), *state, api.AttentionShape(1, heads, Sq, Sk, D, kvH),
                          SegMap.make(qbases, rows), SegMap.make(kbases, seg_k), pos_stride=stride, causal=True, fresh=True,
                          finalize=True)
    assert lib().ra_debug_step_form() == 1 | 16
    lse = api.attention_lse(state[1], state[2]).cpu().numpy()
    assert api.device_status()[0] == 0
    qpos, kpos = (np.concatenate([b + stride * np.arange(n) for b in bases]) for bases, n in ((qbases, rows), (kbases, seg_k)))
    some = [0, heads // 2 + 1]  # (a head of either half; query head h reads KV head h % kvH)
    kv = [h % kvH for h in some]
    want, want_lse = _in_64_bits(q[:, some], k[:, kv], v[:, kv], qpos, kpos, True, 0)
    assert_close(state[0].cpu().numpy()[:, some], want, TOL[dtype], TOL[dtype], "out")
    assert_close(lse[:, some], want_lse, 1e-5, 1e-5, "lse")


@pytest.mark.parametrize("dtype,D", [(torch.float16, 32), (torch.float16, 64), (torch.bfloat16, 128), (torch.float16, 256),
                                     (torch.float32, 32), (torch.float32, 64), (torch.float32, 128)])
@pytest.mark.parametrize("split,pair", [(1, False), (3, False), (1, True)])
@pytest.mark.parametrize("fresh,finalize", [(False, False), (False, True), (True, False), (True, True)])
def test_blocks_without_keys(dtype, D, split, pair, fresh, finalize):
    # the second segment's rows see every key, the first one's none: those keep their state bit for bit, or it is
    # written empty, or divided by l (rows that never saw a key give zeros)
    if pair and D not in (128, 256):
        pytest.skip("the pair form is built for head_dim 128 and 256")
    B, H, kvH, rows, Sk = 2, 4, 2, 333, 200
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(B, h, s, D, generator=g, device="cuda").to(dtype) for h, s in ((H, 2 * rows), (kvH, Sk), (kvH, Sk)))
    out, m, l = (torch.rand(*s, generator=g, device="cuda") + 0.5 for s in ((B, H, 2 * rows, D), (B, H, 2 * rows), (B, H, 2 * rows)))
    m[:, :, 5::7] = float("-inf")
    l[:, :, 5::7] = 0
    out[:, :, 5::7] = 0
    before = [t.clone() for t in (out, m, l)]
    api.attention_step_ex(q, k, v, out, m, l, api.AttentionShape(B, H, 2 * rows, Sk, D, kvH), SegMap.make([0, 1000], rows),
                          SegMap.make([500], Sk), causal=True, fresh=fresh, finalize=finalize, key_split=split, cta_pair=pair)
    torch.cuda.synchronize()
    assert api.device_status()[0] == 0
    o, mm, ll = (t[:, :, :rows] for t in (out, m, l))
    wo, wm, wl = (t[:, :, :rows] for t in before)
    if fresh:
        assert (o == 0).all() and (mm == float("-inf")).all() and (ll == 0).all()
    else:
        assert torch.equal(mm, wm) and torch.equal(ll, wl)
        if finalize:
            inv = torch.where(wl > 0, 1 / wl, torch.zeros_like(wl))[..., None]
            # a product of two roundings on either side
            assert torch.allclose(o, wo * inv, rtol=3e-7, atol=0)
        else:
            assert torch.equal(o, wo)
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("fresh,finalize", [(False, True), (True, False), (True, True)])
def test_light_query_tiles_without_keys(dtype, D, fresh, finalize):
    # Keys from position 350 on: two light tiles of a head see none, their blocks' heavy ones do. Such a tile's rows
    # are staged where the copy of its Q lands, so many calls with the state set anew before each, some right behind
    # other work and some on an idle GPU.
    H, kvH, rows = 40, 20, 700
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(1, h, rows, D, generator=g, device="cuda").to(dtype) for h in (H, kvH, kvH))
    before = [torch.rand(*s, generator=g, device="cuda") + 0.5 for s in ((1, H, rows, D), (1, H, rows), (1, H, rows))]
    shape = api.AttentionShape(1, H, rows, rows, D, kvH)

    def call(state, split):
        for t, b in zip(state, before):
            t.copy_(b)
        api.attention_step_ex(q, k, v, *state, shape, SegMap.make([0], rows), SegMap.make([350], rows), causal=True,
                              fresh=fresh, finalize=finalize, key_split=split)
        return state

    want = call([torch.empty_like(t) for t in before], 1)
    hidden = torch.zeros_like(before[0][:, :, :350])
    if not fresh:  # (the product of two roundings on either side)
        hidden = before[0][:, :, :350] / before[2][:, :, :350, None]
    assert torch.allclose(want[0][:, :, :350], hidden, rtol=3e-7, atol=0)
    state = [torch.empty_like(t) for t in before]
    for i in range(60):
        call(state, 0)
        assert lib().ra_debug_step_form() == 1 | 16
        if i % 3 == 0:
            torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(state, want)), i
    assert api.device_status()[0] == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64, 128, 256])
@pytest.mark.parametrize("form", ["shape", "unsplit", "split", "smem", "pair"])
@pytest.mark.parametrize("rows", [1, 150, 300])
def test_rows_behind_a_ragged_segment_change_nothing(dtype, D, form, rows):
    # The last tile of the first segment holds rows of the second, and they are worked along. Whatever stands
    # there (NaN, infinities, large values, zeros), the first segment's rows are right, for finite values the same bits.
    if form == "pair" and D not in (128, 256):
        pytest.skip("the pair form is built for head_dim 128 and 256")
    H, kvH, Sk = 4, 2, 700
    q, k, v = (round_to(x, dtype) for x in normal_inputs(29 + D, 1, H, kvH, 2 * rows, Sk, D))
    dk, dv = dev(k, dtype), dev(v, dtype)
    shape, qmap, kmap = api.AttentionShape(1, H, 2 * rows, Sk, D, kvH), SegMap.make([Sk - rows, Sk], rows), SegMap.make([0], Sk)
    want, want_lse = _in_64_bits(q[:, :, :rows], k[:, [0, 1, 0, 1]], v[:, [0, 1, 0, 1]], np.arange(rows) + Sk - rows,
                                 np.arange(Sk), True, 0)
    got = []
    for fill in (None, 0.0, 3e4, float("inf"), float("nan")):
        x = q.copy()
        if fill is not None:
            x[:, :, rows:] = fill
        state = poisoned(1, H, 2 * rows, D)
        api.attention_step_ex(dev(x, dtype), dk, dv, *state, shape, qmap, kmap, causal=True, fresh=True, finalize=True,
                              key_split={"unsplit": 1, "split": 3}.get(form, 0), p_in_smem=form == "smem", cta_pair=form == "pair")
        lse = api.attention_lse(state[1], state[2])
        got.append((state[0][:, :, :rows].cpu().numpy(), lse[:, :, :rows].cpu().numpy()))
    assert api.device_status()[0] == 0
    for out, lse in got:
        assert_close(out, want, TOL[dtype], TOL[dtype], "out")
        assert_close(lse, want_lse, 1e-5, 1e-5, "lse")
    # (what is not finite takes its warp through the path that sets reference points anew, which may round P anew)
    for out, lse in got[1:3]:
        assert np.array_equal(out, got[0][0]) and np.array_equal(lse, got[0][1])
