"""Decode calls with more than two query heads to a KV head on caches that the tensor-core kernel does not take (fp32; 16-bit
with head_dim 32), against attention in 64 bits: stage edges, ragged groups of heads, both ways of dealing the rows."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from ring_attention_b200 import api
from util import normal_inputs, round_to

pytestmark = pytest.mark.gpu


def want64(q, k, v, kvH, blocks=1):
    """out and the bound of its error: scores of D products summed as 4 or 8 in a lane and log2 over lanes, one
    exponential (2^-22), and up to a quarter of a block's rows added one after another by a lane, in units of 2^-24."""
    q, k, v = (torch.from_numpy(x.astype(np.float64)) for x in (q, k, v))
    B, H, _, D = q.shape
    of = torch.arange(H) % kvH
    s = (q @ k[:, of].transpose(-1, -2)) / D ** 0.5
    size = ((q.abs() @ k[:, of].abs().nan_to_num(0, 0, 0).transpose(-1, -2)) / D ** 0.5).max().item()
    out = torch.softmax(s, -1) @ v[:, of]
    eps = 2.0 ** -24
    tol = (2 * (16 * eps * size + 2.0 ** -22) + 2 * (k.shape[2] / blocks / 4 + 64 + blocks) * eps) * v.abs().max().item()
    return out.numpy(), tol


@pytest.mark.parametrize("dtype,D", [(torch.float32, 32), (torch.float32, 64), (torch.float32, 128), (torch.float32, 256),
                                     (torch.float16, 32), (torch.bfloat16, 32)])
@pytest.mark.parametrize("B,H,kvH,Sk", [
    (1, 4, 1, 1), (2, 8, 1, 7), (1, 8, 2, 33), (1, 24, 3, 129), (2, 5, 1, 16), (1, 11, 3, 127), (1, 12, 4, 300),
    (1, 9, 1, 257), (1, 20, 1, 100), (1, 8, 1, 3001), (3, 16, 4, 2999), (64, 32, 4, 70)])
def test_group_decode_against_64_bits(dtype, D, B, H, kvH, Sk):
    q, k, v = normal_inputs(31, B, H, kvH, 1, Sk, D)
    q, k, v = (round_to(x, dtype) for x in (q, k, v)) if dtype != torch.float32 else (q, k, v)
    if Sk > 20:  # a key that no head sees (weight 0 whatever its value row)
        q, k = np.abs(q) + (q == 0), k.copy()
        k[:, :, Sk // 2] = -np.inf
    want, tol = want64(q, k, v, kvH)
    dq, dk, dv = (torch.from_numpy(np.ascontiguousarray(x)).cuda().to(dtype) for x in (q, k, v))
    shape = api.AttentionShape(B, H, 1, Sk, D, kvH)
    need = int(api.lib().ra_decode_workspace_bytes(shape.c()))
    for workspace in (None, torch.full((need // 4,), float("nan"), device="cuda")):
        out = torch.full((B, H, 1, D), float("nan"), device="cuda")
        m, l = torch.empty((B, H, 1), device="cuda"), torch.empty((B, H, 1), device="cuda")
        api.launch_attention_init(out, m, l, shape)
        api.launch_attention_decode_step(dq, dk, dv, out, m, l, shape, 0, 0, False, workspace=workspace)
        api.launch_attention_finalize(out, l, shape)
        assert np.abs(out.cpu().numpy() - want).max() <= tol


def test_group_decode_first_called_while_captured():
    """The library's own room for partials cannot grow while a stream is captured: the call is recorded all the same."""
    B, H, kvH, Sk, D = 2, 64, 8, 20011, 256
    q, k, v = normal_inputs(5, B, H, kvH, 1, Sk, D)
    want, tol = want64(q, k, v, kvH)
    dq, dk, dv = (torch.from_numpy(x).cuda() for x in (q, k, v))
    shape = api.AttentionShape(B, H, 1, Sk, D, kvH)
    out = torch.zeros((B, H, 1, D), device="cuda")
    m, l = torch.empty((B, H, 1), device="cuda"), torch.empty((B, H, 1), device="cuda")
    api.launch_attention_init(out, m, l, shape)
    api.launch_attention_finalize(out, l, shape)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        api.launch_attention_init(out, m, l, shape)
        api.launch_attention_decode_step(dq, dk, dv, out, m, l, shape, 0, 0, False)
        api.launch_attention_finalize(out, l, shape)
    graph.replay()
    torch.cuda.synchronize()
    assert np.abs(out.cpu().numpy() - want).max() <= tol


@pytest.mark.parametrize("dtype,B,H,kvH,Sk,D,blocks,lanes", [
    (torch.float16, 2, 64, 16, 262144, 32, 296, 128),   # four heads a block: 32 lane groups, each adds 4 rows of a step up first
    (torch.bfloat16, 2, 64, 16, 262144, 32, 296, 128),
    (torch.float16, 4, 64, 8, 200000, 32, 592, 64),     # eight heads: 2 rows, and long shares are cut in two
    (torch.bfloat16, 4, 64, 8, 200000, 32, 592, 64),
    (torch.float32, 3, 64, 8, 100000, 256, 592, 8)])    # 4 lane groups, 2 rows, cut in two
def test_long_group_decode_adds_no_longer_chains(dtype, B, H, kvH, Sk, D, blocks, lanes):
    """The error of long calls is that of chains of additions: an accumulator has k = rows / blocks / lanes of them. Sums of terms
    of either sign walk like sqrt(i), and so do their roundings (0.3 to 0.5 units of 2^-24, relative): about 0.2 sqrt(k) units,
    beside 3 to 4 of the scores and exponentials. Twice the chain is outside."""
    g = torch.Generator(device="cuda").manual_seed(11)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda").to(dtype) for h, n in ((H, 1), (kvH, Sk), (kvH, Sk)))
    want = torch.empty(B, H, 1, D, dtype=torch.double, device="cuda")
    for b in range(B):
        for j in range(kvH):
            s = q[b, j::kvH, 0].double() @ k[b, j].double().T / D ** 0.5
            want[b, j::kvH, 0] = torch.softmax(s, -1) @ v[b, j].double()
    out, m, l = torch.empty(B, H, 1, D, device="cuda"), torch.empty(B, H, 1, device="cuda"), torch.empty(B, H, 1, device="cuda")
    shape = api.AttentionShape(B, H, 1, Sk, D, kvH)
    api.launch_attention_init(out, m, l, shape)
    api.launch_attention_decode_step(q, k, v, out, m, l, shape, 0, 0, False)
    api.launch_attention_finalize(out, l, shape)
    chain = B * kvH * Sk / blocks / lanes
    assert ((out - want).norm() / want.norm()).item() <= 2.0 ** -24 * (4.5 + 0.2 * chain ** 0.5)


@pytest.mark.parametrize("dtype,D", [(torch.float32, 32), (torch.float32, 64), (torch.float32, 128), (torch.float32, 256), (torch.float16, 32)])
@pytest.mark.parametrize("H,kvH,Sk", [(4, 1, 37), (9, 2, 700), (16, 2, 20000)])
def test_group_decode_is_finite_where_single_heads_are(dtype, D, H, kvH, Sk):
    """Heads that share a butterfly and the weights of a step do not share what is not finite: as with a KV head for each head."""
    g = torch.Generator(device="cuda").manual_seed(Sk)
    q, k, v = (torch.randn(1, h, n, D, generator=g, device="cuda").to(dtype) for h, n in ((H, 1), (kvH, Sk), (kvH, Sk)))
    q[:, 0] = float("nan")
    q[:, H - 1, :, 1] = float("inf")
    q[..., 0].abs_()
    k[:, kvH - 1, Sk // 2, 0] = float("inf")
    v[:, 0, Sk // 3, 3] = float("inf")
    v[:, kvH - 1, Sk - 1, D - 1] = float("nan")
    outs = []
    for n in (kvH, H):
        kk, vv = (t.repeat(1, (H + kvH - 1) // kvH, 1, 1)[:, :H].contiguous() if n == H else t for t in (k, v))
        out, m, l = torch.empty(1, H, 1, D, device="cuda"), torch.empty(1, H, 1, device="cuda"), torch.empty(1, H, 1, device="cuda")
        shape = api.AttentionShape(1, H, 1, Sk, D, n)
        api.launch_attention_init(out, m, l, shape)
        api.launch_attention_decode_step(q, kk, vv, out, m, l, shape, 0, 0, False)
        api.launch_attention_finalize(out, l, shape)
        outs.append(out)
    finite = outs[1].isfinite()
    assert torch.equal(outs[0].isfinite(), finite) and not finite.all() and (finite.any() or kvH == 1)
    # (at most Sk additions of 2^-24 in either, and a few for scores and exponentials)
    if finite.any():
        assert (outs[0] - outs[1])[finite].abs().max().item() <= 2 * (Sk / 32 + 64) * 2.0 ** -24 * v[v.isfinite()].abs().max().item()


CAPTURES = """
import torch
from ring_attention_b200 import api

def call(B, H, kvH, Sk, D, seed, local):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda") for h, n in ((H, 1), (kvH, Sk), (kvH, Sk)))
    out, m, l = torch.empty_like(q), torch.empty(B, H, 1, device="cuda"), torch.empty(B, H, 1, device="cuda")
    shape = api.AttentionShape(B, H, 1, Sk, D, kvH)
    if local:
        cache = api.DeviceKVCache(B, kvH, Sk, D, torch.float32)
        cache.copy_prefill(k, v, Sk)
        return out, lambda: api.run_local_decode_step(q, cache, H, Sk, 0, True, out), cache
    def run():
        api.launch_attention_init(out, m, l, shape)
        api.launch_attention_decode_step(q, k, v, out, m, l, shape, 0, 0, False)
        api.launch_attention_finalize(out, l, shape)
    return out, run, None

def captured(run):
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        run()
    return graph

if cold:  # the library has no room for partials yet and cannot allocate any now: the call is recorded all the same
    out, run, _ = call(2, 64, 8, 20011, 256, 1, False)
    api.launch_attention_init(out, *(torch.empty(2, 64, 1, device="cuda") for _ in "ml"), api.AttentionShape(2, 64, 1, 1, 256, 8))
    graph = captured(run)
    graph.replay()
    torch.cuda.synchronize()
    got = out.clone()
    run()
    torch.cuda.synchronize()
    assert ((got - out).norm() / out.norm()).item() < 1e-6  # (a cluster and a fold add up in another order)
else:  # the room for partials and the scratch for m and l grow while a graph holds the old ones
    for local in (False, True):
        graphs = []
        for n, shape in enumerate([(1, 8, 8, 16384, 64), (2, 64, 8, 20011, 256), (6, 128, 16, 9000, 256)]):
            out, run, keep = call(*shape, n, local)
            run()
            torch.cuda.synchronize()
            want = out.clone()
            graphs.append((captured(run), out, want, keep, run))  # (what a graph reads has to live as long as it does)
            junk = [torch.full((1 << s,), float("nan"), device="cuda") for s in range(8, 24)]  # on what was given back, if anything was
            torch.cuda.synchronize()
            for graph, o, w, *_ in graphs:
                o.fill_(0)
                graph.replay()
                torch.cuda.synchronize()
                assert torch.equal(o, w)
            assert all(j.isnan().all() for j in junk)
            del junk
assert api.device_status()[0] == 0
"""


@pytest.mark.parametrize("cold", [True, False])
def test_graphs_keep_the_partials_they_were_captured_with(cold):
    """In a process of its own: what the library has allocated before decides what a capture meets."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", f"cold = {cold}\n" + CAPTURES], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("dtype,D", [(torch.float32, 64), (torch.float32, 256), (torch.float16, 32)])
@pytest.mark.parametrize("B,kvH,Sk,blocks", [  # blocks: no more than a KV head has of them
    (1, 1, 40000, 64), (1, 4, 20000, 64), (1, 8, 9001, 32), (1, 16, 6000, 16), (3, 16, 4100, 4), (8, 48, 700, 1)])
def test_fold_of_few_and_many_partials(dtype, D, B, kvH, Sk, blocks):
    """One to 128 partials to a row, by the number of groups, on a fresh and on an old state."""
    q, k, v = normal_inputs(17, B, 2 * kvH, kvH, 1, Sk, D)
    v = (v + np.sign(np.sin(np.arange(Sk) / 40.0))[:, None]).astype(np.float32)  # a lost share of the rows shows
    q, k, v = (round_to(x, dtype) for x in (q, k, v)) if dtype != torch.float32 else (q, k, v)
    want, tol = want64(q, k, v, kvH, blocks)
    dq, dk, dv = (torch.from_numpy(np.ascontiguousarray(x)).cuda().to(dtype) for x in (q, k, v))
    out = torch.full((B, 2 * kvH, 1, D), float("nan"), device="cuda")
    m, l = (torch.empty((B, 2 * kvH, 1), device="cuda") for _ in range(2))
    shape = api.AttentionShape(B, 2 * kvH, 1, Sk, D, kvH)
    api.launch_attention_init(out, m, l, shape)
    for _ in range(2):  # the same keys twice: every weight and the sum double, the quotient stays
        api.launch_attention_decode_step(dq, dk, dv, out, m, l, shape, 0, 0, False)
    api.launch_attention_finalize(out, l, shape)
    assert np.abs(out.cpu().numpy() - want).max() <= tol
