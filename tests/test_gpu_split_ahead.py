"""fp32 steps whose K and V are split into fp16 terms by a launch ahead: the same bits as when every block splits them.
(What the bits are worth is tested where every block does: test_gpu_step.py, test_gpu_forms.py.)"""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
from ring_attention_b200 import api
from ring_attention_b200._lib import RA_F32, SegMap, lib
from util import assert_close

pytestmark = pytest.mark.gpu

AHEAD = 256
CAUSAL, FRESH, FINALIZE = 1, 2, 4


def run(q, k, v, state, shape, qmap, kmap, stride, flags, doc, ws, room=0):
    api.check(lib().ra_attention_step_ws(
        RA_F32, *(api._ptr(t) for t in (q, k, v, *state)), C.byref(shape.c()), C.byref(qmap), C.byref(kmap), stride, flags, doc, room,
        ws.data_ptr() if ws is not None else None, ws.numel() if ws is not None else 0, api._stream()))
    return lib().ra_debug_step_form()


def spoil(case, q, k, v):
    """Values that mark tiles, and values that are not finite."""
    if case == "wide V":
        v[:, :, 100:103] *= 2.0 ** -14      # keys far below their tile
        v[:, :, 700:900, 5] *= 2.0 ** -20   # a column
    elif case == "wide Q and K":
        q[..., 3] *= 2.0 ** 20
        k[:, :, 300:420, 3] *= 2.0 ** -24
        k[:, :, 300:420, 7] *= 2.0 ** 6
    elif case == "growing":
        ramp = torch.exp2(torch.linspace(-40, 40, k.shape[2], device="cuda"))[:, None]
        v *= ramp
        k *= torch.linspace(0, 3, k.shape[2], device="cuda")[:, None]
    elif case == "not finite":
        k[:, :, 200, 1] = float("nan")
        v[:, :, 333, 2] = float("inf")
        v[:, :, 1500, 0] = float("nan")
        q[:, :, 7] = float("inf")
    elif case == "zeros":
        k[:, :, 64:256] = 0
        v[:, :, 128:512] = 0


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("split", [0, 1, 3])
@pytest.mark.parametrize("case", ["plain", "segments", "strides", "documents", "ragged", "wide V", "wide Q and K", "growing",
                                  "not finite", "zeros"])
def test_split_ahead_gives_the_same_bits(D, split, case):
    B, H, kvH = 1, 16, 2
    qb, rows, kb, keys, stride, flags, doc = {
        "segments": ([0, 9000], 1100, [0, 3000, 6000], 1400, 1, CAUSAL, 0),
        "strides": ([4301], 2100, [0], 4200, 2, CAUSAL, 0),
        "documents": ([2200], 2050, [0], 4250, 1, CAUSAL, 3900),
        "ragged": ([3000], 1999, [0], 4999, 1, CAUSAL, 0),
    }.get(case, ([0], 2048, [0], 3000, 1, 0, 0))
    g = torch.Generator(device="cuda").manual_seed(D)
    Sq, Sk = rows * len(qb), keys * len(kb)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda") for h, n in ((H, Sq), (kvH, Sk), (kvH, Sk)))
    spoil(case, q, k, v)
    shape, qmap, kmap = api.AttentionShape(B, H, Sq, Sk, D, kvH), SegMap.make(qb, rows), SegMap.make(kb, keys)
    flags |= split << 8
    room = Sk + 33  # a cache with room
    ck, cv = (torch.full((B, kvH, room, D), 7.0, device="cuda") for _ in range(2))
    ck[:, :, :Sk], cv[:, :, :Sk] = k, v
    need = lib().ra_attention_step_workspace_bytes(RA_F32, C.byref(shape.c()), C.byref(qmap), C.byref(kmap), stride, flags, doc)
    assert need > 0
    buf = torch.full((need + 4096,), 0xff, dtype=torch.uint8, device="cuda")  # (NaN where nothing is written)
    ws = buf[:need]
    old = [torch.randn(q.shape, generator=g, device="cuda"), torch.randn(q.shape[:3], generator=g, device="cuda"),
           torch.rand(q.shape[:3], generator=g, device="cuda") + 0.5]
    for extra, (kk, vv, r) in ((FRESH, (k, v, 0)), (FINALIZE, (ck, cv, room))):
        a, b = [t.clone() for t in old], [t.clone() for t in old]
        assert not run(q, kk, vv, a, shape, qmap, kmap, stride, flags | extra, doc, None, r) & AHEAD
        assert run(q, kk, vv, b, shape, qmap, kmap, stride, flags | extra, doc, ws, r) & AHEAD
        for x, y in zip(a, b):
            assert torch.equal(x.view(torch.int32), y.view(torch.int32))
    assert (buf[need:] == 0xff).all() and api.device_status()[0] == 0


@pytest.mark.parametrize("H,kvH,S,causal", [(4, 4, 8192, 1), (6, 2, 5000, 1), (128, 4, 129, 0), (3, 1, 7777, 0)])
def test_head_dim_128_refills_slots_behind_both_issuing_warps(H, kvH, S, causal):
    """Two warps issue, and a ring slot is free when the MMAs of both have read it: long walks, blocks with one and with two
    query tiles, again and again, give the bits of the form with one issuing warp."""
    Sk = max(S, 3000)
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(1, h, n, 128, generator=g, device="cuda") for h, n in ((H, S), (kvH, Sk), (kvH, Sk)))
    shape, qmap, kmap = api.AttentionShape(1, H, S, Sk, 128, kvH), SegMap.make([Sk - S], S), SegMap.make([0], Sk)
    flags = causal * CAUSAL | FRESH | FINALIZE
    ws = torch.empty(2 * kvH * (Sk + 64) * 128 * 4 + kvH * (Sk + 64) * 8, dtype=torch.uint8, device="cuda")
    want, state = ([torch.empty(s, device="cuda") for s in (q.shape, q.shape[:3], q.shape[:3])] for _ in range(2))
    assert not run(q, k, v, want, shape, qmap, kmap, 1, flags, 0, None) & AHEAD
    for _ in range(10):
        for t in state:
            t.fill_(float("nan"))
        assert run(q, k, v, state, shape, qmap, kmap, 1, flags, 0, ws) & AHEAD
        assert all(torch.equal(x, y) for x, y in zip(want, state))
    assert api.device_status()[0] == 0


def test_flash_with_and_without_room_for_the_split():
    B, H, kvH, S, D = 1, 16, 2, 2500, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(B, h, S, D, generator=g, device="cuda") for h in (H, kvH, kvH))
    shape = api.AttentionShape(B, H, S, S, D, kvH)
    need, base = lib().ra_flash_workspace_bytes(C.byref(shape.c()), 0), 2 * B * H * S * 4 + 256
    assert need > base
    ws = torch.empty(need + 8, dtype=torch.uint8, device="cuda")
    outs, forms = [], []
    for p, n in ((ws.data_ptr(), need), (ws.data_ptr(), base), (ws.data_ptr() + 4, need - 512), (ws.data_ptr() + 4, need)):
        outs.append(torch.full_like(q, float("nan")))
        api.check(lib().ra_flash_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), outs[-1].data_ptr(), C.byref(shape.c()), 1, 0, p, n, api._stream()))
        forms.append(lib().ra_debug_step_form() & AHEAD)
    assert forms[0] == AHEAD and forms[1] == forms[2] == 0
    assert all(torch.equal(o, outs[0]) for o in outs)
    assert lib().ra_flash_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), outs[0].data_ptr(), C.byref(shape.c()), 1, 0, ws.data_ptr(), base - 1, api._stream()) == 6
    rows = slice(2400, 2410)
    want = oracle.cpu_attention(q[:, :, :2410].cpu().numpy(), k[:, :, :2410].cpu().numpy(), v[:, :, :2410].cpu().numpy(), True, kv_heads=kvH)
    assert_close(outs[0][:, :, rows].cpu().numpy(), want[:, :, rows], 1e-5, 1e-5, "flash")


def test_calls_run_without_the_split_where_there_is_no_room_for_it():
    B, H, kvH, rows, keys, D = 1, 16, 8, 2048, 20000, 128
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda") for h, n in ((H, rows), (kvH, keys), (kvH, keys)))
    shape, qmap, kmap = api.AttentionShape(B, H, rows, keys, D, kvH), SegMap.make([0], rows), SegMap.make([0], keys)
    state = [torch.empty(s, device="cuda") for s in (q.shape, q.shape[:3], q.shape[:3])]
    flash = torch.empty_like(q)

    def both():
        api.attention_step_ex(q, k, v, *state, shape, qmap, kmap, fresh=True, finalize=True)
        forms = [lib().ra_debug_step_form() & AHEAD]
        api.launch_flash_attention(q, k, v, flash, shape, True)
        return forms + [lib().ra_debug_step_form() & AHEAD]

    assert both() == [AHEAD, AHEAD]
    want = [t.clone() for t in (*state, flash)]
    for t in (*state, flash):
        t.fill_(0)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = torch.cuda.memory_reserved() + (64 << 20)  # K and V in split form take 164 MB
    torch.cuda.set_per_process_memory_fraction(room / torch.cuda.get_device_properties(0).total_memory)
    try:
        assert both() == [0, 0]
        with pytest.raises(torch.OutOfMemoryError):  # not even what the call cannot do without
            api._workspace(1 << 30, lambda: 1 << 29)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert all(torch.equal(a, b) for a, b in zip((*state, flash), want))
    assert both() == [AHEAD, AHEAD]


@pytest.mark.parametrize("D", [64, 128])
def test_split_ahead_steps_that_give_up_keep_their_state(D):
    B, H, kvH, rows, keys = 1, 16, 2, 2048, 3000
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda") for h, n in ((H, rows), (kvH, keys), (kvH, keys)))
    shape, qmap, kmap = api.AttentionShape(B, H, rows, keys, D, kvH), SegMap.make([0], rows), SegMap.make([0], keys)
    state = [torch.full(s, 3.0, device="cuda") for s in (q.shape, q.shape[:3], q.shape[:3])]
    lib().ra_debug_set_wait_limit_ns(5_000_000)
    lib().ra_debug_stall_producer_after(10)
    try:
        api.attention_step_ex(q, k, v, *state, shape, qmap, kmap, finalize=True)
        assert lib().ra_debug_step_form() & AHEAD
        lib().ra_debug_stall_producer_after(-1)
        api.attention_step_ex(q, k, v, *state, shape, qmap, kmap, fresh=True)  # starts beside the first
        torch.cuda.synchronize()
    finally:
        lib().ra_debug_stall_producer_after(-1)
        lib().ra_debug_set_wait_limit_ns(0)
    assert api.device_status()[0] == 5
    assert all((t == 3.0).all() for t in state)
