"""Kernels that start while the one before them in the stream still runs (launch_overlapped): what they
read is what that one wrote, and nothing they read changes under them. Every chain below runs once with
nothing waited for and once with a synchronisation after every call; the results are the same bits."""
import pytest
import torch

from ring_attention_b200 import api

pytestmark = pytest.mark.gpu

DTYPES = [torch.float16, torch.float32]


def chain(dtype, d, rows, wait, stream):
    """Three steps into one state, each on inputs written just before it (and overwritten just after),
    then the log-sum-exp, a half flash call on the result and cached decode steps on that."""
    def step_done():
        if wait:
            torch.cuda.synchronize()

    g = torch.Generator(device="cuda").manual_seed(rows + d)
    B, H, kvH = 1, 4, 2
    src = [torch.randn(3, B, h, rows, d, generator=g, device="cuda") for h in (H, kvH, kvH)]
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        q, k, v = (torch.empty(t.shape[1:], device="cuda", dtype=dtype) for t in src)
        out = torch.empty(B, H, rows, d, device="cuda")
        m, l = torch.empty(B, H, rows, device="cuda"), torch.empty(B, H, rows, device="cuda")
        shape = api.AttentionShape(B, H, rows, rows, d, kvH)
        for i in range(3):
            for t, s in zip((q, k, v), src):
                t.copy_(s[i])
            api.attention_step_ex(q, k, v, out, m, l, shape, api.SegMap.make([2 * rows], rows),
                                  api.SegMap.make([i * rows], rows), causal=True, fresh=i == 0, finalize=i == 2)
            step_done()
            for t in (q, k, v):
                t.fill_(float("nan"))
        lse = api.attention_lse(m, l)
        step_done()
        again = torch.empty_like(out)
        api.launch_flash_attention_fp16(out, src[1][0], src[2][0], again, shape, True)
        step_done()
        cache = api.DeviceKVCache(B, kvH, rows + 4, d, dtype)
        cache.copy_prefill(src[1][1].to(dtype), src[2][1].to(dtype), rows)
        tokens = []
        for i in range(4):
            new = again[:, :kvH, i:i + 1].to(dtype).contiguous()
            cache.append(new, new)
            step_done()
            o = torch.empty(B, H, 1, d, device="cuda")
            api.run_local_decode_step(again[:, :, i:i + 1].to(dtype).contiguous(), cache, H, rows + i, 0, True, o)
            step_done()
            again[:, :, i + 1:i + 2] += o
            tokens.append(o)
        stream.synchronize()
    return [out, lse, again, *tokens]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d,rows", [(64, 130), (64, 1000), (128, 700), (32, 4100), (256, 300)])
def test_back_to_back_is_what_waiting_gives(dtype, d, rows):
    want = chain(dtype, d, rows, True, torch.cuda.Stream())
    for _ in range(3):
        got = chain(dtype, d, rows, False, torch.cuda.Stream())
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    assert api.device_status()[0] == 0


def dependent_calls(dtype, d, heads, wait):
    """Calls of which each needs what the one before it wrote (or must not yet overwrite what that one reads),
    everything prepared beforehand, so that no other kernel stands between two of them. Few blocks that
    walk long: most SMs are free for the next call's blocks all the while."""
    def done():
        if wait:
            torch.cuda.synchronize()

    B, kvH, rows, keys, n = 1, heads // 2, 300, 3000, 6
    g = torch.Generator(device="cuda").manual_seed(d + heads)

    def normal(*shape, dt=dtype):
        return torch.randn(*shape, generator=g, device="cuda").to(dt)

    q, k, v = [normal(B, heads, rows, d) for _ in range(3)], [normal(B, kvH, keys, d) for _ in range(3)], \
        [normal(B, kvH, keys, d) for _ in range(3)]
    out = torch.full((B, heads, rows, d), float("nan"), device="cuda")
    m, l = (torch.full((B, heads, rows), float("nan"), device="cuda") for _ in range(2))
    shape = api.AttentionShape(B, heads, rows, keys, d, kvH)
    maps = api.SegMap.make([3 * keys], rows), [api.SegMap.make([i * keys], keys) for i in range(3)]
    f = [[normal(B, h, s, d, dt=torch.float32) for h, s in ((heads, rows), (kvH, keys), (kvH, keys))] for _ in range(3)]
    flash = [torch.empty(B, heads, rows, d, device="cuda") for _ in range(3)]
    cache = api.DeviceKVCache(B, kvH, keys + n, d, dtype)
    cache.k_view().fill_(float("nan"))
    cache.v_view().fill_(float("nan"))
    cache.copy_prefill(k[0], v[0], keys)
    new = [(normal(B, heads, 1, d), normal(B, kvH, 1, d), normal(B, kvH, 1, d)) for _ in range(n)]
    tokens = [torch.full((B, heads, 1, d), float("nan"), device="cuda") for _ in range(n)]
    torch.cuda.synchronize()
    for i in range(3):
        api.attention_step_ex(q[i], k[i], v[i], out, m, l, shape, maps[0], maps[1][i], causal=True, fresh=i == 0,
                              finalize=i == 2)
        done()
    lse = api.attention_lse(m, l)
    done()
    for i in range(3):  # (the fp16 copies of one call and the next lie in the same memory)
        api.launch_flash_attention_fp16(*f[i], flash[i], shape, True)
        done()
    for i in range(n):
        cache.append(new[i][1], new[i][2])
        done()
        api.run_local_decode_step(new[i][0], cache, heads, keys + i, 0, True, tokens[i])
        done()
    torch.cuda.synchronize()
    return [out, lse, *flash, *tokens]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [32, 64, 128, 256])
@pytest.mark.parametrize("heads", [4, 32])
def test_dependent_calls_with_nothing_between_them(dtype, d, heads):
    want = dependent_calls(dtype, d, heads, True)
    assert all(torch.isfinite(t).all() for t in want)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(dependent_calls(dtype, d, heads, False), want))
    assert api.device_status()[0] == 0
