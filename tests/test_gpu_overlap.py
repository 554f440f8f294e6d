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
