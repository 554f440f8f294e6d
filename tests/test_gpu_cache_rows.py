"""A prompt's rows into the KV cache by one launch, and by device copies where the kernel cannot take them: the cache
holds the source's bits and nothing beside them changes."""
import pytest
import torch

from ring_attention_b200.api import DeviceKVCache

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,D", [(torch.float16, 64), (torch.bfloat16, 128), (torch.float32, 32), (torch.float16, 3), (torch.float32, 1)])
@pytest.mark.parametrize("batch,kv_heads,rows", [(1, 1, 2), (2, 3, 255), (1, 2, 256), (1, 2, 257), (3, 1, 1531)])
@pytest.mark.parametrize("shift", [0, 1])
def test_prompt_rows_reach_the_cache(dtype, D, batch, kv_heads, rows, shift):
    g = torch.Generator(device="cuda").manual_seed(rows)
    n = batch * kv_heads * rows * D
    k, v = (torch.randn(n + 8, generator=g, device="cuda").to(dtype)[shift:shift + n].view(batch, kv_heads, rows, D) for _ in range(2))
    cache = DeviceKVCache(batch, kv_heads, rows + 5, D, dtype)
    views = cache.k_view(), cache.v_view()
    for t in views:
        t.fill_(9)
    cache.copy_prefill(k, v, rows)
    assert cache.current_len() == rows
    for t, src in zip(views, (k, v)):
        assert torch.equal(t[:, :, :rows], src)
        assert (t[:, :, rows:] == 9).all()
    cache.append(k[:, :, :1].contiguous(), v[:, :, :1].contiguous())  # right behind it
    assert torch.equal(views[0][:, :, rows], k[:, :, 0]) and torch.equal(views[1][:, :, rows], v[:, :, 0])
