"""Bulk stores over several layers: the same bytes as a store per layer."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _store_inputs(layers, n, hkv, d, dtype, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    kv = torch.randn(2, layers, n, hkv, d, device="cuda", generator=gen).to(dtype)
    slots = torch.randperm((n + 15) // 16 * 16, device="cuda", generator=gen)[:n]
    slots[1] = -1
    return kv[0], kv[1], slots


# (from 2048 vectors a layer on; groups of eight that end inside a token, fewer groups than warps of the
# grid and more, a step of whole layers and a remainder; both widths of the kernel's CTAs)
@pytest.mark.parametrize("layers,n,hkv,d,bk,bv,dtype", [
    (2, 2049, 1, 128, 4, 4, torch.bfloat16),
    (80, 259, 8, 128, 4, 3, torch.bfloat16),
    (3, 5000, 7, 64, 3, 2, torch.float16),
    (40, 301, 7, 256, 4, 4, torch.bfloat16),
    (5, 1031, 2, 256, 2, 3, torch.float32),
    (7, 2500, 8, 64, 4, 4, torch.float32),
])
def test_all_layers_at_once(layers, n, hkv, d, bk, bv, dtype):
    from fused_turboquant_b200 import PagedKVPool
    key, value, slots = _store_inputs(layers, n, hkv, d, dtype, d + n)
    pools = [PagedKVPool((n + 15) // 16, hkv, d, bk, bv, n_layers=layers, device="cuda") for _ in range(2)]
    for p in pools:
        p.pool.fill_(0xA5)
    pools[0].store(key, value, slots)
    for layer in range(layers):
        pools[1].store(key[layer], value[layer], slots, layer=layer)
    assert torch.equal(pools[0].pool, pools[1].pool)
