"""Bulk stores: several layers at once, and codebooks that the table quantiser does not take.
A comparison byte for byte with smaller stores."""
import numpy as np
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


# (codebooks whose boundaries share a cell of the quantiser table: every boundary is compared then; both
# tensors, one of them, and one of them above the size from which it gets a launch of its own)
@pytest.mark.parametrize("d,bk,bv,n,odd_k,odd_v,dtype", [
    (128, 4, 4, 1031, True, True, torch.bfloat16),
    (128, 4, 3, 2500, True, False, torch.float16),
    (64, 3, 4, 1025, False, True, torch.float32),
    (64, 2, 2, 1030, True, True, torch.bfloat16),
    (256, 3, 3, 1029, True, True, torch.bfloat16),
    (256, 4, 2, 20000, False, True, torch.bfloat16),
    (128, 4, 4, 17000, True, False, torch.bfloat16),
])
def test_any_codebook(d, bk, bv, n, odd_k, odd_v, dtype):
    """The same bytes as from stores of fewer than 2048 vectors, which compare every boundary as well."""
    from fused_turboquant_b200 import PagedKVPool
    key, value, slots = _store_inputs(1, n, 2, d, dtype, d + n)

    def odd(bits):
        b = np.linspace(-0.3, 0.3, (1 << bits) + 1).astype(np.float32)
        b[2] = b[1] + np.float32(1e-4)
        return b

    pools = [PagedKVPool((n + 15) // 16, 2, d, bk, bv, device="cuda") for _ in range(2)]
    for p in pools:
        p.pool.fill_(0xA5)
        if odd_k:
            p.bounds_k = odd(bk)
        if odd_v:
            p.bounds_v = odd(bv)
    pools[0].store(key[0], value[0], slots, layer=0)
    for at in range(0, n, 1000):
        part = slice(at, at + 1000)
        pools[1].store(key[0, part], value[0, part], slots[part], layer=0)
    assert torch.equal(pools[0].pool, pools[1].pool)
