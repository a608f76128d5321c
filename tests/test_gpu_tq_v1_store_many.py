"""Slot-format store of many vectors (csrc/ftq_tq_v1_store2.cuh): byte for byte the cache that the oracle writes, and for
what the oracle has no argument for (rotation in the kernel, NaN and infinities) the cache that the octet kernel writes, which
calls of fewer than 2048 vectors (heads of 256: 5120, FP8 keys 12288) take (tests/test_gpu_tq_v1.py pins that one)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
HKV, BS = 3, 16


def _inputs(n, d, dtype, seed, wild):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(2, n, HKV, d, generator=g)
    x[:, :, :, ::37] *= 10.0
    x[:, 1] = 0.0
    x[:, 2] = -0.0
    x[:, 3, :, 5:] = 0.0
    x[:, 4] = 1.25                       # a range of zero, a rotated vector with one non-zero coordinate
    x[:, 5] *= 2.0 ** -13
    x[:, 6, :, 1] = -0.0
    if dtype is torch.bfloat16:
        x[:, 7] *= 1e-20                 # squares that vanish, quotients by 1e-8
        x[:, 8, :, ::3] *= 1e-30         # tiny elements among ordinary ones
        x[:, 9] *= 1e17
    if wild:
        x[:, 10] *= 1e37 if dtype is torch.bfloat16 else 6000.0   # norms and ranges that overflow
        x[:, 11, :, 7] = float("nan")
        x[:, 12, :, 3] = float("inf")
        x[:, 13, :, 4] = -float("inf")
    return x.to(dtype)


def _store(tq_v1, key, value, nb, cfg, mids, slots, rot, chunk):
    cache = torch.full((nb, BS, HKV, cfg.slot_size_aligned), 0xA5, dtype=torch.uint8, device="cuda")
    for at in range(0, len(slots), chunk):
        tq_v1.launch_store(key[at:at + chunk], value[at:at + chunk], cache, slots[at:at + chunk], mids, cfg, v_rotate=rot)
    return cache


@pytest.mark.parametrize("kb", [3, 4, 8])
@pytest.mark.parametrize("vb", [3, 4])
@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_bytes(oracle, d, kb, vb, dtype):
    from fused_turboquant_b200 import TurboQuantMSE, tq_v1
    # 3093 vectors, with heads of 256 12297: neither whole warps of eight nor whole waves
    n = 1031 if d < 256 else 4099
    cfg = tq_v1.TurboQuantSlotConfig(d, kb, vb)
    _, mids = tq_v1.midpoints_of(TurboQuantMSE(d, bits=kb if kb < 8 else vb, device="cuda").quantizer.levels)
    nb = (n + BS - 1) // BS + 2
    slots = torch.randperm(nb * BS, generator=torch.Generator().manual_seed(d + kb))[:n]
    slots[20], slots[21] = -1, nb * BS   # padding, beyond the end
    for rot in (False, True):
        key, value = (t.cuda() for t in _inputs(n, d, dtype, 100 * d + 10 * kb + vb, wild=True))
        many = _store(tq_v1, key, value, nb, cfg, mids, slots.cuda(), rot, n)
        few = _store(tq_v1, key, value, nb, cfg, mids, slots.cuda(), rot, 600)
        assert torch.equal(many, few)
    key, value = (t.cuda() for t in _inputs(n, d, dtype, 100 * d + 10 * kb + vb, wild=False))
    many = _store(tq_v1, key, value, nb, cfg, mids, slots.cuda(), False, n).cpu().numpy()
    ref = np.full_like(many, 0xA5)
    keep = np.array([s for s in range(n) if 0 <= slots[s] < nb * BS])
    oracle.tq_store(key.float().cpu().numpy()[keep], value.float().cpu().numpy()[keep], ref, slots.numpy()[keep],
                    mids.cpu().numpy(), kb, vb)
    np.testing.assert_array_equal(many, ref)


@pytest.mark.parametrize("offset", [0.0, 0.5])
def test_values_on_midpoints(offset):
    """A midpoint at 0 (zero vectors sit on it), and coordinates that equal midpoints exactly."""
    from fused_turboquant_b200 import tq_v1
    d, n = 64, 800
    cfg = tq_v1.TurboQuantSlotConfig(d, 4, 4)
    mids = torch.arange(-7, 8, dtype=torch.float32) * 0.125 + offset / 64
    key = torch.zeros(n, HKV, d, dtype=torch.bfloat16, device="cuda")
    key[torch.arange(n), :, torch.arange(n) % d] = 1.0      # rotated: +-1/8, the midpoints -1 and 1 of offset 0
    key[::7] = 0.0
    slots = torch.arange(n, device="cuda")
    a = _store(tq_v1, key, key, n // BS, cfg, mids, slots, False, n)
    b = _store(tq_v1, key, key, n // BS, cfg, mids, slots, False, 600)
    assert torch.equal(a, b)


def test_layers_in_one_launch():
    from fused_turboquant_b200 import TurboQuantMSE, tq_v1
    d, L, n = 128, 3, 333
    cfg = tq_v1.TurboQuantSlotConfig(d, 4, 4)
    _, mids = tq_v1.midpoints_of(TurboQuantMSE(d, bits=4, device="cuda").quantizer.levels)
    x = torch.stack([_inputs(n, d, torch.bfloat16, s, True) for s in range(L)]).cuda()   # [L, 2, n, Hkv, d]
    key, value = x[:, 0].contiguous(), x[:, 1].contiguous()
    slots = torch.randperm(352, generator=torch.Generator().manual_seed(1))[:n].cuda()
    cache = torch.zeros(L, 22, BS, HKV, cfg.slot_size_aligned, dtype=torch.uint8, device="cuda")
    tq_v1.launch_store(key, value, cache, slots, mids, cfg, v_rotate=True)
    for layer in range(L):
        one = torch.zeros_like(cache[0])
        tq_v1.launch_store(key[layer], value[layer], one, slots, mids, cfg, v_rotate=True)
        assert torch.equal(cache[layer], one)
