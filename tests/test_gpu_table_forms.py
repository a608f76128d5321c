"""The small tables of the tensor-level calls (signs, boundaries, levels, midpoints) may be numpy arrays of
any type and strides."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _forms(t):
    t = np.ascontiguousarray(t, dtype=np.float32)
    wide = np.zeros((t.size, 3), np.float32)
    wide[:, 1] = t
    return [t.astype(np.float64), wide[:, 1], t[::-1].copy()[::-1], t.astype(">f4")]


def test_every_call_takes_every_form():
    from fused_turboquant_b200 import TurboQuantMSE, kernels, tq_v1
    from fused_turboquant_b200.kernels import _host_table
    d, bits, n, hkv = 128, 4, 40, 2
    gen = torch.Generator("cuda").manual_seed(3)
    tq = TurboQuantMSE(d, bits=bits, device="cuda")
    signs, levels = _host_table(tq.rotation.signs), _host_table(tq.quantizer.levels)
    bounds = _host_table(tq.quantizer.boundaries)
    cent, mids = tq_v1.midpoints_of(tq.quantizer.levels)
    cent, mids = _host_table(cent), _host_table(mids)
    x = torch.randn(1, hkv, n, d, device="cuda", generator=gen).half()
    q = torch.randn(1, 4, 1, d, device="cuda", generator=gen)
    cfg = tq_v1.TurboQuantSlotConfig(d, bits, bits, norm_correction=True)
    kv = torch.randn(2, n, hkv, d, device="cuda", generator=gen).bfloat16()
    table = torch.arange(3, dtype=torch.int32, device="cuda")[None]

    def all_calls(signs, bounds, levels, cent, mids):
        codes, norms = kernels.fused_encode(x, signs, bounds, bits)
        cache = torch.zeros(3, 16, hkv, cfg.slot_size_aligned, dtype=torch.uint8, device="cuda")
        tq_v1.launch_store(kv[0], kv[1], cache, torch.arange(n, device="cuda"), mids, cfg)
        return [codes, norms, cache, kernels.fused_decode(codes, norms, levels, signs, bits, d),
                kernels.rht(x, signs),
                kernels.flash_decode_compressed(q, codes, norms, codes, norms, levels, levels, signs,
                                                d ** -0.5, bits, bits),
                tq_v1.decode_attention(q[:, :, 0], cache, table, torch.tensor([n], device="cuda"), cent, cfg,
                                       d ** -0.5)]

    want = all_calls(signs, bounds, levels, cent, mids)
    for forms in zip(*(_forms(t) for t in (signs, bounds, levels, cent, mids))):
        for got, w in zip(all_calls(*forms), want):
            assert torch.equal(got, w)
    with pytest.raises((TypeError, AttributeError)):
        kernels.rht(x, "signs")
