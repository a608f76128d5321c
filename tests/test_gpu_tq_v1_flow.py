"""Slot-format decode by equal shares of whole pages (csrc/ftq_tq_v1_flow.cuh, 16-bit queries) against the fp32 kernel on the
same cache: partials of every split, merged output and lse.

Bar: that of the tensor-core stage 1 in tests/test_gpu_tq_v1.py (queries, centroids and weights are fp16 operands): at most
1 in 300 elements outside 2e-3 / 1e-3, none by more than 4e-3; lse within 2e-3 relative + 5e-3."""
import numpy as np
import pytest
import torch

from helpers import gate

pytestmark = pytest.mark.gpu


def _batch(D, kb, vb, Hkv, G, lens, bs=16, pad=0, layers=1, nc=True, seed=0):
    from fused_turboquant_b200 import TurboQuantMSE, tq_v1
    cfg = tq_v1.TurboQuantSlotConfig(D, kb, vb, norm_correction=nc)
    cent, mids = tq_v1.midpoints_of(TurboQuantMSE(D, bits=kb, device="cuda").quantizer.levels)
    g = torch.Generator("cuda").manual_seed(seed)
    width = max(1, max((n + bs - 1) // bs for n in lens))
    nb = len(lens) * width + 3
    bt = torch.randperm(nb, generator=g, device="cuda")[:len(lens) * width].view(len(lens), width).to(torch.int32)
    cache = torch.full((layers, nb, bs, Hkv, cfg.slot_size_aligned + pad), 0xFF, dtype=torch.uint8, device="cuda")
    for b, n in enumerate(lens):
        if n == 0:
            continue
        pos = torch.arange(n, device="cuda")
        slots = bt[b].long()[pos // bs] * bs + pos % bs
        for layer in range(layers):
            k = torch.randn(n, Hkv, D, generator=g, device="cuda").bfloat16()
            v = (torch.randn(n, Hkv, D, generator=g, device="cuda") + 0.3).bfloat16()
            tq_v1.launch_store(k, v, cache[layer], slots, mids, cfg)
    q = torch.randn(layers, len(lens), Hkv * G, D, generator=g, device="cuda").bfloat16()
    return cfg, cent, cache, bt, torch.tensor(lens, dtype=torch.int32, device="cuda"), q


def _decode(q, cache, bt, seq, cent, cfg, splits, start=None):
    from fused_turboquant_b200 import tq_v1
    lead, hq, d = q.shape[:-2], q.shape[-2], q.shape[-1]
    mid = torch.full((*lead, hq, splits, d + 1), 7.0, device="cuda")
    lse = torch.empty(*lead, hq, device="cuda")
    out = tq_v1.decode_attention(q, cache, bt, seq, cent, cfg, d ** -0.5, num_kv_splits=splits, kv_start_offset=start,
                                 mid_o=mid, lse=lse, out_dtype=torch.float32)
    return out.cpu().numpy(), mid.cpu().numpy(), lse.cpu().numpy()


def _compare(got, ref):
    (o, m, l), (o_ref, m_ref, l_ref) = got, ref
    live = np.isfinite(m_ref[..., -1])
    np.testing.assert_array_equal(np.isfinite(m[..., -1]), live)
    assert np.all(m[..., :-1][~live] == 0) and np.all(np.isneginf(m[..., -1][~live]))
    for x, y in ((m[..., :-1][live], m_ref[..., :-1][live]), (o, o_ref)):
        if x.size:
            assert gate(x, y) <= x.size // 300 and np.abs(x - y).max() < 4e-3, (gate(x, y), x.size, np.abs(x - y).max())
    np.testing.assert_allclose(m[..., -1][live], m_ref[..., -1][live], rtol=2e-3, atol=5e-3)
    np.testing.assert_allclose(l[np.isfinite(l_ref)], l_ref[np.isfinite(l_ref)], rtol=2e-3, atol=5e-3)


SHAPES = [(128, 4, 4, 8, 4), (128, 4, 4, 8, 8), (128, 4, 4, 16, 2), (128, 3, 4, 8, 1), (128, 4, 3, 8, 4), (128, 3, 3, 8, 8),
          (128, 2, 2, 16, 4), (64, 4, 4, 8, 4), (64, 4, 4, 16, 5), (64, 3, 3, 8, 7), (64, 3, 4, 8, 2), (64, 4, 2, 16, 8),
          (128, 4, 4, 4, 4)]   # (four heads: the item kernel)


@pytest.mark.parametrize("D,kb,vb,Hkv,G", SHAPES)
def test_ragged(D, kb, vb, Hkv, G):
    cfg, cent, cache, bt, seq, q = _batch(D, kb, vb, Hkv, G, [1, 0, 15, 16, 17, 333, 2500, 64], seed=D + Hkv)
    start = torch.tensor([0, 0, 3, 16, 16, 100, 7, 64], dtype=torch.int32, device="cuda")
    for splits, st in ((16, None), (19, start), (64, None), (3, start)):   # (3: the item kernel)
        _compare(_decode(q[0], cache[0], bt, seq, cent, cfg, splits, st),
                 _decode(q[0].float(), cache[0], bt, seq, cent, cfg, splits, st))


@pytest.mark.parametrize("bs,pad,nc", [(32, 0, True), (16, 2, False), (64, 10, True)])
def test_block_sizes_padding_and_long_pieces(bs, pad, nc):
    """Blocks of several pages, slots longer than their contents, shares that cut splits of many pages."""
    cfg, cent, cache, bt, seq, q = _batch(128, 4, 4, 8, 4, [9001, 4000], bs=bs, pad=pad, nc=nc)
    _compare(_decode(q[0], cache[0], bt, seq, cent, cfg, 64), _decode(q[0].float(), cache[0], bt, seq, cent, cfg, 64))


def test_slots_at_an_offset_of_wider_ones():
    """A view whose last page ends 16 bytes behind what a copy of whole slots would read.  (Compared with slots of the same
    pitch, so that the order of the sums is the same.)"""
    cfg, cent, cache, bt, seq, q = _batch(128, 4, 4, 8, 4, [1500, 16, 900], pad=26)   # slots of 160
    slot = cfg.slot_size_aligned
    view = torch.zeros_like(cache[0])[..., 16:16 + slot]
    view.copy_(cache[0, ..., :slot])
    for got, want in zip(_decode(q[0], view, bt, seq, cent, cfg, 64), _decode(q[0], cache[0], bt, seq, cent, cfg, 64)):
        np.testing.assert_array_equal(got, want)


def test_layers_in_several_launches():
    """64 query heads of 128: the workspace holds the rows of six layers, a call of eight is two launches."""
    cfg, cent, cache, bt, seq, q = _batch(128, 4, 4, 8, 8, [700, 90], layers=8)
    o, m, l = _decode(q, cache, bt, seq, cent, cfg, 64)
    for i in range(8):
        o1, m1, l1 = _decode(q[i], cache[i], bt, seq, cent, cfg, 64)
        assert np.array_equal(o[i], o1) and np.array_equal(m[i], m1) and np.array_equal(l[i], l1)


def test_bad_block_poisons_its_rows_only():
    cfg, cent, cache, bt, seq, q = _batch(128, 4, 4, 8, 4, [500, 900, 130])
    good, _, _ = _decode(q[0], cache[0], bt, seq, cent, cfg, 64)
    bt[1, 20] = cache.shape[1] + 5
    bt[2, 40] = -3                       # (beyond sequence 2's end: never read)
    bad, _, _ = _decode(q[0], cache[0], bt, seq, cent, cfg, 64)
    assert np.isnan(bad[1]).all() and np.array_equal(bad[[0, 2]], good[[0, 2]])


def test_captured_and_replayed():
    from fused_turboquant_b200 import tq_v1
    cfg, cent, cache, bt, seq, q = _batch(128, 4, 4, 8, 4, [500, 900, 130])
    mid, out = torch.empty(3, 32, 64, 129, device="cuda"), torch.empty_like(q[0])
    run = lambda: tq_v1.decode_attention(q[0], cache[0], bt, seq, cent, cfg, 128 ** -0.5, num_kv_splits=64, mid_o=mid, output=out)
    run()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        run()
    for n in ([500, 900, 130], [17, 1, 100]):
        seq.copy_(torch.tensor(n, dtype=torch.int32))
        run()
        want = out.clone()
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
