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


def _decode(q, cache, bt, seq, cent, cfg, splits, start=None, **kw):
    from fused_turboquant_b200 import tq_v1
    lead, hq, d = q.shape[:-2], q.shape[-2], q.shape[-1]
    mid = torch.full((*lead, hq, splits, d + 1), 7.0, device="cuda")
    lse = torch.empty(*lead, hq, device="cuda")
    out = tq_v1.decode_attention(q, cache, bt, seq, cent, cfg, d ** -0.5, num_kv_splits=splits, kv_start_offset=start,
                                 mid_o=mid, lse=lse, out_dtype=torch.float32, **kw)
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


def _items():
    """The workspace with which the item kernels run."""
    return torch.empty(0, dtype=torch.uint8, device="cuda")


def _float64(q, cache, bt, seq, cent, cfg):
    """Attention over the cache's bytes in 64 bits: [B, Hq, D]."""
    d, kb, vb, hkv = q.shape[-1], cfg.key_quant_bits, cfg.value_quant_bits, cache.shape[-2]
    had = torch.ones(1, 1, dtype=torch.float64, device="cuda")
    while had.shape[0] < d:
        had = torch.cat([torch.cat([had, had], 1), torch.cat([had, -had], 1)], 0)
    qr, out = q.double() @ (had / d ** 0.5), []

    def codes(rows, bits):
        b = (rows[..., None].int() >> torch.arange(8, device="cuda")) & 1
        return (b.reshape(*rows.shape[:-1], d, bits) << torch.arange(bits, device="cuda")).sum(-1)
    for b, n in enumerate(seq.tolist()):
        rows = cache[bt[b].long()].reshape(-1, hkv, cache.shape[-1])[:n]
        kc, vc = d * kb // 8, d * vb // 8
        k = cent.cuda().double()[codes(rows[..., :kc], kb)]
        norm = rows[..., kc:kc + 2].contiguous().view(torch.float16).double()
        if cfg.norm_correction:
            norm = norm / (k.norm(dim=-1, keepdim=True) ** 2 + 1e-16).sqrt()
        meta = rows[..., kc + 2 + vc:kc + 6 + vc].contiguous().view(torch.float16).double()
        v = codes(rows[..., kc + 2:kc + 2 + vc], vb).double() * meta[..., :1] + meta[..., 1:]
        s = torch.einsum("hgd,nhd->hgn", qr[b].view(hkv, -1, d), k * norm) * d ** -0.5
        out.append(torch.einsum("hgn,nhd->hgd", s.softmax(-1), v).reshape(-1, d))
    return torch.stack(out)


@pytest.mark.parametrize("D,kb,vb,Hkv,G,n,splits", [(128, 4, 4, 8, 4, 4096, 32), (128, 4, 4, 8, 8, 20000, 32), (128, 3, 3, 8, 4, 20000, 32),
                                                    (64, 3, 4, 16, 2, 9000, 32), (128, 4, 4, 8, 4, 40000, 32)])
def test_error_is_no_larger_than_the_item_kernels(D, kb, vb, Hkv, G, n, splits):
    """Against 64 bits, where a warp adds up the pages of a split in one accumulator (up to 80 pages there)."""
    cfg, cent, cache, bt, seq, q = _batch(D, kb, vb, Hkv, G, [n] * 4)
    ref = _float64(q[0], cache[0], bt, seq, cent, cfg).cpu().numpy()
    err = [(np.linalg.norm(_decode(q[0], cache[0], bt, seq, cent, cfg, splits, workspace=w)[0] - ref, axis=-1) /
            np.linalg.norm(ref, axis=-1)).mean() for w in (None, _items())]
    print(f"mean error: shares {err[0]:.3e}, items {err[1]:.3e}")
    assert err[0] < 1.02 * err[1]     # (means over 128 rows and more of errors of the same size)


@pytest.mark.parametrize("D,layers", [(128, 1), (64, 1), (128, 8)])   # (eight layers of 64 heads of 128: two launches)
def test_rotation_and_prefix(D, layers):
    """What the merge does after the sums, a sequence without tokens and one without a prefix among them."""
    cfg, cent, cache, bt, seq, q = _batch(D, 4, 4, 8, 8 if layers > 1 else 4, [700, 0, 90, 333], layers=layers)
    q, cache = (q, cache) if layers > 1 else (q[0], cache[0])
    g = torch.Generator("cuda").manual_seed(5)
    pre = torch.randn(q.shape, generator=g, device="cuda").bfloat16()
    pre_lse = torch.randn(q.shape[:-1], generator=g, device="cuda") + 4.0
    pre_lse[..., 2, :] = -float("inf")
    for kw in (dict(v_rotate=True), dict(prefix_output=pre, prefix_lse=pre_lse),
               dict(v_rotate=True, prefix_output=pre, prefix_lse=pre_lse)):
        (o, _, l), (o_ref, _, l_ref) = (_decode(q, cache, bt, seq, cent, cfg, 32, workspace=w, **kw) for w in (None, _items()))
        assert gate(o, o_ref) <= o.size // 300 and np.abs(o - o_ref).max() < 4e-3
        assert np.array_equal(np.isneginf(l), np.isneginf(l_ref))
        live = np.isfinite(l_ref)
        np.testing.assert_allclose(l[live], l_ref[live], rtol=2e-3, atol=5e-3)
