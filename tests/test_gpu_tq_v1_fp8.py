"""Slot-format decode with FP8 keys: the tensor-core kernel (16-bit queries) against 64-bit arithmetic on the
cache's bytes, and its error against that of the fp32 kernel, which fp32 queries take."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(q, cache, table, lens, d, vb, hkv, scale):
    """float64, torch on the GPU: [B, Hq, D]."""
    had = torch.ones(1, 1, dtype=torch.float64, device="cuda")
    while had.shape[0] < d:
        had = torch.cat([torch.cat([had, had], 1), torch.cat([had, -had], 1)], 0)
    qr = q.double() @ (had / d ** 0.5)
    out = []
    for b, n in enumerate(lens.tolist()):
        rows = cache[table[b].long()].reshape(-1, hkv, cache.shape[-1])[:n]
        k = rows[..., :d].contiguous().view(torch.float8_e4m3fn).double()
        bits = (rows[..., d:d + d * vb // 8, None].int() >> torch.arange(8, device="cuda")) & 1
        code = (bits.reshape(n, hkv, d, vb) << torch.arange(vb, device="cuda")).sum(-1).double()
        meta = rows[..., d + d * vb // 8:d + d * vb // 8 + 4].contiguous().view(torch.float16).double()
        v = code * meta[..., :1] + meta[..., 1:]
        group = q.shape[1] // hkv
        s = torch.einsum("hgd,nhd->hgn", qr[b].view(hkv, group, d), k) * scale
        out.append(torch.einsum("hgn,nhd->hgd", s.softmax(-1), v).reshape(-1, d))
    return torch.stack(out)


def _by_shares(q, cache, table, cfg, splits):
    """Does the call take the kernel that streams whole pages?"""
    from fused_turboquant_b200 import _lib
    return _lib.load().ftq_tq_decode_layers_workspace_bytes(
        _lib.BF16, q.shape[0], q.shape[1], cache.shape[2], q.shape[2], cache.data_ptr(), *cache.stride()[:3], cache.shape[1],
        table.shape[1], cfg.key_quant_bits, cfg.value_quant_bits, 0, splits, 1, 0) > 0


# (one token; less than a page; pages that not every warp has; remainders; groups on both sides of four;
# splits without tokens; one and several layers of items per CTA.  The last six: 128 units and more of 8 and 16 heads, by shares of
# pages, with unwritten slots in the pages that it reads whole)
@pytest.mark.parametrize("d,vb,hkv,group,lens,splits,dtype", [
    (128, 4, 2, 4, [1, 15, 16, 17], 8, "bf16"),
    (128, 4, 8, 4, [1000, 4096, 333], 8, "bf16"),
    (128, 3, 2, 7, [700, 90], 4, "fp16"),
    (128, 2, 1, 8, [513], 1, "bf16"),
    (64, 4, 4, 1, [129, 2000], 8, "fp16"),
    (64, 3, 2, 8, [40, 300], 3, "bf16"),
    (64, 2, 1, 3, [77] * 40, 16, "bf16"),
    (128, 4, 8, 4, [1, 15, 16, 17, 700, 3000], 32, "bf16"),
    (128, 3, 8, 1, [5, 9001], 64, "fp16"),
    (128, 2, 16, 3, [513] * 8, 16, "bf16"),
    (64, 4, 8, 7, [1000, 90], 64, "fp16"),
    (64, 3, 16, 2, [40, 300, 5000, 1], 32, "bf16"),
    (64, 2, 8, 8, [7000, 77, 16], 60, "bf16"),
])
def test_fp32_precision(d, vb, hkv, group, lens, splits, dtype):
    from fused_turboquant_b200 import tq_v1
    gen = torch.Generator("cuda").manual_seed(d + vb + group)
    cfg = tq_v1.TurboQuantSlotConfig(d, 8, vb, norm_correction=True)
    per = [(n + 15) // 16 for n in lens]
    cache = torch.randint(0, 255, (sum(per) + 1, 16, hkv, cfg.slot_size_aligned), dtype=torch.uint8, device="cuda",
                          generator=gen)       # (unwritten slots hold anything, NaN keys and scales too)
    ids = torch.randperm(sum(per) + 1, device="cuda", generator=gen)
    table = torch.zeros(len(lens), max(per), dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(lens):
        table[b, :per[b]] = ids[at:at + per[b]].int()
        pos = torch.arange(n, device="cuda")
        slots = ids[at:at + per[b]][pos // 16] * 16 + pos % 16
        kv = torch.randn(2, n, hkv, d, device="cuda", generator=gen)
        kv[..., 1] *= 5.0
        tq_v1.launch_store(kv[0].bfloat16(), kv[1].bfloat16(), cache, slots, None, cfg)
        at += per[b]
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q = torch.randn(len(lens), hkv * group, d, device="cuda", generator=gen)
    q = q.to(torch.bfloat16 if dtype == "bf16" else torch.float16)
    assert _by_shares(q, cache, table, cfg, splits) == (hkv >= 8 and len(lens) * splits >= 128)

    def run(x):
        out = torch.empty(x.shape, dtype=torch.float32, device="cuda")
        tq_v1.decode_attention(x, cache, table, sl, None, cfg, d ** -0.5, num_kv_splits=splits, output=out)
        return out

    ref = _exact(q, cache, table, sl, d, vb, hkv, d ** -0.5)
    new, old = ((run(x).double() - ref).norm().item() / ref.norm().item() for x in (q, q.float()))
    # fp32 exponentials, sums over up to 4096 tokens: a few 2^-24
    print(f"relative error: tensor cores {new:.2e}, fp32 kernel {old:.2e}")
    assert new < 1e-6 and new < 2.0 * old + 1e-7


def test_slots_off_the_word_stay_on_the_fp32_kernel():
    """A cache whose slots start on 2-byte boundaries gives the same result through the other kernel."""
    from fused_turboquant_b200 import tq_v1
    d, hkv, n = 128, 2, 50
    gen = torch.Generator("cuda").manual_seed(1)
    cfg = tq_v1.TurboQuantSlotConfig(d, 8, 4, norm_correction=True)
    size = cfg.slot_size_aligned
    kv = torch.randn(2, n, hkv, d, device="cuda", generator=gen).bfloat16()
    q = torch.randn(1, 8, d, device="cuda", generator=gen).bfloat16()
    table = torch.arange(4, dtype=torch.int32, device="cuda")[None]
    sl = torch.tensor([n], dtype=torch.int32, device="cuda")
    outs = []
    for pad in (0, 2):
        cache = torch.zeros(4, 16, hkv, size + pad, dtype=torch.uint8, device="cuda")[..., :size]
        tq_v1.launch_store(kv[0], kv[1], cache, torch.arange(n, device="cuda"), None, cfg)
        out = torch.empty(1, 8, d, dtype=torch.float32, device="cuda")
        tq_v1.decode_attention(q, cache, table, sl, None, cfg, d ** -0.5, num_kv_splits=4, output=out)
        outs.append(out.cpu().numpy())
    assert np.allclose(outs[0], outs[1], rtol=0, atol=2e-6)


@pytest.mark.parametrize("d,vb,group", [(128, 4, 4), (128, 3, 8), (64, 4, 7)])
@pytest.mark.parametrize("n,splits,scale,shift,wide", [
    (4096, 8, 1.0, 0.0, 10.0),      # 1 % of the channels ten times larger, as real keys have them
    (4096, 8, 1e-4, 0.0, 10.0),     # small value scales
    (4096, 8, 1.0, 10.0, 1.0),      # a value channel that is never near zero
    (30000, 8, 1.0, 0.0, 10.0),     # 30 pages a warp
    (4096, 32, 1.0, 0.0, 10.0),     # by shares of pages (groups of 128 up to four, of 64 up to eight), 8 pages a split
    (16384, 32, 1.0, 0.0, 10.0),    # ... up to 16 pages a warp
    (16384, 32, 1e-4, 10.0, 1.0),
])
def test_error_is_no_larger_than_the_fp32_kernels(d, vb, group, n, splits, scale, shift, wide):
    from fused_turboquant_b200 import tq_v1
    gen = torch.Generator("cuda").manual_seed(d + vb + group + n)
    hkv, B = (2 if n > 20000 else 8), 4
    cfg = tq_v1.TurboQuantSlotConfig(d, 8, vb, norm_correction=True)
    per = (n + 15) // 16
    cache = torch.zeros(B * per, 16, hkv, cfg.slot_size_aligned, dtype=torch.uint8, device="cuda")
    table = torch.randperm(B * per, device="cuda", generator=gen).int().view(B, per)
    pos = torch.arange(n, device="cuda")
    for b in range(B):
        kv = torch.randn(2, n, hkv, d, device="cuda", generator=gen)
        outlier = torch.rand(hkv, d, device="cuda", generator=gen) < 0.01
        outlier[0, 1] = True
        kv = torch.where(outlier, kv * wide, kv)
        kv[1, ..., 2] += shift
        kv[1] *= scale
        slots = table[b].long()[pos // 16] * 16 + pos % 16
        tq_v1.launch_store(kv[0].bfloat16(), kv[1].bfloat16(), cache, slots, None, cfg)
    sl = torch.full((B,), n, dtype=torch.int32, device="cuda")
    q = torch.randn(B, hkv * group, d, device="cuda", generator=gen).bfloat16()
    assert _by_shares(q, cache, table, cfg, splits) == (splits == 32 and (d == 64 or group <= 4))
    ref = _exact(q, cache, table, sl, d, vb, hkv, d ** -0.5)
    err = []
    for x in (q, q.float()):
        out = torch.empty(q.shape, dtype=torch.float32, device="cuda")
        tq_v1.decode_attention(x, cache, table, sl, None, cfg, d ** -0.5, num_kv_splits=splits, output=out)
        err.append(((out.double() - ref).norm(dim=-1) / ref.norm(dim=-1)).mean().item())
    # means over 32 heads and more of errors of the same size; 0.57 to 1.02 measured
    print(f"mean error: tensor cores {err[0]:.2e}, fp32 kernel {err[1]:.2e}")
    assert err[0] < 1.15 * err[1]
