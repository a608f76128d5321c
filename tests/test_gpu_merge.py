"""The split-KV merges in both widths: a warp per vector up to 16 vectors per SM, an octet above."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rotate", [False, True])
def test_slot_format(rotate):
    """The splits do not depend on the batch, so the same rows go through both widths (sums of 5 or 8
    weighted partials in two orders: a few 2^-24 of the largest)."""
    from fused_turboquant_b200 import tq_v1
    d, hkv, group, n, splits = 64, 1, 16, 200, 7
    B = 16 * torch.cuda.get_device_properties(0).multi_processor_count // group
    gen = torch.Generator("cuda").manual_seed(2)
    cfg = tq_v1.TurboQuantSlotConfig(d, 8, 4, norm_correction=True)
    cache = torch.zeros(13, 16, hkv, cfg.slot_size_aligned, dtype=torch.uint8, device="cuda")
    kv = torch.randn(2, n, hkv, d, device="cuda", generator=gen).bfloat16()
    tq_v1.launch_store(kv[0], kv[1], cache, torch.arange(n, device="cuda"), None, cfg, v_rotate=rotate)
    table = torch.arange(13, dtype=torch.int32, device="cuda").repeat(B + 1, 1)
    lens = torch.randint(1, n + 1, (B + 1,), device="cuda", generator=gen).int()   # (splits without tokens)
    q = torch.randn(B + 1, group, d, device="cuda", generator=gen)

    def run(rows):
        lse = torch.empty(rows, group, dtype=torch.float32, device="cuda")
        out = tq_v1.decode_attention(q[:rows], cache, table[:rows], lens[:rows], None, cfg, d ** -0.5,
                                     num_kv_splits=splits, v_rotate=rotate, lse=lse)
        return out, lse

    (wide, lse_w), (narrow, lse_n) = run(B), run(B + 1)
    assert not torch.equal(wide, narrow[:B])     # (the border is where the test takes it to be)
    torch.testing.assert_close(wide, narrow[:B], rtol=0, atol=2e-6)
    torch.testing.assert_close(lse_w, lse_n[:B], rtol=0, atol=2e-6)


@pytest.mark.parametrize("above", [0, 1])
def test_contiguous_format(above):
    """Queries on both sides of the border against 64-bit arithmetic on the decoded vectors."""
    from fused_turboquant_b200 import TurboQuantMSE, kernels
    d, group, n, bits = 64, 16, 1999, 4
    B = 16 * torch.cuda.get_device_properties(0).multi_processor_count // group + above
    gen = torch.Generator("cuda").manual_seed(5)
    tq = TurboQuantMSE(d, bits=bits, device="cuda")
    k, v = (tq.encode(torch.randn(B, 1, n, d, device="cuda", generator=gen).bfloat16()) for _ in range(2))
    q = torch.randn(B, group, 1, d, device="cuda", generator=gen)
    got = kernels.flash_decode_compressed(q, k.indices, k.norms, v.indices, v.norms, tq.quantizer.levels,
                                          tq.quantizer.levels, tq.rotation.signs, d ** -0.5, bits, bits,
                                          q_is_rotated=False)
    kd, vd = tq.decode(k).double(), tq.decode(v).double()
    ref = ((q.double() @ kd.transpose(-1, -2)) * d ** -0.5).softmax(-1) @ vd
    err = (got.double() - ref).norm(dim=-1) / ref.norm(dim=-1)
    # fp32 scores of a few units, exponentials and sums over 2000 tokens; the decoded vectors are fp32
    assert err.max().item() < 2e-5
