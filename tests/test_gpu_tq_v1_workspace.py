"""Scratch of the slot-format decode: a call that supplies its buffers allocates nothing unless the kernel that streams whole
pages runs, that kernel takes the caller's workspace, and without memory for one the item kernels answer."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(D=128, kb=4, hkv=8, group=4, B=16, splits=8, layers=1, dtype=torch.bfloat16):
    from fused_turboquant_b200 import TurboQuantMSE, tq_v1
    cfg = tq_v1.TurboQuantSlotConfig(D, kb, 4)
    cent, mids = tq_v1.midpoints_of(TurboQuantMSE(D, bits=kb if kb < 8 else 4, device="cuda").quantizer.levels)
    cent = cent.cpu().numpy()
    g = torch.Generator("cuda").manual_seed(B + hkv)
    cache = torch.zeros(layers, 3 * B, 16, hkv, cfg.slot_size_aligned, dtype=torch.uint8, device="cuda")
    for layer in range(layers):
        kv = torch.randn(2, 48 * B, hkv, D, device="cuda", generator=g).bfloat16()
        tq_v1.launch_store(kv[0], kv[1], cache[layer], torch.arange(48 * B, device="cuda"), mids, cfg)
    table = torch.arange(3 * B, dtype=torch.int32, device="cuda").view(B, 3)
    lens = torch.arange(B, dtype=torch.int32, device="cuda") % 48 + 1
    q = torch.randn(layers, B, hkv * group, D, device="cuda", generator=g).to(dtype)
    mid = torch.empty(layers, B, hkv * group, splits, D + 1, device="cuda")
    out = torch.empty_like(q)

    def run(workspace=None):
        out.zero_()
        if layers == 1:
            tq_v1.decode_attention(q[0], cache[0], table, lens, cent, cfg, D ** -0.5, num_kv_splits=splits, mid_o=mid[0],
                                   output=out[0], workspace=workspace)
        else:
            tq_v1.decode_attention(q, cache, table, lens, cent, cfg, D ** -0.5, num_kv_splits=splits, mid_o=mid, output=out,
                                   workspace=workspace)
        return out.clone()
    run.bytes = tq_v1.decode_workspace_bytes(B, hkv * group, D, layers)
    return run


def _allocations(run, *args):
    run(*args)
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    run(*args)
    return torch.cuda.memory_stats()["allocation.all.allocated"] - before - 1   # (the result's clone)


@pytest.mark.parametrize("kw", [dict(dtype=torch.float32), dict(D=256), dict(hkv=4), dict(splits=7), dict(hkv=12),
                                dict(kb=8, group=8)])
def test_nothing_is_allocated_where_the_item_kernels_run(kw):
    assert _allocations(_call(**kw)) == 0


@pytest.mark.parametrize("kb", [4, 8])
def test_the_callers_workspace_is_used(kb):
    run = _call(kb=kb)
    ws = torch.empty(run.bytes, dtype=torch.uint8, device="cuda")
    assert _allocations(run) == 1 and _allocations(run, ws) == 0
    ws.fill_(0xFF)
    assert torch.equal(run(ws), run()) and ws.ne(0xFF).any()
    ws.fill_(0xFF)
    small = ws[:-1]
    assert torch.equal(run(small), run(ws[:0])) and ws.eq(0xFF).all()


def test_without_memory_for_it_the_item_kernels_answer():
    run = _call(group=8, B=16, layers=14)      # 64 MiB
    items = run(torch.empty(0, dtype=torch.uint8, device="cuda"))
    torch.cuda.empty_cache()
    spare = torch.empty(8 << 20, dtype=torch.uint8, device="cuda")     # (what run() clones into stays allowed)
    torch.cuda.set_per_process_memory_fraction(0.0)
    fill = []
    try:
        with pytest.raises(torch.OutOfMemoryError):
            while True:
                fill.append(torch.empty(2 << 20, dtype=torch.uint8, device="cuda"))
        del spare
        got = run()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, items)
