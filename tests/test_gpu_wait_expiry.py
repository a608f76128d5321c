"""The give-up path of the decode kernels' bounded waits, executed on purpose.

Every wait in device code has a poll limit; a wait that runs out marks the rows concerned NaN, sets
a bit in the call's status word and lets the kernel finish.  In the product library that path
only runs when a copy is lost, so this test uses the second library the build script makes
(`libftq_b200_waittest.so`): identical, except that in the head_dim-128 decode kernels warp 5 of
CTA 0 announces its first page copy to the mbarrier without issuing it, and the poll limit is 64.
Nothing faults, traps or spins without bound: the wait simply expires.
"""
import ctypes
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _test_lib():
    from fused_turboquant_b200 import _lib, build
    if not os.path.exists(build.TEST_LIB_PATH):
        pytest.skip("libftq_b200_waittest.so has not been built")
    lib = ctypes.CDLL(build.TEST_LIB_PATH)
    for name, (res, args) in _lib.SIGNATURES.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    return lib


@pytest.mark.parametrize("G", [4, 8])   # streaming kernel / equal-share kernel
def test_an_expired_wait_poisons_its_rows_and_nothing_else(G):
    from fused_turboquant_b200 import PagedKVPool, _lib
    bad_lib, good_lib = _test_lib(), _lib.load()
    d, bk, bv, Hkv = 128, 4, 4, 2
    # equal lengths: every work item exists and is long enough for warp 5 to own a page of it,
    # whichever item CTA 0 draws first
    seq_lens = [4096, 4096, 4096]
    B = len(seq_lens)
    max_blocks = (max(seq_lens) + 15) // 16
    rng = np.random.default_rng(3)
    bt = torch.from_numpy(rng.permutation(B * max_blocks).reshape(B, max_blocks).astype(np.int32)).cuda()
    pool = PagedKVPool(B * max_blocks, Hkv, d, bk, bv, n_layers=1, device="cuda")
    g = torch.Generator("cpu").manual_seed(9)
    n_tok = sum(seq_lens)
    key = torch.randn(n_tok, Hkv, d, generator=g).bfloat16().cuda()
    val = torch.randn(n_tok, Hkv, d, generator=g).bfloat16().cuda()
    slots = torch.cat([bt[b, torch.arange(s, device="cuda") // 16].long() * 16 +
                       torch.arange(s, device="cuda") % 16 for b, s in enumerate(seq_lens)])
    pool.store(key, val, slots, layer=0)
    q = torch.randn(B, Hkv * G, d, generator=g).bfloat16().cuda()
    sl = torch.tensor(seq_lens, dtype=torch.int32).cuda()
    ws = torch.empty(pool.workspace_bytes(B, Hkv * G, max(seq_lens), 1), dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def run(lib):
        out = torch.full(q.shape, 7.0, dtype=torch.float32, device="cuda")
        rc = lib.ftq_paged_decode_attn(
            p(q), _lib.BF16, p(out), _lib.F32, p(pool.pool[0]), pool.num_blocks, pool.layer_stride, 1,
            p(bt), bt.shape[1], p(sl), max(seq_lens), B, Hkv * G, Hkv, d, bk, bv,
            _lib.fptr(pool.levels_k), _lib.fptr(pool.levels_v), _lib.fptr(pool.signs), d ** -0.5,
            p(ws), ws.numel(), stream)
        assert rc == 0, lib.ftq_last_error()
        bits = ctypes.c_int(-1)
        rc = lib.ftq_paged_decode_status(p(ws), B, Hkv * G, Hkv, d, max(seq_lens), 1, stream,
                                         ctypes.byref(bits))
        return out.cpu().numpy(), rc, bits.value

    good, rc, bits = run(good_lib)
    assert rc == 0 and bits == 0 and np.isfinite(good).all()

    got, rc, bits = run(bad_lib)          # returns: the wait gave up after its 64 polls
    assert rc == -5 and bits == 2, (rc, bits)
    # exactly one (sequence, KV head) unit -- the one whose chunk CTA 0 started with -- is
    # poisoned, all of its rows; every other unit is untouched by the lost copy
    units = got.reshape(B, Hkv, G, d)
    poisoned = np.isnan(units).any(axis=(2, 3))
    assert poisoned.sum() == 1, poisoned
    assert np.isnan(units[poisoned]).all()
    np.testing.assert_array_equal(units[~poisoned], good.reshape(B, Hkv, G, d)[~poisoned])

    again, rc, bits = run(good_lib)       # the context is as usable as before
    assert rc == 0 and bits == 0
    np.testing.assert_array_equal(again, good)


def test_an_expired_wait_of_the_chunk_kernel_poisons_its_rows_and_nothing_else():
    """One dequantising warp of CTA (0, 0, 0) does not report its second tile: the CTA gives up (its MMAs
    drained, TMEM freed), the 256 rows it works on are NaN, the rest of the call is untouched."""
    from fused_turboquant_b200 import PagedKVPool, _lib
    bad_lib, good_lib = _test_lib(), _lib.load()
    d, bits, Hkv, G, B, q_len, n = 128, 4, 2, 4, 2, 100, 2000
    per = (n + 15) // 16
    g = torch.Generator("cuda").manual_seed(9)
    bt = torch.randperm(B * per, device="cuda", generator=g).int().view(B, per)
    pool = PagedKVPool(B * per, Hkv, d, bits, bits, n_layers=1, device="cuda")
    pos = torch.arange(n, device="cuda")
    for b in range(B):
        kv = torch.randn(2, n, Hkv, d, device="cuda", generator=g).bfloat16()
        pool.store(kv[0], kv[1], bt[b, pos // 16].long() * 16 + pos % 16, layer=0)
    q = torch.randn(B, q_len, Hkv * G, d, device="cuda", generator=g).bfloat16()
    sl = torch.full((B,), n, dtype=torch.int32, device="cuda")
    need = good_lib.ftq_paged_chunk_workspace_bytes(B, q_len, Hkv * G, Hkv, d, n)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def run(lib):
        out = torch.full(q.shape, 7.0, dtype=torch.float32, device="cuda")
        rc = lib.ftq_paged_chunk_attn(
            p(q), _lib.BF16, p(out), _lib.F32, p(pool.pool[0]), pool.num_blocks, p(bt), per, p(sl), n, B,
            q_len, Hkv * G, Hkv, d, bits, bits, _lib.fptr(pool.levels_k), _lib.fptr(pool.levels_v),
            _lib.fptr(pool.signs), d ** -0.5, p(ws), ws.numel(), stream)
        assert rc == 0, lib.ftq_last_error()
        status = ctypes.c_int(-1)
        rc = lib.ftq_paged_decode_status(p(ws), 1, Hkv * G, Hkv, d, n, 1, stream, ctypes.byref(status))
        return out, rc, status.value

    good, rc, status = run(good_lib)
    assert rc == 0 and status == 0 and torch.isfinite(good).all()
    got, rc, status = run(bad_lib)
    assert rc == -5 and status == 2, (rc, status)
    lost = torch.zeros(B, q_len, Hkv * G, dtype=torch.bool, device="cuda")
    lost[0, :256 // G, :G] = True                 # two row tiles: 64 queries of KV head 0's group
    assert torch.isnan(got[lost]).all()
    assert torch.equal(got[~lost], good[~lost])
    again, rc, status = run(good_lib)
    assert rc == 0 and status == 0 and torch.equal(again, good)


@pytest.mark.parametrize("G", [4, 8])
def test_an_expired_wait_of_the_slot_decode_by_shares_is_nan_everywhere(G):
    """The first page of CTA 0 is announced but not copied: its warps and the producer give up, and the merge, which can
    not know whose rows are missing, returns NaN for the call."""
    from fused_turboquant_b200 import TurboQuantMSE, _lib, tq_v1
    bad_lib, good_lib = _test_lib(), _lib.load()
    d, Hkv, B, n, splits = 128, 8, 16, 700, 8
    cfg = tq_v1.TurboQuantSlotConfig(d, 4, 4)
    cent, mids = tq_v1.midpoints_of(TurboQuantMSE(d, bits=4, device="cuda").quantizer.levels)
    g = torch.Generator("cuda").manual_seed(2)
    per = (n + 15) // 16
    bt = torch.randperm(B * per, device="cuda", generator=g).int().view(B, per)
    cache = torch.zeros(B * per, 16, Hkv, cfg.slot_size_aligned, dtype=torch.uint8, device="cuda")
    kv = torch.randn(2, B * per * 16, Hkv, d, device="cuda", generator=g).bfloat16()
    tq_v1.launch_store(kv[0], kv[1], cache, torch.arange(B * per * 16, device="cuda"), mids, cfg)
    q = torch.randn(B, Hkv * G, d, device="cuda", generator=g).bfloat16()
    sl = torch.full((B,), n, dtype=torch.int32, device="cuda")
    ws = torch.empty(tq_v1.decode_workspace_bytes(B, Hkv * G, d), dtype=torch.uint8, device="cuda")
    mid = torch.empty(B, Hkv * G, splits, d + 1, device="cuda")
    levels = cent.cpu().numpy().astype(np.float32)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def run(lib):
        out = torch.full(q.shape, 7.0, dtype=torch.float32, device="cuda")
        rc = lib.ftq_tq_decode_layers_ws(
            p(q), _lib.BF16, B, Hkv * G, Hkv, d, p(cache), *cache.stride()[:3], 16, p(bt), per, p(sl), None, 4, 4, 1, 0, 0,
            _lib.fptr(levels), d ** -0.5, splits, p(mid), p(out), _lib.F32, None, None, 0, None, 1, 0, B * per, p(ws),
            ws.numel(), stream)
        assert rc == 0, lib.ftq_last_error()
        torch.cuda.synchronize()
        return out

    good = run(good_lib)
    assert torch.isfinite(good).all()
    assert torch.isnan(run(bad_lib)).all()
    assert torch.equal(run(good_lib), good)
