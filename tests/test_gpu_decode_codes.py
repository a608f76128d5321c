"""The tensor-core decode kernel over every pair of code widths (how codes become centroids differs with the width of the
keys, of the values, whether both share a codebook, the head size and the GQA group) and over its two ways to split
a batch: a cluster of CTAs per (sequence, KV head) unit, equal shares of all units."""
import ctypes

import numpy as np
import pytest
import torch

from test_gpu_guards import _filled_pool
from test_gpu_stream_plan import _oracle_bad

pytestmark = pytest.mark.gpu

# at the edges of a page, of a stage of two pages, of a round of all warps
LENS = [1, 15, 17, 32, 33, 255, 513, 16 * 24 + 1]


def _decode(pool, bt, lens, q):
    out = torch.empty(q.shape, dtype=torch.float32, device="cuda")
    pool.decode_attention(q, torch.from_numpy(bt).cuda(), torch.tensor(lens, dtype=torch.int32).cuda(), max(lens), layer=0, out=out)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("times", [1, 10])      # 16 units: clusters; 160 units: equal shares
@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("group", [3, 7])
@pytest.mark.parametrize("bk", [2, 3, 4])
@pytest.mark.parametrize("bv", [2, 3, 4])
def test_code_widths(oracle, d, group, bk, bv, times):
    lens = LENS * times
    pool, bt, key, val, _, _ = _filled_pool(d, bk, bv, 2, lens, seed=d + bk + bv)
    g = torch.Generator("cpu").manual_seed(group)
    q = torch.randn(len(lens), 2 * group, d, generator=g).bfloat16().cuda()
    got = _decode(pool, bt, lens, q)
    assert np.isfinite(got).all()
    which = sorted({*range(8), *range(len(lens) - 8, len(lens))})
    # (the gate is that of the 16-bit operands: 1e-3 + 2e-3 |ref|)
    assert _oracle_bad(oracle, pool, key, val, q, np.array(lens), got, d, bk, bv, which) == 0


@pytest.mark.parametrize("n_seq", [1, 7, 9, 16, 17, 36, 38, 74, 75])
def test_cluster_sizes(oracle, n_seq):
    """Two KV heads: 2 to 150 units, i.e. clusters of 8, 4, 2 and 1 CTAs and equal shares; sequences without tokens,
    with fewer pages than a cluster has parts, and the longest at the end."""
    d, group, bits = 128, 4, 4
    lens = [([0, 1, 130, 16, 900][i % 5]) for i in range(n_seq - 1)] + [3000]
    pool, bt, key, val, _, _ = _filled_pool(d, bits, bits, 2, lens, seed=n_seq)
    g = torch.Generator("cpu").manual_seed(n_seq)
    q = torch.randn(n_seq, 2 * group, d, generator=g).bfloat16().cuda()
    got = _decode(pool, bt, lens, q)
    np.testing.assert_array_equal(got, _decode(pool, bt, lens, q))
    for b, n in enumerate(lens):
        assert n or (got[b] == 0).all()
    which = [b for b, n in enumerate(lens) if n][-6:]
    assert _oracle_bad(oracle, pool, key, val, q, np.array(lens), got, d, bits, bits, which) == 0


@pytest.mark.parametrize("times", [1, 30])
def test_a_block_id_outside_the_pool(times):
    """Its sequence comes back as NaN, the others as before, and the status word says so (30 times: equal shares)."""
    lens = [700, 1300, 90] * times
    pool, bt, *_, used = _filled_pool(128, 4, 4, 2, lens)
    q = torch.randn(len(lens), 8, 128, generator=torch.Generator("cpu").manual_seed(5)).bfloat16().cuda()
    good = _decode(pool, bt, lens, q)
    assert pool.decode_status() == 0
    pool.num_blocks = used           # (eight blocks more are allocated)
    bad = bt.copy()
    bad[1, 3] = used + 2
    got = _decode(pool, bad, lens, q)
    assert np.isnan(got[1]).all() and pool.decode_status() == 1
    rest = [b for b in range(len(lens)) if b != 1]
    np.testing.assert_array_equal(got[rest], good[rest])


@pytest.mark.parametrize("G", [4, 8])
def test_an_expired_wait_of_equal_shares(G):
    """The give-up path with a batch that is cut into equal shares: 160 units (see test_gpu_wait_expiry.py)."""
    from test_gpu_wait_expiry import _test_lib

    from fused_turboquant_b200 import _lib
    d, bits, Hkv, lens = 128, 4, 2, [4096] * 80
    pool, bt, *_ = _filled_pool(d, bits, bits, Hkv, lens)
    q = torch.randn(len(lens), Hkv * G, d, generator=torch.Generator("cpu").manual_seed(9)).bfloat16().cuda()
    sl, table = torch.tensor(lens, dtype=torch.int32).cuda(), torch.from_numpy(bt).cuda()
    ws = torch.empty(pool.workspace_bytes(len(lens), Hkv * G, 4096, 1), dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def run(lib):
        out = torch.full(q.shape, 7.0, dtype=torch.float32, device="cuda")
        rc = lib.ftq_paged_decode_attn(
            p(q), _lib.BF16, p(out), _lib.F32, p(pool.pool[0]), pool.num_blocks, pool.layer_stride, 1, p(table),
            table.shape[1], p(sl), 4096, len(lens), Hkv * G, Hkv, d, bits, bits, _lib.fptr(pool.levels_k),
            _lib.fptr(pool.levels_v), _lib.fptr(pool.signs), d ** -0.5, p(ws), ws.numel(), stream)
        assert rc == 0, lib.ftq_last_error()
        status = ctypes.c_int(-1)
        rc = lib.ftq_paged_decode_status(p(ws), len(lens), Hkv * G, Hkv, d, 4096, 1, stream, ctypes.byref(status))
        return out.cpu().numpy(), rc, status.value

    good, rc, status = run(_lib.load())
    assert (rc, status) == (0, 0) and np.isfinite(good).all()
    got, rc, status = run(_test_lib())
    assert (rc, status) == (-5, 2)
    units = got.reshape(len(lens), Hkv, G, d)
    poisoned = np.isnan(units).any(axis=(2, 3))
    assert poisoned.sum() == 1 and np.isnan(units[poisoned]).all()
    np.testing.assert_array_equal(units[~poisoned], good.reshape(units.shape)[~poisoned])
    again, rc, status = run(_lib.load())
    assert (rc, status) == (0, 0)
    np.testing.assert_array_equal(again, good)


@pytest.mark.parametrize("G", [4, 8])
@pytest.mark.parametrize("n_seq", [3, 80])      # clusters, equal shares
def test_an_epoch_that_nobody_sees(G, n_seq):
    """CTA 0 does not publish its epoch (in the test library): nobody may use the counters of the cut units, which come back
    as NaN; units that one half or one cluster has finished need none and are as ever."""
    from test_gpu_wait_expiry import _test_lib

    from fused_turboquant_b200 import _lib
    d, Hkv, lens = 128, 2, [4096 - 1000 * (i % 3) for i in range(n_seq)]
    pool, bt, *_ = _filled_pool(d, 4, 4, Hkv, lens)
    q = torch.randn(n_seq, Hkv * G, d, generator=torch.Generator("cpu").manual_seed(9)).bfloat16().cuda()
    sl, table = torch.tensor(lens, dtype=torch.int32).cuda(), torch.from_numpy(bt).cuda()
    ws = torch.empty(pool.workspace_bytes(n_seq, Hkv * G, 4096, 1), dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def run(lib):
        out = torch.full(q.shape, 7.0, dtype=torch.float32, device="cuda")
        rc = lib.ftq_paged_decode_attn(
            p(q), _lib.BF16, p(out), _lib.F32, p(pool.pool[0]), pool.num_blocks, pool.layer_stride, 1, p(table),
            table.shape[1], p(sl), 4096, n_seq, Hkv * G, Hkv, d, 4, 4, _lib.fptr(pool.levels_k),
            _lib.fptr(pool.levels_v), _lib.fptr(pool.signs), d ** -0.5, p(ws), ws.numel(), stream)
        assert rc == 0, lib.ftq_last_error()
        status = ctypes.c_int(-1)
        rc = lib.ftq_paged_decode_status(p(ws), n_seq, Hkv * G, Hkv, d, 4096, 1, stream, ctypes.byref(status))
        return out.cpu().numpy().reshape(n_seq, Hkv, G, d), rc, status.value

    good, rc, status = run(_lib.load())
    assert (rc, status) == (0, 0) and np.isfinite(good).all()
    lib = _test_lib()
    assert lib.ftq_test_withhold_epoch(1) == 0
    try:
        got, rc, status = run(lib)
    finally:
        assert lib.ftq_test_withhold_epoch(0) == 0
    assert (rc, status) == (-5, 2)
    poisoned = np.isnan(got).any(axis=(2, 3))
    assert np.isnan(got[poisoned]).all()
    np.testing.assert_array_equal(got[~poisoned], good[~poisoned])
    # (160 units of up to 284 places on 296 halves: shares are shorter than most units)
    assert poisoned.sum() > poisoned.size // 2 if n_seq == 80 else not poisoned.any()
    again, rc, status = run(_lib.load())
    assert (rc, status) == (0, 0)
    np.testing.assert_array_equal(again, good)


@pytest.mark.parametrize("times", [1, 40])      # clusters, equal shares
@pytest.mark.parametrize("d,bk,bv,G", [(128, 4, 4, 4), (128, 3, 3, 8), (64, 2, 3, 7), (256, 4, 2, 2)])
@pytest.mark.parametrize("pages", ["first", "last", "all"])
def test_keys_that_are_not_numbers(times, d, bk, bv, G, pages):
    """Pages of nothing but NaN key norms are not taken for pages without tokens: the (sequence, KV head) they belong to is
    NaN, the others are as before."""
    lens = [1, 16, 17, 40, 200, 700] * times
    pool, bt, *_ = _filled_pool(d, bk, bv, 2, lens)
    q = torch.randn(len(lens), 2 * G, d, generator=torch.Generator("cpu").manual_seed(5)).bfloat16().cuda()
    good = _decode(pool, bt, lens, q).reshape(len(lens), 2, G, d)
    for b in range(0, len(lens), 2):
        last = (lens[b] + 15) // 16
        for page in {"first": [0], "last": [last - 1], "all": range(last)}[pages]:
            norms = pool.pool[0, int(bt[b, page]), 1, 2 * d * bk:2 * d * bk + 32]
            norms.copy_(torch.full((16,), float("nan"), dtype=torch.float16).view(torch.uint8))
    got = _decode(pool, bt, lens, q).reshape(good.shape)
    assert np.isnan(got[::2, 1]).all()
    np.testing.assert_array_equal(got[:, 0], good[:, 0])
    np.testing.assert_array_equal(got[1::2], good[1::2])
    assert pool.decode_status() == 0


@pytest.mark.parametrize("d,bk,bv,G", [(128, 4, 4, 4), (64, 2, 3, 12), (256, 4, 2, 1)])
@pytest.mark.parametrize("S", [1, 16, 40, 700])
@pytest.mark.parametrize("where", ["first page", "all"])
def test_keys_that_are_not_numbers_fp32(d, bk, bv, G, S, where):
    """The same for the fp32 kernel, from contiguous tensors and from the pool: one (sequence, KV head) is NaN."""
    from fused_turboquant_b200 import TurboQuantMSE, kernels
    g = torch.Generator("cuda").manual_seed(S)
    x = torch.randn(2, 2, 2, S, d, device="cuda", generator=g)
    tk, tv = TurboQuantMSE(d, bits=bk, device="cuda"), TurboQuantMSE(d, bits=bv, device="cuda")
    k, v = tk.encode(x[0]), tv.encode(x[1])
    q = torch.randn(2, 2 * G, 1, d, device="cuda", generator=g)
    n = min(16, S) if where == "first page" else S

    def flash():
        return kernels.flash_decode_compressed(
            q, k.indices, k.norms, v.indices, v.norms, tk.quantizer.levels, tv.quantizer.levels, tk.rotation.signs,
            d ** -0.5, bk, bv).reshape(2, 2, G, d)
    good = flash()
    k.norms[1, 0, :n] = float("nan")
    got = flash()
    assert torch.isnan(got[1, 0]).all()
    assert torch.equal(got[0], good[0]) and torch.equal(got[1, 1], good[1, 1])

    pool, bt, *_ = _filled_pool(d, bk, bv, 2, [S, S])
    good = _decode(pool, bt, [S, S], q[:, :, 0]).reshape(2, 2, G, d)
    for page in range((n + 15) // 16):
        norms = pool.pool[0, int(bt[1, page]), 0, 2 * d * bk:2 * d * bk + 32]
        norms.copy_(torch.full((16,), float("nan"), dtype=torch.float16).view(torch.uint8))
    got = _decode(pool, bt, [S, S], q[:, :, 0]).reshape(2, 2, G, d)
    assert np.isnan(got[1, 0]).all() and pool.decode_status() == 0
    np.testing.assert_array_equal(got[0], good[0])
    np.testing.assert_array_equal(got[1, 1], good[1, 1])


def _time_of_calls(pool, bt, lens, q):
    """Microseconds of a call among twenty in a graph, the least of ten replays."""
    table, sl = torch.from_numpy(bt).cuda(), torch.tensor(lens, dtype=torch.int32).cuda()
    out = torch.empty_like(q)
    ws = torch.empty(pool.workspace_bytes(q.shape[0], q.shape[1], max(lens), 1), dtype=torch.uint8, device="cuda")
    call = lambda: pool.decode_attention(q, table, sl, max(lens), layer=0, out=out, workspace=ws)
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(20):
            call()
    times = []
    for _ in range(10):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) * 50)
    return min(times)


def test_many_short_sequences_use_the_whole_device():
    """Twice the units of a device of 148 SMs, a page each, in equal shares: not much more than one unit per SM in clusters
    (three times as much where their pages alone sized the grid)."""
    times = []
    for n_seq in (140, 280):
        pool, bt, *_ = _filled_pool(64, 4, 3, 1, [8] * n_seq)
        times.append(_time_of_calls(pool, bt, [8] * n_seq, torch.randn(n_seq, 4, 64, device="cuda").bfloat16()))
    assert times[1] < 2 * times[0], times


@pytest.mark.parametrize("longest", [24 * 16, 24 * 16 + 1, 32 * 16, 32 * 16 + 1])
@pytest.mark.parametrize("mix", ["alike", "ragged", "mostly empty"])
@pytest.mark.parametrize("d,bits,group,n_seq", [(128, 4, 4, 80), (64, 3, 8, 100), (256, 4, 1, 75), (128, 4, 4, 400)])
def test_short_units_are_not_cut(d, bits, group, n_seq, mix, longest):
    """150 to 800 units on either side of the lengths (24 pages for heads of 256, else 32) from which units are cut, alike (as many to each half) and ragged (shares
    that start inside a unit, that hold none, and sequences without tokens), against the fp32 kernel."""
    r = np.random.default_rng(n_seq)
    lens = np.full(n_seq, longest) if mix == "alike" else r.integers(1, longest + 1, n_seq)
    if mix == "mostly empty":
        lens[r.random(n_seq) < 0.7] = 0
    lens[n_seq // 2] = longest
    lens = [int(n) for n in lens]
    pool, bt, *_ = _filled_pool(d, bits, bits, 2, lens, seed=n_seq)
    q = torch.randn(n_seq, 2 * group, d, generator=torch.Generator("cpu").manual_seed(3)).bfloat16().cuda()
    got, ref = _decode(pool, bt, lens, q), _decode(pool, bt, lens, q.float())
    np.testing.assert_array_equal(got, _decode(pool, bt, lens, q))
    some = np.array(lens) > 0
    assert (got[~some] == 0).all()
    # 16-bit operands: 3e-4 in the middle of a call, the bar is that of test_gpu_stream_plan.py
    err = np.linalg.norm(got - ref, axis=-1)[some] / np.linalg.norm(ref, axis=-1)[some]
    assert err.max() < 1e-2


@pytest.mark.parametrize("d,bits,group", [(128, 4, 8), (128, 3, 5), (64, 4, 7), (64, 2, 1), (256, 4, 8), (256, 3, 3)])
@pytest.mark.parametrize("n_seq,top", [(1, 40000), (3, 20000), (40, 12000)])
def test_units_of_many_parts(d, bits, group, n_seq, top):
    """Few long sequences, cut into more parts than a merge takes up at a time, among sequences of a few parts and of one; two
    runs of the same call are the same whoever merges what."""
    lens = [max(1, top // (1 + 7 * (i % 5))) for i in range(n_seq)]
    pool, bt, *_ = _filled_pool(d, bits, bits, 1, lens, seed=top)
    q = torch.randn(n_seq, group, d, generator=torch.Generator("cpu").manual_seed(3)).bfloat16().cuda()
    got, ref = _decode(pool, bt, lens, q), _decode(pool, bt, lens, q.float())
    for _ in range(5):
        np.testing.assert_array_equal(got, _decode(pool, bt, lens, q))
    err = np.linalg.norm(got - ref, axis=-1) / np.linalg.norm(ref, axis=-1)
    assert err.max() < 1e-2        # (16-bit operands, as above)


def test_the_merge_of_many_parts_keeps_up_with_the_heads():
    """Eight heads of a long sequence against four: the pages are the same, the rows to merge twice as many (1.8 times the time
    with an octet a head, two rows at a time)."""
    lens, times = [131072], []
    pool, bt, *_ = _filled_pool(128, 4, 4, 1, lens)
    for group in (4, 8):
        times.append(_time_of_calls(pool, bt, lens, torch.randn(1, group, 128, device="cuda").bfloat16()))
    assert times[1] < 1.5 * times[0], times


@pytest.mark.parametrize("over", [0, 1])         # clusters up to here, equal shares from one token more on
@pytest.mark.parametrize("d,group,n_seq,line", [
    (64, 7, 4, 112 * 8 * 2), (128, 4, 4, 112 * 8 * 2), (64, 4, 13, 72 * 4 * 2), (128, 8, 74, 72 * 2), (256, 2, 4, 112 * 8)])
def test_the_lines_between_clusters_and_equal_shares(oracle, d, group, n_seq, line, over):
    """Two KV heads; line = pages of the longest context (pages of a half's part, CTAs, halves), the others far shorter:
    parts without pages, shares that end among a unit's extra places, halves without pages."""
    bits = 4
    lens = [([16, 0, 700, 1, 33, 16 * 28][i % 6]) for i in range(n_seq - 1)] + [line * 16 + over]
    pool, bt, key, val, _, _ = _filled_pool(d, bits, bits, 2, lens, seed=n_seq)
    g = torch.Generator("cpu").manual_seed(n_seq + d)
    q = torch.randn(n_seq, 2 * group, d, generator=g).bfloat16().cuda()
    got = _decode(pool, bt, lens, q)
    assert np.isfinite(got).all()
    np.testing.assert_array_equal(got, _decode(pool, bt, lens, q))
    for b, n in enumerate(lens):
        assert n or (got[b] == 0).all()
    which = [b for b, n in enumerate(lens) if n][-6:]
    assert _oracle_bad(oracle, pool, key, val, q, np.array(lens), got, d, bits, bits, which) == 0
