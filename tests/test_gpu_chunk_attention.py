"""The chunk attention kernel (continuation_attention with 16-bit queries) against the fp32 decode kernel
run on one synthetic sequence per query."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pool(d, bk, bv, hkv, lens, seed):
    from fused_turboquant_b200 import PagedKVPool
    gen = torch.Generator("cuda").manual_seed(seed)
    per = [(n + 15) // 16 for n in lens]
    ids = torch.randperm(sum(per) + 3, device="cuda", generator=gen)
    table = torch.zeros(len(lens), max(per), dtype=torch.int32, device="cuda")
    pool = PagedKVPool(sum(per) + 3, hkv, d, bk, bv, n_layers=2, device="cuda")
    at = 0
    for b, n in enumerate(lens):
        table[b, :per[b]] = ids[at:at + per[b]].int()
        pos = torch.arange(n, device="cuda")
        slots = ids[at:at + per[b]][pos // 16] * 16 + pos % 16
        kv = torch.randn(2, n, hkv, d, device="cuda", generator=gen)
        kv[..., 3] *= 6.0
        pool.store(kv[0].bfloat16(), kv[1].bfloat16(), slots, layer=1)
        at += per[b]
    return pool, table, torch.tensor(lens, dtype=torch.int32, device="cuda"), gen


# (sizes around the tiles of 32 / 64 tokens and 128 rows: fewer rows than a tile, one tile, a second
# one that is partly filled, more than the two of a CTA; contexts shorter than the chunk, one token,
# remainders of a page and of a tile; one part and many)
@pytest.mark.parametrize("d,bk,bv,hkv,group,q_len,lens,dtype", [
    (128, 4, 4, 2, 4, 5, [40, 23], "bf16"),
    (128, 4, 4, 8, 4, 64, [4096, 777, 63, 65], "bf16"),
    (128, 3, 3, 2, 8, 33, [1000, 64, 20], "fp16"),
    (128, 4, 2, 1, 1, 130, [513, 130], "bf16"),
    (128, 2, 4, 2, 7, 19, [320, 1], "fp16"),
    (64, 3, 3, 2, 7, 40, [700, 129], "bf16"),
    (64, 4, 4, 1, 1, 2, [2, 1, 8000], "fp16"),
    (64, 2, 2, 4, 8, 100, [300], "bf16"),
    (256, 4, 2, 2, 2, 64, [400, 33, 31], "bf16"),
    (256, 3, 4, 1, 8, 50, [1111, 95], "fp16"),
    (256, 4, 4, 8, 1, 3, [50, 2], "bf16"),
])
def test_matches_fp32_decode(d, bk, bv, hkv, group, q_len, lens, dtype):
    pool, table, sl, gen = _pool(d, bk, bv, hkv, lens, d + q_len)
    dt = torch.bfloat16 if dtype == "bf16" else torch.float16
    q = torch.randn(len(lens), q_len, hkv * group, d, device="cuda", generator=gen).to(dt)
    assert pool._takes_chunk_kernel(q, table, sl, max(lens), 1)
    got = pool.continuation_attention(q, table, sl, max(lens), layer=1)
    assert pool.decode_status() == 0
    ref = pool.continuation_attention(q.float(), table, sl, max(lens), layer=1)
    assert got.dtype == dt and got.shape == q.shape
    dead = (sl[:, None] - q_len + 1 + torch.arange(q_len, device="cuda")[None]) <= 0
    assert (got[dead] == 0).all()
    err = (got.float() - ref).norm(dim=-1) / ref.norm(dim=-1).clamp_min(1e-6)
    # 16-bit output (2^-9 bf16, 2^-12 fp16) and fp16 operands (queries, centroids, weights: 2^-12
    # each, of scores of a few units): 4e-3 / 2e-3 per vector with a factor of two to spare
    assert err[~dead].max().item() < (8e-3 if dtype == "bf16" else 5e-3)


def test_other_calls_stay_on_the_decode_kernel():
    pool, table, sl, gen = _pool(64, 4, 4, 1, [70], 3)
    q = torch.randn(1, 4, 16, 64, device="cuda", generator=gen).bfloat16()
    assert not pool._takes_chunk_kernel(q, table, sl, 70, 1)              # group 16
    q8 = q[:, :, :8]
    assert not pool._takes_chunk_kernel(q8.float(), table, sl, 70, 1)
    assert not pool._takes_chunk_kernel(q8, table, sl, 70, None)
    # few queries over much context; the limit, and one tile more
    assert pool._takes_chunk_kernel(q8, table, sl, 64 * 1776, 1)
    assert not pool._takes_chunk_kernel(q8, table, sl, 64 * 1776 + 1, 1)
    assert pool._takes_chunk_kernel(q8.repeat(1, 2, 1, 1), table, sl, 64 * 1776 + 1, 1)


def test_block_id_out_of_range_is_reported():
    pool, table, sl, gen = _pool(128, 4, 4, 2, [300, 300], 5)
    q = torch.randn(2, 20, 8, 128, device="cuda", generator=gen).half()
    good = pool.continuation_attention(q, table, sl, 300, layer=1)
    table[1, 2] = pool.num_blocks + 5
    out = pool.continuation_attention(q, table, sl, 300, layer=1)
    assert pool.decode_status() == 1
    assert torch.isnan(out[1]).all()
    assert torch.equal(out[0], good[0])
    table[1, 2] = 0
    pool.continuation_attention(q, table, sl, 300, layer=1)
    assert pool.decode_status() == 0


def test_a_captured_call_replays():
    pool, table, sl, gen = _pool(128, 4, 4, 2, [200], 6)
    q = torch.randn(1, 16, 8, 128, device="cuda", generator=gen).half()
    want = pool.continuation_attention(q, table, sl, 200, layer=1)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = pool.continuation_attention(q, table, sl, 200, layer=1)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want.cpu().numpy())


@pytest.mark.parametrize("d,bk,bv,group,q_len,n", [(128, 4, 4, 4, 20, 300), (64, 3, 3, 7, 40, 129),
                                                   (256, 4, 2, 1, 130, 200)])
@pytest.mark.parametrize("bad", [6e4, float("nan")])
def test_a_later_token_without_a_finite_value_norm_is_nobody_elses(d, bk, bv, group, q_len, n, bad):
    """The last two tokens' value vectors are longer than fp16 holds, or NaN: queries before them are bit
    for bit what they are with ordinary values there."""
    pool, table, sl, gen = _pool(d, bk, bv, 2, [n], d + q_len)
    q = torch.randn(1, q_len, 2 * group, d, device="cuda", generator=gen).bfloat16()
    assert pool._takes_chunk_kernel(q, table, sl, n, 1)
    good = pool.continuation_attention(q, table, sl, n, layer=1)
    key = torch.randn(2, 2, d, device="cuda", generator=gen).bfloat16()
    pos = torch.tensor([n - 2, n - 1], device="cuda")
    slots = table[0].long()[pos // 16] * 16 + pos % 16
    pool.store(key, torch.full_like(key, bad), slots, layer=1)
    got = pool.continuation_attention(q, table, sl, n, layer=1)
    assert torch.equal(got[:, :-2], good[:, :-2])
    if bad != bad:
        assert torch.isnan(got[:, -2:]).all() and pool.decode_status() == 0
    else:
        assert torch.isfinite(got).all() and not torch.equal(got[:, -2:], good[:, -2:])


def test_block_id_out_of_range_concerns_the_queries_that_attend_it():
    """The chunk's last page has a bad id: the queries whose context ends before it are untouched."""
    n, q_len = 320, 24                       # the last page holds the last 16 queries' tokens
    pool, table, sl, gen = _pool(128, 4, 4, 2, [n], 7)
    q = torch.randn(1, q_len, 8, 128, device="cuda", generator=gen).half()
    good = pool.continuation_attention(q, table, sl, n, layer=1)
    table[0, n // 16 - 1] = pool.num_blocks + 1
    out = pool.continuation_attention(q, table, sl, n, layer=1)
    assert pool.decode_status() == 1
    assert torch.equal(out[:, :8], good[:, :8])
    assert torch.isnan(out[:, 8:]).all()


@pytest.mark.parametrize("lens", [[20000, 300, 64, 1], [300] * 3 + [20000], [20000, 9000, 20000, 19000], [0, 20000, 10, 0]])
@pytest.mark.parametrize("d,hkv,group", [(128, 8, 4), (256, 4, 2)])
def test_contexts_of_different_lengths(d, hkv, group, lens):
    """One long context among short ones is cut into more parts than contexts of one length."""
    pool, table, sl, gen = _pool(d, 4, 4, hkv, lens, 11)
    q_len, top = 9, 20000
    q = torch.randn(len(lens), q_len, hkv * group, d, device="cuda", generator=gen).half()
    got = pool.continuation_attention(q, table, sl, top, layer=1)
    assert pool.decode_status() == 0
    ref = pool.continuation_attention(q.float(), table, sl, top, layer=1)
    dead = (sl[:, None] - q_len + 1 + torch.arange(q_len, device="cuda")[None]) <= 0
    assert (got[dead] == 0).all()
    err = (got.float() - ref).norm(dim=-1) / ref.norm(dim=-1).clamp_min(1e-6)
    assert err[~dead].max().item() < 5e-3     # (as in test_matches_fp32_decode)


@pytest.mark.parametrize("d,bits,lens", [(128, 4, [64, 300]), (64, 3, [1500]), (256, 2, [40] * 4)])
def test_reads_what_the_store_before_it_has_just_written(d, bits, lens):
    """The same pages stored anew and attended, time after time without a pause (the kernel is launched while the store
    drains), against the same calls one at a time."""
    pool, table, sl, gen = _pool(d, bits, bits, 2, lens, 13)
    q_len, n = 8, sum(lens)
    q = torch.randn(len(lens), q_len, 8, d, device="cuda", generator=gen).half()
    pos = torch.cat([torch.arange(k, device="cuda") for k in lens])
    row = torch.repeat_interleave(torch.arange(len(lens), device="cuda"), sl.long())
    slots = table[row, pos // 16].long() * 16 + pos % 16
    kv = torch.randn(30, 2, n, 2, d, device="cuda", generator=gen).half()

    def run(pause):
        out = []
        for key, value in kv:
            pool.store(key, value, slots, layer=1)
            pause()
            out.append(pool.continuation_attention(q, table, sl, max(lens), layer=1))
            pause()
        return torch.stack(out)

    want = run(torch.cuda.synchronize)
    assert torch.isfinite(want).all() and not torch.equal(want[0], want[1])
    for _ in range(10):
        assert torch.equal(run(lambda: None), want)
