"""The equal-share decode kernel's launch protocol (3-bit codes and groups of 5 to 8 run on it): batches
above its 1024 sequences per launch, the counters and the status word it clears itself, replays."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

D, BITS, HKV, GROUP = 128, 3, 2, 8


def _batch(lens, seed):
    """(pool, block table, seq_lens, queries) of a batch on shuffled pages."""
    from fused_turboquant_b200 import PagedKVPool
    rng = np.random.default_rng(seed)
    lens = np.asarray(lens, np.int32)
    per = (lens + 15) // 16
    perm = rng.permutation(int(per.sum())).astype(np.int32)
    bt = np.zeros((len(lens), max(int(per.max()), 1)), np.int32)
    at = 0
    for b, n in enumerate(per):
        bt[b, :n] = perm[at:at + n]
        at += n
    slots = np.concatenate([bt[b, np.arange(n) // 16].astype(np.int64) * 16 + np.arange(n) % 16
                            for b, n in enumerate(lens)])
    gen = torch.Generator("cuda").manual_seed(seed)
    pool = PagedKVPool(int(per.sum()) + 8, HKV, D, BITS, BITS, device="cuda")
    kv = torch.randn(2, int(lens.sum()), HKV, D, device="cuda", generator=gen).bfloat16()
    pool.store(kv[0], kv[1], torch.from_numpy(slots).cuda(), layer=0)
    q = torch.randn(len(lens), HKV * GROUP, D, device="cuda", generator=gen).bfloat16()
    return pool, torch.from_numpy(bt).cuda(), torch.from_numpy(lens).cuda(), q


def _run(pool, q, bt, sl, top, ws=None):
    return pool.decode_attention(q, bt, sl, top, layer=0, workspace=ws,
                                 out=torch.empty(q.shape, dtype=torch.float32, device="cuda"))


def test_status_of_a_batch_above_one_launch():
    """1100 sequences are two launches: what either met is in the call's status word."""
    rng = np.random.default_rng(2)
    lens = rng.integers(1, 100, 1100)
    lens[[17, 1050]] = 0
    pool, bt, sl, q = _batch(lens, 3)
    top = int(lens.max())
    good = _run(pool, q, bt, sl, top)
    assert pool.decode_status() == 0
    assert torch.isfinite(good).all() and (good[[17, 1050]] == 0).all()
    # a sequence's sums do not depend on the others but for where shares end: fp32 order and fp16 weights
    ref = torch.cat([_run(pool, q[:600], bt[:600], sl[:600], top), _run(pool, q[600:], bt[600:], sl[600:], top)])
    err = (good - ref).norm(dim=-1) / ref.norm(dim=-1).clamp_min(1e-6)
    assert err.max().item() < 4e-3
    for b in (5, 1090):
        bad = bt.clone()
        bad[b, 0] = pool.num_blocks + 3
        out = _run(pool, q, bad, sl, top)
        assert pool.decode_status() == 1
        rows = torch.isnan(out).any(dim=-1).any(dim=-1)
        assert rows.nonzero().flatten().tolist() == [b] and torch.isnan(out[b]).all()
        assert torch.equal(out[~rows], good[~rows])
    _run(pool, q, bt, sl, top)
    assert pool.decode_status() == 0
