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


# (batches that leave units cut by shares' ends, units within a share, and CTAs without work)
BIG, SMALL = [5000, 3100, 4096, 77] * 12, [900, 33]


def test_one_uninitialised_workspace_serves_calls_of_different_shapes():
    """The kernel clears the counters in the workspace tail itself: garbage there is harmless, and so is
    alternating between shapes whose tails lie at different places of one buffer."""
    runs = []
    for lens, seed in ((BIG, 1), (SMALL, 2)):
        pool, bt, sl, q = _batch(lens, seed)
        runs.append((pool, q, bt, sl, max(lens)))
    need = max(p.workspace_bytes(q.shape[0], q.shape[1], top, 1) for p, q, _, _, top in runs)
    ws = torch.randint(0, 256, (need,), dtype=torch.uint8, device="cuda")
    ws[-8192:] = 0xFF
    want = [_run(*r) for r in runs]
    assert all(torch.isfinite(w).all() for w in want)
    for i in (0, 1, 0, 1, 1, 0):
        assert torch.equal(_run(*runs[i], ws=ws), want[i])


@pytest.mark.parametrize("lens", [BIG, SMALL, [60] * 1100])
def test_replays_of_a_captured_call(lens):
    """A captured launch carries its epoch with it (both launches of 1100 sequences the same one)."""
    pool, bt, sl, q = _batch(lens, 4)
    qs = [q, q.flip(0).contiguous(), -q]
    eager = [_run(pool, x, bt, sl, max(lens)) for x in qs]
    q_static, out = q.clone(), torch.empty(q.shape, dtype=torch.float32, device="cuda")
    ws = torch.empty(pool.workspace_bytes(q.shape[0], q.shape[1], max(lens), 1), dtype=torch.uint8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pool.decode_attention(q_static, bt, sl, max(lens), layer=0, out=out, workspace=ws)
    for i in (1, 2, 0, 2):
        q_static.copy_(qs[i])
        graph.replay()
        graph.replay()          # back to back: the second replay starts from the first one's leftovers
        assert torch.equal(out, eager[i]), f"replay with query set {i}"
