"""Sizes that callers plan with: what a decode call needs as scratch (CPU: the planner runs on the host)."""
import pytest

STATIC_SCRATCH = 8 << 20


@pytest.mark.parametrize("B,Hq,Hkv,d,ctx,layers", [
    (471, 8, 8, 64, 64, 8), (473, 2, 2, 64, 299, 32), (947, 1, 1, 64, 76, 32), (47, 8, 8, 64, 59, 80),
    (1966, 1, 1, 128, 20, 8),
])
def test_batches_of_short_contexts_fit_the_built_in_scratch(B, Hq, Hkv, d, ctx, layers):
    """One chunk per context: a row of d + 4 floats per query head and one counter per (layer, sequence,
    KV head) next to the 256-byte header, all within the 8 MiB that ftq_paged_decode_attn_static has."""
    from fused_turboquant_b200 import _lib
    need = _lib.load().ftq_decode_workspace_bytes(B, Hq, Hkv, d, ctx, layers)
    rows, counters = layers * B * Hq * (d + 4) * 4, 256 + layers * B * Hkv * 4
    assert rows + counters <= need <= rows + (counters + 255) // 256 * 256 <= STATIC_SCRATCH
