"""Which steps the scans take in chunks and which they walk, and which tiles the 32-bit attention takes, on both sides of the
lines between them."""
from __future__ import annotations

from types import SimpleNamespace

import pytest

# (kind, key size, value size, heads, segments, in chunks): where the two forms were measured apart
STEPS = [
    ("decay", 128, 128, 16, [2048], True), ("gated", 128, 128, 32, [128], True), ("delta", 128, 128, 16, [396, 592, 789], True),
    ("decay", 128, 128, 4, [128], False), ("gated", 128, 128, 4, [128] * 4, False), ("decay", 128, 128, 4, [128] * 16, True),
    ("decay", 128, 128, 4, [160], True), ("delta", 128, 128, 64, [192] * 8, True), ("delta", 128, 128, 16, [191], False),
    ("decay", 64, 64, 64, [160] * 16, False), ("gated", 64, 64, 64, [160] * 16, False), ("decay", 64, 64, 4, [160] * 16, True),
    ("decay", 64, 64, 64, [128] * 16, True), ("decay", 64, 128, 64, [160] * 16, True),
    ("delta", 64, 64, 32, [192] * 8, False), ("delta", 64, 64, 64, [192] * 8, False), ("delta", 64, 64, 16, [256] * 8, False),
    ("delta", 64, 64, 64, [192], True), ("delta", 64, 64, 64, [1024] * 2, True), ("delta", 64, 64, 16, [512] * 4, True),
    ("delta", 64, 128, 64, [200, 40, 300], False), ("delta", 64, 128, 64, [192], True), ("delta", 64, 128, 32, [256] * 4, False),
    ("delta", 128, 64, 32, [300, 300, 300, 20, 30, 40], False), ("delta", 128, 64, 32, [256] * 4, True),
    ("decay", 128, 128, 16, [1024, 1, 1, 1, 1], True), ("decay", 128, 128, 16, [1024] + [1] * 16, False),
]


@pytest.mark.parametrize("kind, dim, vdim, heads, lengths, chunked", STEPS)
def test_a_step_is_walked_where_the_walk_is_the_faster_form(kind, dim, vdim, heads, lengths, chunked):
    from mrun_b200.kernels import ops
    ctx = SimpleNamespace(segments=[SimpleNamespace(q_len=n) for n in lengths], shared={}, num_segments=len(lengths),
                          max_q_len=max(lengths))
    tokens = sum(lengths)
    least = ops._chunk_least(ctx, tokens, kind == "delta", heads, dim, vdim)
    assert bool(ops._chunks(ctx, tokens, least)) == chunked


@pytest.mark.parametrize("ratio, kv_heads, portions, rows", [(4, 8, [2], 4), (4, 8, [17, 1, 1], 4), (4, 8, [33], 4), (4, 8, [100], 16),
                                                             (4, 8, [207, 310], 64), (16, 1, [2], 16), (8, 1, [150], 16), (3, 4, [400], 64), (3, 4, [300], 16)])
def test_tiles_of_the_32_bit_attention_follow_the_blocks_they_make(ratio, kv_heads, portions, rows):
    from mrun_b200.kernels.attention import f32_tile_rows
    ctx = SimpleNamespace(segments=[SimpleNamespace(q_len=n) for n in portions])
    assert f32_tile_rows(ctx, ratio, kv_heads, 148) == rows
