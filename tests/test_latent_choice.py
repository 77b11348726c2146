"""Which prompt steps of a latent attention make keys and values from the latents, on both sides of the line."""
from __future__ import annotations

from types import SimpleNamespace

import pytest

# heads, (tokens before, new tokens) of every segment, made: where the two forms were measured apart
STEPS = [
    (16, [(0, 64)], False), (16, [(0, 384)], False), (16, [(0, 512)], False), (16, [(0, 1024)], True), (16, [(1000, 512)], True),
    (16, [(0, 256)] * 2, False), (16, [(0, 512)] * 2, False), (16, [(0, 768)] * 2, True), (16, [(700, 760), (350, 1140)], True),
    (16, [(0, 25)] * 4, False), (16, [(0, 384)] * 4, False), (16, [(0, 500)] * 4, True), (16, [(0, 250)] * 8, False),
    (64, [(0, 64)], False), (64, [(0, 512)], True), (64, [(0, 128)] * 4, False), (64, [(0, 192)] * 8, True),
]


@pytest.mark.parametrize("heads, segments, made", STEPS)
def test_keys_and_values_are_made_where_that_costs_less(heads, segments, made):
    from mrun_b200.parts.latent_attention import LatentAttention
    part = LatentAttention.__new__(LatentAttention)
    part.spec, part.expandable, part.costly = SimpleNamespace(heads=heads), True, True
    tokens, reach = sum(n for _, n in segments), max(before + n for before, n in segments)
    ctx = SimpleNamespace(segments=[SimpleNamespace(pos_start=before, q_len=n) for before, n in segments], num_tokens=tokens,
                          max_q_len=max(n for _, n in segments), max_kv_len=reach)
    assert bool(part._scratch_rows(ctx)) == made
