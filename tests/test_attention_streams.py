"""How prompt portions are cut for the tcgen05 attention (host only), and its two ways of taking a tile, rows of the
streams' own and shared rows, at the edges of both."""
from __future__ import annotations

import pytest
import torch

from mrun_b200.engine.batch import SegmentInfo
from mrun_b200.kernels import attention


class Step:
    def __init__(self, portions):
        self.segments, self.shared, row = [], {}, 0
        for slot, (before, n) in enumerate(portions):
            self.segments.append(SegmentInfo(slot, row, n, before))
            row += n

    def upload(self, host):
        return torch.from_numpy(host.copy())


@pytest.mark.parametrize("streams", [1, 2])
@pytest.mark.parametrize("window", [0, 200, -256])
@pytest.mark.parametrize("tokens,portions", [(32, [(0, 17)]), (32, [(9000, 1531)]), (128, [(0, 129), (700, 128), (5, 1)]),
                                             (1, [(3, 40)]), (18, [(0, 2048), (1000, 37), (10, 8)])])
def test_blocks_cover_every_token_once(streams, window, tokens, portions):
    step = Step(portions)
    first, count, n = attention.tc5_tiles(step, tokens, 8, streams, window, 148 / 8)
    seen = []
    for at, c in zip(first.tolist(), count.tolist()):
        assert 0 < c <= streams * tokens
        assert any(seg.q_start <= at and at + c <= seg.q_start + seg.q_len for seg in step.segments)
        seen += range(at, at + c)
    assert len(first) == n and sorted(seen) == [t for seg in step.segments if seg.q_len > 8
                                                for t in range(seg.q_start, seg.q_start + seg.q_len)]


def test_a_step_without_long_portions_has_no_blocks():
    assert attention.tc5_tiles(Step([(0, 8), (5, 1)]), 32, 8, 2, 0, 18.5) == (None, None, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("pair_cost", [0.01, 100.0])             # every tile that can be a pair is one; none is
@pytest.mark.parametrize("heads,kv_heads,head_dim,window", [(8, 2, 128, 0), (4, 4, 64, 0), (6, 2, 128, 130), (16, 1, 64, 0)])
def test_both_ways_at_their_edges(monkeypatch, pair_cost, heads, kv_heads, head_dim, window):
    """Portions one token short of, at and past a stream's rows and a pair's, contexts that end at and around a key tile, so
    that streams have one tile, none, or unlike numbers of them."""
    from mrun_b200.kernels import lib, ops
    from test_attention_gpu import DEV, Case
    from test_attention_tc5_gpu import reference
    monkeypatch.setattr(attention, "TC5_PAIR_TILE", pair_cost)
    per = 128 // (heads // kv_heads)
    segments = [(0, per - 1), (0, per), (1, per + 1), (127, 2 * per - 1), (128, 2 * per), (255, 2 * per + 1), (129, per)]
    case = Case(segments, heads, kv_heads, head_dim, 16, torch.bfloat16, seed=5, window=window)
    assert attention.prefill_uses_tcgen05(lib.attention(head_dim), heads // kv_heads, 16)
    scale = head_dim ** -0.5
    out = case.run(scale).float()
    ops.tc5_check(torch.device(DEV))
    want = reference(case, scale)
    # P and the result are bfloat16: 2^-9 of the largest value that enters, about 4 standard deviations, twice
    torch.testing.assert_close(out, want, rtol=0.0, atol=2 * 4 * 2.0 ** -9)
