"""The tcgen05 prompt attention gives a token the same bits however its step is dealt to blocks: as one of a pair of streams, as
a stream alone, and whatever other portions the step holds."""
from __future__ import annotations

import pytest
import torch

from test_attention_gpu import DEV, Case

pytestmark = pytest.mark.gpu
PAIRS, SINGLES = 0.01, 100.0          # us a tile of a pair: every block that can be a pair is one; none is


def run(case, monkeypatch, pair_cost, form=None, sink=None):
    from mrun_b200.kernels import attention, ops
    if pair_cost is not None:
        monkeypatch.setattr(attention, "TC5_PAIR_TILE", pair_cost)
    case.ctx.shared.clear()
    out = torch.full((case.tokens, case.heads * case.head_dim), 3.0, dtype=torch.bfloat16, device=DEV)
    cache = Case.Cache()
    cache.k, cache.v = case.kd, case.vd
    attention.paged_attention(case.qd, case.qd.stride(0), out, cache, case.group, case.ctx, case.heads, case.head_dim ** -0.5,
                              case.window, sink=sink, form=None if form is None else attention.score_form(out, **form))
    ops.tc5_check(torch.device(DEV))
    return out


@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size,window", [
    (8, 2, 128, 16, 0), (4, 4, 64, 16, 0), (6, 2, 128, 1, 130), (14, 2, 64, 128, -96), (16, 1, 64, 16, 0), (5, 1, 128, 8, 300)])
@pytest.mark.parametrize("formed", [False, True])
@pytest.mark.parametrize("sinks", [False, True])
def test_pairs_and_single_streams_agree_in_bits(monkeypatch, heads, kv_heads, head_dim, page_size, window, formed, sinks):
    """Portions around one and two streams, contexts that end around a key tile; scores plain, and capped with a bias a distance
    and gated outputs; sinks."""
    from mrun_b200.kernels import attention, lib
    per = 128 // (heads // kv_heads)
    segments = [(0, per + 1), (127, 2 * per - 1), (128, 2 * per), (255, 2 * per + 1), (900, 3 * per + 5), (129, per)]
    case = Case(segments, heads, kv_heads, head_dim, page_size, torch.bfloat16, seed=heads + head_dim, window=window)
    assert attention.prefill_uses_tcgen05(lib.attention(head_dim, head_dim, formed), heads // kv_heads, page_size)
    g = torch.Generator().manual_seed(7)
    form = sink = None
    if formed:
        form = {"soft_cap": 5.0, "bias": torch.randn(heads, 150, generator=g).to(DEV),
                "gate": torch.randn(case.tokens, heads * head_dim, generator=g).to(torch.bfloat16).to(DEV)}
    if sinks:
        sink = torch.linspace(-1.0, 3.0, heads, device=DEV)
    pairs = run(case, monkeypatch, PAIRS, form, sink)
    singles = run(case, monkeypatch, SINGLES, form, sink)
    assert torch.equal(pairs, singles)
    monkeypatch.setattr(attention, "TC5_PREFILL", False)
    older = run(case, monkeypatch, None, form, sink).double()
    assert (pairs.double() - older).abs().max() <= 2e-2 * older.abs().max()     # both round P and the result to bfloat16


def test_a_portion_has_the_same_bits_beside_others(monkeypatch):
    """The first portion and its pages come first from the seed, so they are the same in every step; the others decide which of
    its blocks are pairs."""
    from mrun_b200.kernels import attention
    alone, beside = [(3000, 700)], [(3000, 700), (9000, 900), (0, 300), (512, 1)]
    case = Case(beside, 32, 8, 128, 16, torch.bfloat16, seed=3)
    whole = run(case, monkeypatch, None)
    dealt = attention.tc5_tiles(case.ctx, 32, 16, 2, 0, 148 / 8)
    small = Case(alone, 32, 8, 128, 16, torch.bfloat16, seed=3)
    # the same keys, values and queries as in the larger step
    small.kd, small.vd, small.qd = case.kd, case.vd, case.qd[:700].contiguous()
    small.table.fill_(-1)
    pages = case.seg_pages[0]
    small.table[small.infos[0].slot, :len(pages)] = torch.tensor(pages, dtype=torch.int32, device=DEV)
    assert torch.equal(run(small, monkeypatch, None), whole[:700])
    monkeypatch.setattr(attention, "TC5_PAIR_TILE", PAIRS)
    case.ctx.shared.clear()
    assert attention.tc5_tiles(case.ctx, 32, 16, 2, 0, 148 / 8)[2] != dealt[2]  # dealt another way, and the same again
    assert torch.equal(run(case, monkeypatch, PAIRS), whole)
