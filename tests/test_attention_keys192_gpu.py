"""Keys of 192 features with values of 64 and 128 on the tcgen05 prompt kernel: every form of the call (groups, page sizes,
windows, chunks, sinks, portions beside single tokens) against plain attention in 64 bits and the mma.sync kernel."""
from __future__ import annotations

import pytest
import torch

from test_attention_gpu import DEV, Case

pytestmark = pytest.mark.gpu
SEGMENTS = [(0, 530), (700, 300), (1, 1), (250, 129), (130, 2)]


def exact(case: Case, values: torch.Tensor, scale: float, sink) -> torch.Tensor:
    from_pages = lambda pages, s: torch.stack([pages[case.seg_pages[s][p // case.page_size], :, p % case.page_size]
                                               for p in range(sum(case.segments[s]))]).to(DEV).double()
    out = torch.zeros(case.tokens, case.heads, values.shape[3], dtype=torch.float64, device=DEV)
    group = case.heads // case.kv_heads
    for s, info in enumerate(case.infos):
        k, v = from_pages(case.k, s), from_pages(values, s)
        rows = slice(info.q_start, info.q_start + info.q_len)
        q = case.qd[rows, :case.heads * 192].double().view(info.q_len, case.heads, 192)
        pos = torch.arange(info.pos_start, info.pos_start + info.q_len, device=DEV)
        keys = torch.arange(k.shape[0], device=DEV)
        first = pos * 0 if not case.window else pos - case.window + 1 if case.window > 0 else pos - pos % -case.window
        seen = (keys[None] <= pos[:, None]) & (keys[None] >= first[:, None])
        for h in range(case.heads):
            scores = (q[:, h] @ k[:, h // group].T * scale).masked_fill(~seen, float("-inf"))
            if sink is not None:
                scores = torch.cat([scores, sink[h].double().expand(info.q_len, 1)], 1)
            out[rows, h] = torch.softmax(scores, -1)[:, :k.shape[0]] @ v[:, h // group]
    return out.flatten(1)


@pytest.mark.parametrize("heads, kv_heads, page_size", [(6, 2, 16), (4, 4, 1), (16, 1, 128), (3, 1, 8), (2, 1, 256)])
@pytest.mark.parametrize("vdim", [64, 128])
@pytest.mark.parametrize("window", [0, 200, -96])
@pytest.mark.parametrize("sinks", [False, True])
def test_keys_of_192_features(heads, kv_heads, page_size, vdim, window, sinks, monkeypatch):
    from mrun_b200.kernels import attention, lib, ops
    assert attention.prefill_uses_tcgen05(lib.attention(192, vdim), heads // kv_heads, page_size)
    case = Case(SEGMENTS, heads, kv_heads, 192, page_size, torch.bfloat16, seed=heads + vdim, window=window)
    values = case.v[..., :vdim].contiguous()
    cache = Case.Cache()
    cache.k, cache.v = case.kd, values.to(DEV)
    sink = torch.linspace(-1.0, 3.0, heads, device=DEV) if sinks else None
    scale = 192 ** -0.5
    want = exact(case, values, scale, sink)

    def run():
        case.ctx.shared.clear()
        out = torch.full((case.tokens, heads * vdim), 3.0, dtype=torch.bfloat16, device=DEV)
        attention.paged_attention(case.qd, case.qd.stride(0), out, cache, case.group, case.ctx, heads, scale, window, sink=sink)
        ops.tc5_check(torch.device(DEV))
        return out.double()
    got = run()
    monkeypatch.setattr(attention, "TC5_PREFILL", False)
    older = run()
    # probabilities and outputs are rounded to bfloat16 in both kernels
    assert (got - want).abs().max() <= 2e-2 * want.abs().max()
    assert (got - want).norm() <= 1.1 * (older - want).norm()
