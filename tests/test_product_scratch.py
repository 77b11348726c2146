"""The memory budget counts what 32-bit products take beside their operands (host only)."""
from types import SimpleNamespace

import torch

from mrun_b200.cache import PagedKV
from mrun_b200.engine import budget
from mrun_b200.engine.budget import GIB, DeviceMemory
from mrun_b200.engine.engine import _sizing
from mrun_b200.engine.model import Model
from mrun_b200.kernels import ops


def model(dtype, k):
    m = Model.__new__(Model)
    m.spec = SimpleNamespace(hidden_size=256, vocab_size=1000, max_positions=1 << 22)
    m.runtime = SimpleNamespace(precision=SimpleNamespace(act=dtype))
    m.final_norm, m.embedding, m.head, m.embedder = None, torch.empty(8, 256, dtype=dtype), torch.empty(8, 256, dtype=dtype), None
    m.order, m.blocks = [], [SimpleNamespace(feed_forward=SimpleNamespace(w=torch.empty(512, k, dtype=dtype)))]
    m.cache_needs, m.cache_shares = (lambda: [PagedKV(8, 128)]), (lambda: [None])
    return m


def test_the_split_rows_are_part_of_the_scratch():
    memory = budget.plan(DeviceMemory(80 * GIB, 80 * GIB), 2)
    scratch = lambda m, tokens: _sizing(memory, None, 16, 4, tokens)(m)[1].scratch
    plain = lambda m, tokens: budget.scratch_estimate(256, 0, 1000, tokens, 4, 2 if m.runtime.precision.act == torch.bfloat16 else 4)
    for tokens in (1, 512, 1 << 16):
        m = model(torch.float32, 4100)
        taken = scratch(m, tokens) - plain(m, tokens)
        assert taken == min(tokens, ops.F32_TC_SCRATCH // (6 * 4104)) * 6 * 4104
        for without in (model(torch.float32, 1024), model(torch.bfloat16, 4100)):
            assert scratch(without, tokens) == plain(without, tokens)
