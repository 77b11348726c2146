"""How prompt portions are dealt to the blocks of the tcgen05 attention: the host library against the rule restated here, and
what it costs a step."""
from __future__ import annotations

import heapq
import random
import time

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


def makespan(costs, machines):
    if len(costs) <= machines:
        return max(costs, default=0.0)
    free = [0.0] * machines
    for cost in costs:
        heapq.heapreplace(free, free[0] + cost)
    return max(free)


def rule(step, tokens, longer_than, streams, window, at_once):
    """The longest blocks are pairs, of none, all, and as many as fill the device evenly what ends first."""
    def keys_of(end, count):
        low = end - count
        low = 0 if window == 0 else max(0, low - window + 1) if window > 0 else low // -window * -window
        return (end - 1) // 128 - low // 128 + 1
    wide = []
    for seg in step.segments:
        if seg.q_len > longer_than:
            for t0 in range(0, seg.q_len, streams * tokens):
                count = min(streams * tokens, seg.q_len - t0)
                wide.append((keys_of(seg.pos_start + t0 + count, count), seg.pos_start + t0 + count, seg.q_start + t0, count))
    wide.sort(key=lambda w: (-w[0], -w[1]))
    single = lambda keys: attention.TC5_SINGLE_TILE * keys + attention.TC5_BLOCK
    best, found = None, [(single(keys), first, count) for keys, _, first, count in wide]
    if streams == 2 and any(w[3] > tokens for w in wide):
        for pairs in sorted({len(wide), int(len(wide) // at_once * at_once), 0}, reverse=True):
            blocks = []
            for i, (keys, end, first, count) in enumerate(wide):
                if count <= tokens:
                    blocks.append((single(keys), first, count))
                elif i < pairs:
                    blocks.append((attention.TC5_PAIR_TILE * keys + attention.TC5_BLOCK, first, count))
                else:
                    rest = count - tokens
                    blocks.append((single(keys_of(end, rest)), first + tokens, rest))
                    blocks.append((single(keys_of(end - rest, tokens)), first, tokens))
            blocks.sort(key=lambda b: -b[0])
            ends = makespan([b[0] for b in blocks], max(1, int(at_once)))
            if best is None or ends < best:
                best, found = ends, blocks
    return [b[1] for b in found], [b[2] for b in found]


@pytest.mark.parametrize("seed", range(60))
def test_the_host_library_deals_by_the_rule(seed):
    rng = random.Random(seed)
    portions = [(rng.choice([0, rng.randint(1, 9000)]), rng.choice([1, rng.randint(1, 40), rng.randint(40, 1200)]))
                for _ in range(rng.choice([1, 2, 7, 40]))]
    arguments = (rng.choice([1, 2, 18, 32, 128]), rng.choice([0, 8, 16]), rng.choice([1, 2, 2]), rng.choice([0, 130, -256]),
                 148 / rng.choice([1, 2, 7, 8, 32, 200]))
    first, count, n = attention.tc5_tiles(Step(portions), *arguments)
    want = rule(Step(portions), *arguments)
    assert n == len(want[0])
    assert n == 0 or (first.tolist(), count.tolist()) == want


@pytest.mark.parametrize("portions", [[(0, 2048)], [(0, 300)] * 64, [(0, 65536)]])
def test_dealing_costs_a_step_no_more_than_plain_tiles(portions):
    """Tiles of one stream each in plain order are what a step was cut into before; both are made anew for every step of a service."""
    def least(go):
        best = 1.0
        for _ in range(15):
            step = Step(portions)
            start = time.perf_counter()
            go(step)
            best = min(best, time.perf_counter() - start)
        return best
    attention.tc5_tiles(Step(portions), 32, 16, 2, 0, 148 / 8)
    dealt = least(lambda step: attention.tc5_tiles(step, 32, 16, 2, 0, 148 / 8))
    assert dealt <= 1.2 * least(lambda step: attention.prefill_tiles(step, 32, longer_than=16))
