"""The chunked scans against the recurrence token by token in 64 bits, at the edges of chunks and runs, and against
the walk they take over from."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def context(lengths, slots):
    at = [0]
    for n in lengths:
        at.append(at[-1] + n)
    order = [(5 * i + 2) % slots for i in range(len(lengths))]
    assert len(set(order)) == len(order)
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    return SimpleNamespace(segments=[SimpleNamespace(q_len=n) for n in lengths], num_segments=len(lengths), max_q_len=max(lengths),
                           shared={}, seg_q_start=dev(at), seg_slot=dev(order))


def exact(q, k, v, g, ctx, state, beta=None):
    """q, k, g: float64 [tokens, heads, dim], v: [tokens, heads, vdim]; (outputs, states)."""
    new, out, at = state.double().clone(), torch.empty_like(v), ctx.seg_q_start.tolist()
    for s, slot in enumerate(ctx.seg_slot.tolist()):
        for t in range(at[s], at[s + 1]):
            new[slot] *= g[t][:, :, None]
            u = v[t]
            if beta is not None:
                u = beta[t][:, None] * (u - (new[slot] * k[t][:, :, None]).sum(1))
            new[slot] += k[t][:, :, None] * u[:, None, :]
            out[t] = (new[slot] * q[t][:, :, None]).sum(1)
    return out.flatten(1), new


LENGTHS = [[64], [63, 1, 65], [128], [129, 16, 17, 15], [1, 200, 33], [300]]


def check(run, want, monkeypatch, chunks_taken):
    """``run()`` -> (outputs, states) by the chunks and by the walk; both within 32-bit sums of ``want``: up to 192
    terms a sum and a decay of a few roundings a token, 2^-24 each."""
    from mrun_b200.kernels import ops
    monkeypatch.setattr(ops, "_chunks", lambda ctx, tokens, least: sum(-(-seg.q_len // ops.CHUNK) for seg in ctx.segments))
    taken = []
    for name in ("_chunked_scan", "_chunked_delta_scan"):
        monkeypatch.setattr(ops, name, lambda *a, inner=getattr(ops, name): taken.append(inner(*a)) or taken[-1])
    results = [run()]
    assert taken == [chunks_taken]
    monkeypatch.setattr(ops, "_chunks", lambda ctx, tokens, least: 0)
    results.append(run())
    for got in results:
        for x, y in zip(got, want):
            assert float((x.double() - y).abs().max() / y.abs().max()) <= 2e-5
            assert float((x.double() - y).norm() / y.norm()) <= 5e-6


@pytest.mark.parametrize("heads, dim, vdim", [(3, 128, 128), (2, 64, 64), (1, 64, 128), (2, 128, 64)])
@pytest.mark.parametrize("lengths", LENGTHS, ids=str)
@pytest.mark.parametrize("silu", [False, True])
def test_decay_scan_in_chunks(heads, dim, vdim, lengths, silu, monkeypatch):
    from mrun_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(sum(lengths) + dim)
    ctx, tokens = context(lengths, 7), sum(lengths)
    y = torch.randn(tokens, heads * (2 * dim + vdim) + 4, generator=gen, device=DEV).bfloat16()
    q, k, v = y[:, :heads * dim], y[:, heads * dim:2 * heads * dim], y[:, 2 * heads * dim:2 * heads * dim + heads * vdim]
    decay = torch.tensor([0.999, 0.05, 0.8][:heads], device=DEV)
    start = torch.randn(7, heads, dim, vdim, generator=gen, device=DEV)
    fn = torch.nn.functional.silu if silu else (lambda t: t)
    wide = [fn(t.double()).unflatten(1, (heads, -1)) for t in (q, k, v)]
    want = exact(*wide, decay.double()[None, :, None].expand(tokens, heads, dim), ctx, start)

    def run():
        state = start.clone()
        return ops.decay_scan(q, k, v, decay, state, ctx, heads, dim, vdim, silu), state
    check(run, want, monkeypatch, True)


@pytest.mark.parametrize("heads, dim, vdim", [(3, 128, 128), (2, 64, 64), (1, 64, 128), (2, 128, 64)])
@pytest.mark.parametrize("lengths", LENGTHS, ids=str)
@pytest.mark.parametrize("centre, spread", [(2.0, 1.5), (9.0, 1.0), (-300.0, 100.0), (0.0, 60.0)])
def test_gated_scan_in_chunks(heads, dim, vdim, lengths, centre, spread, monkeypatch):
    """Decays near one, decays that forget a token within a step (their products underflow), and both side by side."""
    from mrun_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(sum(lengths) + dim)
    ctx, tokens = context(lengths, 7), sum(lengths)
    y = torch.randn(tokens, heads * (2 * dim + vdim) + 4, generator=gen, device=DEV).bfloat16()
    q, k, v = y[:, :heads * dim], y[:, heads * dim:2 * heads * dim], y[:, 2 * heads * dim:2 * heads * dim + heads * vdim]
    a = torch.randn(tokens, heads * dim, generator=gen, device=DEV)
    bias = centre + spread * torch.randn(heads * dim, generator=gen, device=DEV)
    start = torch.randn(7, heads, dim, vdim, generator=gen, device=DEV)
    split = lambda t: t.double().unflatten(1, (heads, -1))
    g = torch.exp(torch.nn.functional.logsigmoid((a + bias).double()) / 8.0).unflatten(1, (heads, dim))
    want = exact(split(q) * dim ** -0.5, split(k), split(v), g, ctx, start)

    def run():
        state = start.clone()
        return ops.gated_scan(q, k, v, a, bias, 8.0, state, ctx, heads, dim, vdim), state
    check(run, want, monkeypatch, True)


@pytest.mark.parametrize("heads, kv_heads, dim, vdim", [(3, 3, 128, 128), (4, 2, 64, 64), (2, 1, 64, 128), (2, 2, 128, 64)])
@pytest.mark.parametrize("lengths", LENGTHS, ids=str)
@pytest.mark.parametrize("centre, spread, alike", [(-3.0, 2.0, 0.0), (-9.0, 1.0, 0.0), (-9.0, 1.0, 1.0), (0.0, 40.0, 0.5)])
def test_delta_scan_in_chunks(heads, kv_heads, dim, vdim, lengths, centre, spread, alike, monkeypatch):
    """Keys apart and (``alike``) nearly the same key again and again, which couples a chunk's writes the most."""
    from mrun_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(sum(lengths) + dim)
    ctx, tokens = context(lengths, 7), sum(lengths)
    y = torch.randn(tokens, 2 * kv_heads * dim + heads * vdim + 4, generator=gen, device=DEV)
    y[:, kv_heads * dim:2 * kv_heads * dim] += 4 * alike * torch.randn(kv_heads * dim, generator=gen, device=DEV)
    y = y.bfloat16()
    q, k = y[:, :kv_heads * dim], y[:, kv_heads * dim:2 * kv_heads * dim]
    v = y[:, 2 * kv_heads * dim:2 * kv_heads * dim + heads * vdim]
    a = torch.randn(tokens, heads * dim, generator=gen, device=DEV)
    b = torch.randn(tokens, heads + 3, generator=gen, device=DEV).bfloat16()[:, :heads]
    a_log = torch.rand(heads, generator=gen, device=DEV) * 3 - 3
    dt_bias = centre + spread * torch.randn(heads * dim, generator=gen, device=DEV)
    start = torch.randn(7, heads, dim, vdim, generator=gen, device=DEV)
    unit = lambda t: (lambda x: x / torch.sqrt((x ** 2).sum(-1, keepdim=True) + 1e-6))(t.double().unflatten(1, (kv_heads, dim)))
    both = lambda t: t.repeat_interleave(heads // kv_heads, dim=1)
    g = torch.exp(-torch.exp(a_log.double())[None, :, None] * torch.nn.functional.softplus((a + dt_bias).double()).unflatten(1, (heads, dim)))
    want = exact(both(unit(q)) * dim ** -0.5, both(unit(k)), v.double().unflatten(1, (heads, vdim)), g, ctx, start,
                 torch.sigmoid(b.double()))

    def run():
        state = start.clone()
        return ops.delta_scan(q, k, v, a, b, a_log, dt_bias, state, ctx, heads, kv_heads, dim, vdim), state
    check(run, want, monkeypatch, True)


@pytest.mark.parametrize("dim, vdim", [(128, 128), (64, 64)])
@pytest.mark.parametrize("kind", ["decay", "gated", "delta"])
def test_earlier_tokens_do_not_meet_later_values_that_are_no_numbers(kind, dim, vdim, monkeypatch):
    """A key or a value that is infinite or no number spoils its own token and later ones of its request, as in the walk; the
    tokens before it keep their bits."""
    from mrun_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(dim)
    heads, ctx, tokens = 2, context([150, 70], 7), 220
    y = torch.randn(tokens, heads * (2 * dim + vdim), generator=gen, device=DEV).bfloat16()
    a, bias = torch.randn(tokens, heads * dim, generator=gen, device=DEV), torch.full((heads * dim,), 2.0, device=DEV)
    b = torch.randn(tokens, heads, generator=gen, device=DEV).bfloat16()
    rate = torch.full((heads,), -2.0, device=DEV)
    monkeypatch.setattr(ops, "_chunks", lambda ctx, tokens, least: sum(-(-seg.q_len // ops.CHUNK) for seg in ctx.segments))

    def run(y):
        q, k, v = y[:, :heads * dim], y[:, heads * dim:2 * heads * dim], y[:, 2 * heads * dim:]
        state = torch.ones(7, heads, dim, vdim, device=DEV)
        if kind == "decay":
            return ops.decay_scan(q, k, v, torch.full((heads,), 0.9, device=DEV), state, ctx, heads, dim, vdim, True)
        if kind == "gated":
            return ops.gated_scan(q, k, v, a, bias, 8.0, state, ctx, heads, dim, vdim)
        return ops.delta_scan(q, k, v, a, b, rate, bias, state, ctx, heads, heads, dim, vdim)
    want = run(y)
    assert torch.isfinite(want).all()
    keys, values = slice(heads * dim, 2 * heads * dim), slice(2 * heads * dim, None)
    for at in (0, 1, 37, 63, 64, 79, 149):         # the chunk's and the runs' edges, both halves of a chunk
        for what in (float("inf"), float("nan")):
            for spoilt in (keys, values):
                rows = y.clone()
                rows[at, spoilt] = what
                got = run(rows)
                assert torch.equal(got[:at], want[:at]) and torch.equal(got[150:], want[150:]), (at, what, spoilt)
                assert not torch.isfinite(got[at]).any()


def test_which_steps_are_scanned_in_chunks():
    """Long segments, and short ones beside them as long as they pad little; never a captured step."""
    from mrun_b200.kernels import ops

    def chunks(lengths):
        return ops._chunks(SimpleNamespace(segments=[SimpleNamespace(q_len=n) for n in lengths], shared={}, num_segments=len(lengths),
                                           max_q_len=max(lengths)), sum(lengths), ops.CHUNK_MIN_TOKENS)
    assert chunks([ops.CHUNK_MIN_TOKENS - 1]) == 0
    assert chunks([ops.CHUNK_MIN_TOKENS]) == -(-ops.CHUNK_MIN_TOKENS // ops.CHUNK)
    assert chunks([640, 640, 1, 1]) == 22
    assert chunks([256] + [1] * 20) == 0
    assert ops._chunks(SimpleNamespace(segments=[], shared={}, num_segments=4, max_q_len=500), 4, 1) == 0


def test_rows_without_a_chunked_form_are_walked(monkeypatch):
    """32-bit rows, other sizes and rows off their 8 bytes go to the walk as before."""
    from mrun_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(1)
    ctx = context([150], 7)
    for dtype, dim, off in ((torch.float32, 64, 0), (torch.bfloat16, 48, 0), (torch.bfloat16, 64, 1)):
        y = torch.randn(150, 3 * dim + 4, generator=gen, device=DEV).to(dtype)
        q, k, v = (y[:, off + i * dim:off + (i + 1) * dim] for i in range(3))
        decay, start = torch.tensor([0.9], device=DEV), torch.zeros(7, 1, dim, dim, device=DEV)
        want = exact(*(t.double()[:, None] for t in (q, k, v)), torch.full((150, 1, dim), 0.9, device=DEV).double(), ctx, start)

        def run():
            state = start.clone()
            return ops.decay_scan(q, k, v, decay, state, ctx, 1, dim, dim, False), state
        with monkeypatch.context() as m:
            check(run, want, m, False)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("groups, n", [(3, 8), (5, 64), (2, 72), (7, 128), (3, 136), (2, 256), (5, 264), (2, 1016), (1, 1024), (2, 8192), (1, 8200)])
@pytest.mark.parametrize("shared", [False, True])
def test_gated_norm_in_pieces(dtype, groups, n, shared):
    """Group sizes on both sides of every number of threads, weights a group or a row long, strided gates and outputs."""
    from mrun_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(n)
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    for tokens in (1, 13):
        o, gate, weight = rand(tokens, groups * n), rand(tokens, groups * n + 8).to(dtype)[:, 8:], rand(n if shared else groups * n)
        out = torch.full((tokens, groups * n + 16), 7.0, dtype=dtype, device=DEV)
        ops.gated_norm(o, weight, gate, 1e-5, groups, dtype, gate_function="silu", out=out[:, :groups * n], scale=0.5)
        x = o.double().view(tokens, groups, n)
        want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * weight.double().view(1, -1, n)
        want = 0.5 * want.flatten(1) * torch.nn.functional.silu(gate.double())
        # a few roundings of 2^-24 behind a sum of n squares; bfloat16 rounds the result to 8 bits
        assert ((out[:, :groups * n].double() - want).abs() <= (2e-6 if dtype == torch.float32 else 2.0 ** -8) * want.abs() + 1e-6).all()
        assert (out[:, groups * n:] == 7.0).all()


@pytest.mark.parametrize("kind", ["decay", "gated", "delta"])
@pytest.mark.parametrize("dim, vdim", [(128, 128), (64, 128), (128, 64), (64, 64)])
def test_a_mixer_holds_no_more_than_it_declares(kind, dim, vdim):
    """Beside its inputs and outputs, over a step whose segments pad the chunks nearly as much as a chunked step may."""
    from mrun_b200.config import spec as specs
    from mrun_b200.engine import StepEntry
    from mrun_b200.engine.batch import HostStaging, build_context
    from mrun_b200.cache import CacheManager
    from mrun_b200.kernels import ops
    from mrun_b200.parts import MIXERS, Precision, Runtime
    hidden, heads, lengths = 256, 16, [641] * 3 + [1] * 4
    spec = {"decay": lambda: specs.DecayAttentionSpec(hidden=hidden, heads=heads, dim=dim, vdim=vdim, eps=1e-5, decay=(0.9,) * heads),
            "gated": lambda: specs.GatedLinearAttentionSpec(hidden=hidden, heads=heads, dim=dim, vdim=vdim, tau=8.0, rank=16, eps=1e-5),
            "delta": lambda: specs.ChannelDeltaSpec(hidden=hidden, heads=heads, kv_heads=heads, dim=dim, vdim=vdim, conv=4, decay_rank=16,
                                                    gate_rank=16, eps=1e-5)}[kind]()
    rt = Runtime(torch.device(DEV), Precision.of("bfloat16"), 16)
    gen = torch.Generator().manual_seed(1)
    weights = {t.name[2:]: 0.1 * torch.randn(t.shape, generator=gen) for t in MIXERS.tensor_specs(spec, "m")}
    part = MIXERS.build(spec, weights, rt)
    manager = CacheManager([part.cache_need()], [None], 16, 200, len(lengths), device=torch.device(DEV), dtype=torch.bfloat16)
    requests = [manager.admit(i) for i in range(len(lengths))]
    manager.plan_append(list(zip(requests, lengths)))
    ctx = build_context([StepEntry(r, [0] * n) for r, n in zip(requests, lengths)], manager, HostStaging(torch.device(DEV)))
    tokens = sum(lengths)
    assert ops._chunks(ctx, tokens, ops._chunk_least(ctx, tokens, kind == "delta", heads, dim, vdim))
    x = torch.randn(tokens, hidden, device=DEV).bfloat16()
    part.forward(x, ctx, manager.entries[0])                     # the vendor library's workspace
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    part.forward(x, ctx, manager.entries[0])
    held = torch.cuda.max_memory_allocated() - before
    chunk = heads * ops.chunk_scratch_elements(dim, vdim, kind == "delta") * ops.CHUNK * 2         # the one chunk beside the quarter
    assert held <= 2 * tokens * (part.activation_elements() + hidden) + chunk


def test_declared_scratch_is_the_kernels():
    """The estimate's floats of a chunk are those that the kernels ask for."""
    from mrun_b200.kernels import ops
    like = torch.empty(64, 128, device=DEV)
    q = torch.empty(64, 128, device=DEV, dtype=torch.bfloat16)
    for delta in (False, True):
        for dim in (64, 128):
            for vdim in (64, 128):
                size = ops._lib.core().function("mrun_chunked_scan_floats")
                size.restype = ops._c_long
                floats = size(ops._c_int(delta), ops._ptr(q), ops._ptr(q), ops._ptr(q), ops._c_long(128), ops._c_int(ops.dtype_code(q.dtype)),
                              ops._ptr(like), ops._ptr(like), ops._ptr(like), ops._ptr(like), ops._c_int(1), ops._c_int(1), ops._c_int(dim),
                              ops._c_int(vdim))
                assert ops.chunk_scratch_elements(dim, vdim, delta) == -(-5 * 2 * floats // (4 * ops.CHUNK))


@pytest.mark.parametrize("kind", ["decay", "gated", "delta"])
def test_a_short_segment_beside_a_long_one(kind, record_property):
    """A step is walked or goes in chunks as a whole, so a short segment's outputs and its state move beside a long one: in
    the rounding of 32-bit sums only."""
    from mrun_b200.kernels import ops
    heads, dim, vdim, short = 16, 128, 128, 16
    gen = torch.Generator(device=DEV).manual_seed(2)
    y = torch.randn(short + 512, heads * (2 * dim + vdim), generator=gen, device=DEV).bfloat16()
    a, bias = torch.randn(short + 512, heads * dim, generator=gen, device=DEV), torch.full((heads * dim,), 1.0, device=DEV)
    b = torch.randn(short + 512, heads, generator=gen, device=DEV).bfloat16()
    rate, decay = torch.full((heads,), -2.0, device=DEV), torch.full((heads,), 0.95, device=DEV)
    start = torch.randn(7, heads, dim, vdim, generator=gen, device=DEV)
    results = []
    for lengths in ([short], [short, 512]):
        ctx, n = context(lengths, 7), sum(lengths)
        least = ops._chunk_least(ctx, n, kind == "delta", heads, dim, vdim)
        assert bool(ops._chunks(ctx, n, least)) == (len(lengths) == 2)
        q, k, v = y[:n, :heads * dim], y[:n, heads * dim:2 * heads * dim], y[:n, 2 * heads * dim:]
        state = start.clone()
        if kind == "decay":
            out = ops.decay_scan(q, k, v, decay, state, ctx, heads, dim, vdim, True)
        elif kind == "gated":
            out = ops.gated_scan(q, k, v, a[:n], bias, 8.0, state, ctx, heads, dim, vdim)
        else:
            out = ops.delta_scan(q, k, v, a[:n], b[:n], rate, bias, state, ctx, heads, heads, dim, vdim)
        results.append((out[:short], state[ctx.seg_slot[0]]))
    for name, alone, beside in zip(("outputs", "state"), *results):
        moved = float((beside - alone).norm() / alone.norm())
        record_property(f"{kind} {name}", moved)
        print(f"{kind}: a short segment's {name} move by {moved:.2e} beside a long one")
        assert moved <= 5e-6
