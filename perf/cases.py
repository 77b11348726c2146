"""What the engine's speed is measured on: decode steps through the executor, and the layers that its
decoders are made of, each through the entry point that a program calls (``Executor.decode_step``, a part
built from its spec and run with ``forward``).

A case names a kind of work and its sizes; ``listed()`` holds the cases by name, ``draw()`` gives others of
the same ranges.  Sizes are those of the repository's own configurations: the Qwen3-8B and 4B layer
shapes and the sizes that ``bench.py`` measures the other decoders at.  Weights and inputs are random, made
on the device from the seed.

Kinds
-----
step        a captured decode step of a Qwen3 model of two layers and its whole output head: one token for
            each of ``requests`` requests, whose contexts reach up to ``depth`` tokens
block       a pre-norm Qwen3 block (norm, attention, norm, gated feed-forward, the next block's norm) in
            ``dtype`` over prompt portions or decoding requests
attention   the Qwen3 attention layer alone: prompt portions behind contexts of up to ``depth`` tokens, with
            ``beside`` decoding requests in the same step
decay, delta, gated
            the recurrent mixers: one decay a head, the gated delta rule, a decay a key channel
latent      attention over one cached latent row a token (rows of 576 features)
"""
from __future__ import annotations

import math

import torch

from mrun_b200.cache import CacheManager
from mrun_b200.config import qwen3
from mrun_b200.config import spec as specs
from mrun_b200.engine import StepEntry
from mrun_b200.engine.batch import HostStaging, build_context
from mrun_b200.engine.loading import executor_from_config
from mrun_b200.kernels import ops
from mrun_b200.parts import ARRANGEMENTS, MIXERS, NORMS, Precision, Runtime
from mrun_b200.weights import random_tensors
from mrun_b200.weights.random_init import random_tensor

DEV = "cuda:0"
PAGE = 16
EPS = 1e-6
THETA = 1e6
VOCAB = 151936
# hidden, heads, kv heads, head size, intermediate: the Qwen3 layer shapes of the repository's benchmark
SHAPES = {"8b": (4096, 32, 8, 128, 12288), "4b": (2560, 32, 8, 128, 9728)}
BF16_OUT = {"rel": 0.016, "max": 0.16}       # a layer in bfloat16 is about 0.004 off 64 bits
F32_OUT = {"rel": 1e-5, "max": 1e-4}         # a block in 32-bit is about 2.5e-6 off 64 bits


def listed():
    return [
        # one user's chat: the smallest decode step, where latency counts
        {"name": "decode_one", "kind": "step", "dtype": "bfloat16", "shape": "8b", "requests": 1, "depth": 1023},
        # a busy server: 64 requests with contexts of up to 1,100 tokens decode side by side
        {"name": "decode_many", "kind": "step", "dtype": "bfloat16", "shape": "8b", "requests": 64, "depth": 1100},
        # the 32-bit mode (parity runs, replays): a few requests decode
        {"name": "f32_decode", "kind": "block", "dtype": "float32", "shape": "8b", "requests": 4, "tokens": 4, "depth": 300},
        # the 32-bit mode: two ragged prompts
        {"name": "f32_prompt", "kind": "block", "dtype": "float32", "shape": "8b", "requests": 2, "tokens": 517, "depth": 0},
        # three prompts of one step through a whole block
        {"name": "block_prompt", "kind": "block", "dtype": "bfloat16", "shape": "8b", "requests": 3, "tokens": 1337, "depth": 0},
        # the headline prompt
        {"name": "attention_prompt", "kind": "attention", "dtype": "bfloat16", "shape": "8b", "requests": 1, "tokens": 2048,
         "depth": 0, "beside": 0},
        # a served step: a portion of a long prompt beside the decoding of others
        {"name": "attention_served", "kind": "attention", "dtype": "bfloat16", "shape": "4b", "requests": 1, "tokens": 1531,
         "depth": 9000, "beside": 11},
        # prompts through the recurrent mixers of the Balivik and Fikudra decoders
        {"name": "decay_prompt", "kind": "decay", "dtype": "bfloat16", "width": 2048, "heads": 16, "requests": 1, "tokens": 2048},
        {"name": "delta_prompt", "kind": "delta", "dtype": "bfloat16", "width": 2048, "heads": 16, "requests": 3, "tokens": 1777},
        {"name": "gated_prompt", "kind": "gated", "dtype": "bfloat16", "width": 4096, "heads": 32, "requests": 1, "tokens": 2048},
        # two prompts, one of them in its second portion, through the Zasesun decoder's attention
        {"name": "latent_prompt", "kind": "latent", "dtype": "bfloat16", "width": 2048, "heads": 16, "requests": 2, "tokens": 1900,
         "depth": 700},
        # eight requests decode through a recurrent mixer: the smallest call, launches and latency
        {"name": "gated_decode", "kind": "gated", "dtype": "bfloat16", "width": 2048, "heads": 16, "requests": 8, "tokens": 8},
    ]


def _between(rng, low, high):
    """Spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["step", "step", "block32", "block32", "block", "attention", "attention", "decay", "delta", "gated",
                       "latent"])
    if kind == "step":
        return {"kind": "step", "dtype": "bfloat16", "shape": rng.choice(["8b", "4b"]), "requests": _between(rng, 1, 64),
                "depth": _between(rng, 40, 1900)}
    if kind == "block32":
        if rng.random() < 0.5:
            n = _between(rng, 1, 24)
            return {"kind": "block", "dtype": "float32", "shape": rng.choice(["8b", "4b"]), "requests": n, "tokens": n,
                    "depth": _between(rng, 20, 900)}
        n = _between(rng, 20, 500)
        return {"kind": "block", "dtype": "float32", "shape": rng.choice(["8b", "4b"]), "requests": rng.randint(1, 3), "tokens": n,
                "depth": rng.choice([0, _between(rng, 20, 400)])}
    if kind == "block":
        n = _between(rng, 6, 1300)
        return {"kind": "block", "dtype": "bfloat16", "shape": rng.choice(["8b", "4b"]), "requests": rng.randint(1, min(n, 6)),
                "tokens": n, "depth": rng.choice([0, _between(rng, 20, 2000)])}
    if kind == "attention":
        n = _between(rng, 40, 2048)
        return {"kind": "attention", "dtype": "bfloat16", "shape": rng.choice(["8b", "4b"]), "requests": rng.randint(1, 4),
                "tokens": n, "depth": rng.choice([0, _between(rng, 100, 8000)]), "beside": rng.choice([0, rng.randint(1, 15)])}
    if kind in ("decay", "delta", "gated"):
        width, heads = rng.choice([(2048, 16), (4096, 32)])
        if rng.random() < 0.2:
            n = _between(rng, 1, 64)
            return {"kind": kind, "dtype": "bfloat16", "width": width, "heads": heads, "requests": n, "tokens": n}
        n = _between(rng, 3, 2048)
        return {"kind": kind, "dtype": "bfloat16", "width": width, "heads": heads, "requests": rng.randint(1, min(n, 5)), "tokens": n}
    n = _between(rng, 4, 1900)
    return {"kind": "latent", "dtype": "bfloat16", "width": 2048, "heads": 16, "requests": rng.randint(1, min(n, 4)),
            "tokens": n, "depth": rng.choice([0, _between(rng, 100, 2000)])}


# ------------------------------------------------------------------ sizes of a case

def _portions(case):
    """(context before, new tokens) of every request of the step: uneven portions, uneven contexts."""
    n, total, depth = case.get("requests", 1), case["tokens"], case.get("depth", 0)
    shares = [1.0 + (7 * i % 5) / 4 for i in range(n)]
    counts = [max(1, int(total * s / sum(shares))) for s in shares]
    while sum(counts) > total:
        counts[counts.index(max(counts))] -= 1
    counts[0] += total - sum(counts)
    before = [depth - i * depth // n if depth else 0 for i in range(n)]
    beside = case.get("beside", 0)
    return list(zip(before, counts)) + [(max(1, depth - (3 * i + 1) * depth // (3 * beside + 1)) if depth else 5 + 9 * i, 1)
                                        for i in range(beside)]


def _contexts(case):
    """Tokens each request of a decode step holds before it."""
    n, depth = case["requests"], case["depth"]
    return [max(2, depth - i * depth // (2 * n)) for i in range(n)]


def _spec(case):
    kind = case["kind"]
    if kind in ("step", "block", "attention"):
        hidden, heads, kv, dim, ff = SHAPES[case["shape"]]
        attention = specs.AttentionSpec(hidden=hidden, heads=heads, kv_heads=kv, head_dim=dim, softmax_scale=dim ** -0.5,
                                        qk_norm=specs.RMSNormSpec(dim, EPS), position=specs.RotarySpec(dim, dim, THETA))
        if kind == "attention":
            return attention
        norm = specs.RMSNormSpec(hidden, EPS)
        return specs.LayerSpec(prefix="p", mixer=attention, feed_forward=specs.GatedMLPSpec(hidden, ff, "silu"), mixer_norm=norm,
                               feed_forward_norm=norm)
    width, heads = case["width"], case.get("heads", 0)
    if kind == "decay":
        return specs.DecayAttentionSpec(hidden=width, heads=heads, dim=128, vdim=128, eps=EPS,
                                        decay=tuple(1.0 - 2.0 ** -(2 + 6 * i / max(1, heads - 1)) for i in range(heads)))
    if kind == "delta":
        return specs.ChannelDeltaSpec(hidden=width, heads=heads, kv_heads=heads, dim=128, vdim=128, conv=4, decay_rank=width // 16,
                                      gate_rank=width // 16, eps=EPS)
    if kind == "gated":
        return specs.GatedLinearAttentionSpec(hidden=width, heads=heads, dim=128, vdim=128, tau=8.0, rank=width // 16, eps=EPS)
    return specs.LatentAttentionSpec(hidden=width, heads=heads, dim=128, rot_dim=64, vdim=128, q_rank=1536, kv_rank=512,
                                     softmax_scale=192 ** -0.5, eps=EPS,
                                     position=specs.ScaledRotarySpec(64, 10000.0, scaling=(4.0, 4096, 32.0, 1.0)))


# values that a trained layer has and N(0, 0.02) would not give: decays from quick to almost none
_CENTRES = {"delta": {"p.dt_bias": (-3.0, 2.0)}, "gated": {"p.a2.b": (2.0, 1.5)}}


def _weights(case, seed, tensor_specs):
    store = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    centres = _CENTRES.get(case["kind"], {})
    out = {}
    for t in tensor_specs:
        if t.optional:
            continue
        if t.name in centres:
            mean, std = centres[t.name]
            out[t.name] = (mean + std * torch.randn(t.shape, generator=_generator(seed, 5), device=DEV)).to(store)
        elif t.name.endswith(".conv"):
            out[t.name] = (0.25 + 0.25 * torch.randn(t.shape, generator=_generator(seed, 6), device=DEV)).to(store)
        else:
            out[t.name] = random_tensor(t, seed, 0.02, 0.1, store, device=DEV)
    return out


def _tensor_specs(case, spec):
    if case["kind"] == "block":
        return ARRANGEMENTS.get("pre_norm").tensor_specs(spec)
    return MIXERS.tensor_specs(spec, "p")


def _generator(seed, salt):
    return torch.Generator(device=DEV).manual_seed((seed + 1) * 1000003 + salt)


def _local(tensors, prefix="p."):
    return {name[len(prefix):]: t for name, t in tensors.items() if name.startswith(prefix)}


def _input(case, seed, rows, width):
    """Rows as a norm leaves them (a block's: the 32-bit stream in front of its norm)."""
    x = torch.randn((rows, width), generator=_generator(seed, 1), device=DEV)
    return x if case["kind"] == "block" else x.to(Precision.of(case["dtype"]).act)


# ------------------------------------------------------------------ prepare and run

def _cache(case, seed, need, precision):
    """A cache manager that holds the step's requests with random contexts, the step planned, and its context."""
    portions = _portions(case)
    pages = sum(-(-(before + n) // PAGE) for before, n in portions) + 8
    manager = CacheManager([need], [None], PAGE, pages, len(portions), device=torch.device(DEV), dtype=precision.act)
    requests = [manager.admit(i) for i in range(len(portions))]
    held = [(r, before) for r, (before, _) in zip(requests, portions) if before]
    if held:
        manager.commit(manager.plan_append(held))
    plan = manager.plan_append([(r, n) for r, (_, n) in zip(requests, portions)])
    staging = HostStaging(torch.device(DEV))
    ctx = build_context([StepEntry(r, [0] * n) for r, (_, n) in zip(requests, portions)], manager, staging)
    entry = manager.entries[0]
    generator = _generator(seed, 2)
    for pool in ([] if entry.k is None else [entry.k] if entry.v is entry.k else [entry.k, entry.v]):
        pool.copy_(torch.randn(pool.shape, generator=generator, device=DEV))
    if entry.k is not None and entry.v is entry.k and entry.need.width > 576:
        entry.k[..., 576:].zero_()
    states = {}
    for name, state in entry.states.items():
        state.copy_(torch.randn(state.shape, generator=generator, device=DEV))
        states[name] = state.clone()
    return {"manager": manager, "requests": requests, "plan": plan, "ctx": ctx, "entry": entry, "states": states}


def prepare(case, seed):
    torch.cuda.set_device(0)
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    spec = _spec(case)
    precision = Precision.of(case["dtype"])
    rt = Runtime(torch.device(DEV), precision, PAGE)
    tensors = _weights(case, seed, _tensor_specs(case, spec))
    state = {"kind": case["kind"]}
    if case["kind"] == "block":
        part = ARRANGEMENTS.get("pre_norm")(spec, tensors, rt)
        hidden, mixer = spec.mixer.hidden, part.mixer
        state["next_norm"] = NORMS.build(specs.RMSNormSpec(hidden, EPS), {"weight": torch.ones(hidden, device=DEV)}, rt)
        state["stream"] = torch.empty((sum(n for _, n in _portions(case)), hidden), device=DEV)
    else:
        part = mixer = MIXERS.build(spec, _local(tensors), rt)
        hidden = spec.hidden
    state.update(part=part, **_cache(case, seed, mixer.cache_need(), precision))
    state["x"] = _input(case, seed, state["ctx"].num_tokens, hidden)
    return state


def _model(case):
    hidden, heads, kv, dim, ff = SHAPES[case["shape"]]
    return qwen3.Qwen3Config.from_dict(dict(
        architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=2, hidden_size=hidden, num_attention_heads=heads,
        num_key_value_heads=kv, head_dim=dim, intermediate_size=ff, vocab_size=VOCAB, max_position_embeddings=8192, rms_norm_eps=EPS,
        rope_theta=THETA, tie_word_embeddings=case["shape"] == "4b"))


def _step_tokens(case, seed):
    contexts = _contexts(case)
    flat = torch.randint(0, VOCAB, (sum(contexts) + len(contexts),), generator=torch.Generator().manual_seed(seed + 11)).tolist()
    out, at = [], 0
    for n in contexts:
        out.append(flat[at:at + n + 1])
        at += n + 1
    return out


def _prepare_step(case, seed):
    contexts = _contexts(case)
    pages = sum(n // PAGE + 1 for n in contexts) + 8
    executor = executor_from_config(_model(case), seed, dtype=case["dtype"], page_size=PAGE, num_pages=pages,
                                    max_requests=len(contexts))
    requests = [executor.admit(i) for i in range(len(contexts))]
    tokens = _step_tokens(case, seed)
    group, held = [], 0
    for i, (r, t) in enumerate(zip(requests, tokens)):       # the prompts, in steps of about 2,048 tokens
        group.append(StepEntry(r, t[:-1], []))
        held += len(t) - 1
        if held >= 2048 or i == len(requests) - 1:
            executor.step(group)
            group, held = [], 0
    state = {"kind": "step", "executor": executor, "requests": requests, "contexts": contexts,
             "entries": [StepEntry(r, t[-1:], [0]) for r, t in zip(requests, tokens)]}
    run(state)                                               # a program that serves has its captured step
    return state


def run(state):
    kind = state["kind"]
    if kind == "step":
        executor = state["executor"]
        tokens = executor.decode_step(state["entries"])
        logits = executor.decode_logits(state["entries"])
        for r, n in zip(state["requests"], state["contexts"]):       # so that the same step can come again
            executor.trim(r, n)
        return {"logits": logits, "tokens": tokens}
    entry = state["entry"]
    for name, start in state["states"].items():                      # the requests' states as the steps before left them
        entry.states[name].copy_(start)
    if kind == "block":
        stream = state["stream"]
        stream.copy_(state["x"])
        delta = state["part"].forward(stream, None, state["ctx"], entry)
        rows = state["next_norm"].add_forward(stream, delta)
        out = {"stream": stream, "rows": rows.finish() if isinstance(rows, ops.NormedRows) else rows}
    else:
        out = {"y": state["part"].forward(state["x"], state["ctx"], entry)}
    if entry.k is not None:
        out["k"] = entry.k
        if entry.v is not entry.k:
            out["v"] = entry.v
    for name in entry.states:
        out[name] = entry.states[name]
    return out


# ------------------------------------------------------------------ what a pass cannot do without

def _count(t):
    n = 1
    for extent in t.shape:
        n *= extent
    return n


def work(case):
    kind, unit = case["kind"], 4 if case["dtype"] == "float32" else 2
    spec = _spec(case)
    if kind == "step":
        hidden, heads, kv, dim, ff = SHAPES[case["shape"]]
        contexts = _contexts(case)
        layer = 2 * hidden * (heads + kv) * dim + 3 * hidden * ff
        keys = sum(n + 1 for n in contexts)
        return {"bytes": unit * (2 * layer + VOCAB * hidden + 2 * keys * 2 * kv * dim + len(contexts) * hidden) + 4 * len(contexts) * VOCAB,
                "flops": 2.0 * len(contexts) * (2 * layer + VOCAB * hidden) + 2 * 4.0 * keys * heads * dim}
    weights = sum(_count(t) for t in _tensor_specs(case, spec) if not t.optional)
    portions = _portions(case)
    rows = sum(n for _, n in portions)
    keys = sum(before + n for before, n in portions)
    pairs = sum(n * before + n * (n + 1) // 2 for before, n in portions)      # (token, visible key)
    if kind in ("block", "attention"):
        att = spec.mixer if kind == "block" else spec
        cache = unit * 2 * (keys + rows) * att.kv_heads * att.head_dim
        ends = (4 + 4 + unit) * rows * att.hidden if kind == "block" else 2 * unit * rows * att.hidden
        return {"bytes": unit * weights + cache + ends, "flops": 2.0 * rows * weights + 4.0 * pairs * att.heads * att.head_dim}
    ends = 2 * unit * rows * spec.hidden
    if kind == "latent":
        row = spec.kv_rank + spec.rot_dim
        return {"bytes": unit * (weights + (keys + rows) * row) + ends,
                "flops": 2.0 * rows * weights + 2.0 * pairs * spec.heads * (spec.dim + spec.rot_dim + spec.vdim)}
    state = len(portions) * spec.heads * spec.dim * spec.vdim
    per_token = 2.0 * (4 if kind == "delta" else 2) * spec.heads * spec.dim * spec.vdim
    return {"bytes": unit * weights + 8 * state + ends, "flops": rows * (2.0 * weights + per_token)}


def tolerance(case):
    if case["dtype"] == "float32":
        return dict(F32_OUT)
    if case["kind"] == "step":
        return {"rel": 0.03, "max": 0.3, "differ": 0.01}       # two layers and the head: logits about 0.01 off 64 bits
    return dict(BF16_OUT)


# ------------------------------------------------------------------ the same in 64 bits

def _norm64(x, weight):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * weight.double()


def _rotate64(x, positions, theta=THETA):
    """x: [tokens, heads, dim], half-split pairs."""
    half = x.shape[-1] // 2
    angle = positions.double()[:, None] * (theta ** (-torch.arange(half, dtype=torch.float64, device=DEV) / half))[None, :]
    cos, sin = angle.cos()[:, None, :], angle.sin()[:, None, :]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _attend64(q, k, v, scale, start):
    """q: [n, heads, d] at positions start.., k: [keys, kv, d], v: [keys, kv, dv]."""
    n, heads, _ = q.shape
    ratio = heads // k.shape[1]
    ahead = torch.arange(k.shape[0], device=DEV)[None, :] > start + torch.arange(n, device=DEV)[:, None]
    out = torch.empty((n, heads, v.shape[2]), dtype=torch.float64, device=DEV)
    for h in range(heads):
        s = (q[:, h] @ k[:, h // ratio].T * scale).masked_fill_(ahead, -math.inf)
        out[:, h] = torch.softmax(s, dim=-1) @ v[:, h // ratio]
    return out


def _attention64(x, w, att, segments, kept):
    """x: float64 [rows, hidden]; segments: (first row, context, tokens); kept(i): keys and values before segment i."""
    q = _norm64((x @ w["q_proj.weight"].double().T).unflatten(1, (att.heads, -1)), w["q_norm.weight"])
    k = _norm64((x @ w["k_proj.weight"].double().T).unflatten(1, (att.kv_heads, -1)), w["k_norm.weight"])
    v = (x @ w["v_proj.weight"].double().T).unflatten(1, (att.kv_heads, -1))
    out = torch.empty((x.shape[0], att.heads, att.head_dim), dtype=torch.float64, device=DEV)
    for i, (row, before, n) in enumerate(segments):
        at = torch.arange(before, before + n, device=DEV)
        ks, vs = _rotate64(k[row:row + n], at), v[row:row + n]
        if before:
            k0, v0 = kept(i)
            ks, vs = torch.cat([k0, ks]), torch.cat([v0, vs])
        out[row:row + n] = _attend64(_rotate64(q[row:row + n], at), ks, vs, att.softmax_scale, before)
    return out.flatten(1) @ w["o_proj.weight"].double().T


def _block64(x, w, spec, segments, kept):
    x = x + _attention64(_norm64(x, w["input_layernorm.weight"]), _local(w, "self_attn."), spec.mixer, segments, kept)
    h = _norm64(x, w["post_attention_layernorm.weight"])
    g = torch.nn.functional.silu(h @ w["mlp.gate_proj.weight"].double().T)
    return x + (g * (h @ w["mlp.up_proj.weight"].double().T)) @ w["mlp.down_proj.weight"].double().T


def _step64(case, seed):
    model = _model(case)
    spec = model.to_spec()
    w = {}
    for name, t in random_tensors(spec, seed, 0.02, 0.0, torch.bfloat16, device=DEV):
        w[name] = t
    head = w["lm_head.weight"] if "lm_head.weight" in w else w["model.embed_tokens.weight"]
    rows = []
    for tokens in _step_tokens(case, seed):
        x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=DEV)].double()
        for i in range(2):
            x = _block64(x, _local(w, f"model.layers.{i}."), spec.layers[i], [(0, 0, len(tokens))], None)
        rows.append(_norm64(x[-1:], w["model.norm.weight"]))
    h = torch.cat(rows)
    logits = torch.cat([h @ part.double().T for part in head.split(16384)], dim=1)
    return {"logits": logits, "tokens": None}


def _segments(case):
    out, row = [], 0
    for before, n in _portions(case):
        out.append((row, before, n))
        row += n
    return out


def _short_conv64(x, weight, before):
    """SiLU of a causal convolution per channel; ``before``: the inputs in front of the rows."""
    taps = weight.shape[1]
    padded = torch.cat([before.double(), x])
    y = sum(padded[j:j + x.shape[0]] * weight[:, j].double() for j in range(taps))
    return torch.nn.functional.silu(y)


def _recurrent64(case, x, w, spec, states, requests):
    """(the mixer's output, the states afterwards)."""
    H, D, V = spec.heads, spec.dim, spec.vdim
    lin = lambda name, t=x: t @ w[name].double().T
    kind = case["kind"]
    q, k, v = lin("q"), lin("k"), lin("v")
    new = {name: s.double() for name, s in states.items()}
    beta = None
    if kind == "decay":
        q, k, v = (torch.nn.functional.silu(t) for t in (q, k, v))
        g = torch.tensor(spec.decay, dtype=torch.float64, device=DEV)[None, :, None].expand(x.shape[0], H, D)
    elif kind == "gated":
        q = q * D ** -0.5
        g = torch.exp(torch.nn.functional.logsigmoid(lin("a2", lin("a1")) + w["a2.b"].double()) / spec.tau).unflatten(1, (H, D))
    else:
        raw = torch.cat([q, k, v], dim=1)
        weight = torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]])
        mixed = torch.empty_like(raw)
        for (row, _, n), r in zip(_segments(case), requests):
            mixed[row:row + n] = _short_conv64(raw[row:row + n], weight, states["conv"][r.slot])
            new["conv"][r.slot] = torch.cat([states["conv"][r.slot].double(), raw[row:row + n]])[-(spec.conv - 1):]
        q, k, v = mixed.split([H * D, H * D, H * V], dim=1)
        unit = lambda t: (t.unflatten(1, (H, D)) / torch.sqrt((t.unflatten(1, (H, D)) ** 2).sum(-1, keepdim=True) + 1e-6)).flatten(1)
        q, k = unit(q) * D ** -0.5, unit(k)
        step = torch.nn.functional.softplus(lin("a2", lin("a1")) + w["dt_bias"].double()).unflatten(1, (H, D))
        g = torch.exp(-torch.exp(w["A_log"].double())[None, :, None] * step)
        beta = torch.sigmoid(lin("b"))
    q, k, v = q.unflatten(1, (H, D)), k.unflatten(1, (H, D)), v.unflatten(1, (H, V))
    o = torch.empty_like(v)
    for (row, _, n), r in zip(_segments(case), requests):
        S = new["state"][r.slot].clone()
        for t in range(row, row + n):
            S = S * g[t, :, :, None]
            u = v[t]
            if beta is not None:
                u = beta[t][:, None] * (u - (S * k[t, :, :, None]).sum(1))
            S = S + k[t, :, :, None] * u[:, None, :]
            o[t] = (S * q[t, :, :, None]).sum(1)
        new["state"][r.slot] = S
    if kind == "decay":
        y = _norm64(o.flatten(1), w["norm"]) * torch.sigmoid(lin("g"))
    elif kind == "gated":
        y = _norm64(o, w["norm"]).flatten(1) * torch.nn.functional.silu(lin("g"))
    else:
        y = _norm64(o, w["norm"]).flatten(1) * torch.sigmoid(lin("g2", lin("g1")))
    return lin("o", y), new


def _latent64(case, x, w, spec, segments, kept):
    """kept(i): the cached rows in front of segment i."""
    n_rows, R = x.shape[0], spec.kv_rank
    q = (_norm64(x @ w["dq"].double().T, w["dq.norm"]) @ w["uq"].double().T).unflatten(1, (spec.heads, -1))
    down = x @ w["dkv"].double().T
    latent, shared = _norm64(down[:, :R], w["dkv.norm"]), down[:, R:]
    factor, original, fast, slow = spec.position.scaling
    dims, base = spec.position.dims, spec.position.base
    turn = lambda t: dims * math.log(original / (2 * math.pi * t)) / (2 * math.log(base))
    lo, hi = max(math.floor(turn(fast)), 0), min(math.ceil(turn(slow)), dims - 1)
    pair = torch.arange(dims // 2, dtype=torch.float64, device=DEV)
    f = base ** (-2 * pair / dims)
    r = ((pair - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    f = f / factor * r + f * (1 - r)
    magnitude = 0.1 * math.log(factor) + 1.0

    def rotate(t, at):                                       # neighbouring pairs
        angle = at.double()[:, None] * f[None, :]
        cos, sin = magnitude * angle.cos(), magnitude * angle.sin()
        cos, sin = (c.view(c.shape[0], *([1] * (t.dim() - 2)), -1) for c in (cos, sin))
        a, b = t[..., 0::2], t[..., 1::2]
        return torch.stack([a * cos - b * sin, b * cos + a * sin], dim=-1).flatten(-2)

    out = torch.empty((n_rows, spec.heads, spec.vdim), dtype=torch.float64, device=DEV)
    uk, uv = w["uk"].double().unflatten(0, (spec.heads, spec.dim)), w["uv"].double().unflatten(0, (spec.heads, spec.vdim))
    for i, (row, before, n) in enumerate(segments):
        at = torch.arange(before, before + n, device=DEV)
        c, kr = latent[row:row + n], rotate(shared[row:row + n], at)
        if before:
            rows = kept(i)
            c, kr = torch.cat([rows[:, :R], c]), torch.cat([rows[:, R:R + spec.rot_dim], kr])
        qs = torch.cat([q[row:row + n, :, :spec.dim], rotate(q[row:row + n, :, spec.dim:], at)], dim=-1)
        ks = torch.cat([torch.einsum("tr,hdr->thd", c, uk), kr[:, None, :].expand(-1, spec.heads, -1)], dim=-1)
        out[row:row + n] = _attend64(qs, ks, torch.einsum("tr,hdr->thd", c, uv), spec.softmax_scale, before)
    return out.flatten(1) @ w["o"].double().T


def exact(case, seed):
    torch.cuda.set_device(0)
    kind = case["kind"]
    with torch.no_grad():
        if kind == "step":
            return _step64(case, seed)
        spec = _spec(case)
        w = _local(_weights(case, seed, _tensor_specs(case, spec)))
        precision = Precision.of(case["dtype"])
        rt = Runtime(torch.device(DEV), precision, PAGE)
        part = MIXERS.build(spec.mixer, _local(w, "self_attn."), rt) if kind == "block" else MIXERS.build(spec, w, rt)
        held = _cache(case, seed, part.cache_need(), precision)
        entry, manager = held["entry"], held["manager"]
        segments = _segments(case)

        def rows_before(pool, i):                            # [context, kv heads, features] out of the pages
            pages = torch.tensor(manager.groups[entry.group_key].table[held["requests"][i].slot].copy(), device=DEV).long()
            before = segments[i][1]
            used = pages[:-(-before // PAGE)]
            return pool[used].transpose(1, 2).flatten(0, 1)[:before].double()

        x = _input(case, seed, held["ctx"].num_tokens, spec.mixer.hidden if kind == "block" else spec.hidden).double()
        pair = lambda i: (rows_before(entry.k, i), rows_before(entry.v, i))
        if kind == "block":
            stream = _block64(x, w, spec, segments, pair)
            h = _norm64(stream, torch.ones(x.shape[1], device=DEV))
            # a block leaves its own last product to the norm behind it, which adds it to the stream
            return {"stream": stream, "rows": h, "k": None, "v": None}
        if kind == "attention":
            return {"y": _attention64(x, w, spec, segments, pair), "k": None, "v": None}
        if kind == "latent":
            return {"y": _latent64(case, x, w, spec, segments, lambda i: rows_before(entry.k, i)[:, 0]), "k": None}
        y, new = _recurrent64(case, x, w, spec, held["states"], held["requests"])
        return {"y": y, **new}
