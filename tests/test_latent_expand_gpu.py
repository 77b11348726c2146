"""Latent attention with a rotated key part whose prompt steps make keys and values from the latents: against the
plain formulas in every cutting, beside steps that stay with the latent."""
from __future__ import annotations

import pytest
import torch

import plain_zasesun as plain
import test_zasesun_gpu as zasesun

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# heads, dim, rot_dim, vdim, q_rank, kv_rank, scale, (rotating features, base, stretch)
SHAPES = {
    "192": (3, 128, 64, 128, 40, 512, 0.05, (64, 1000.0, (4.0, 32, 8.0, 1.0))),
    "192, some features do not rotate": (2, 160, 32, 64, 24, 264, 0.05, (16, 100.0, None)),
    "128": (5, 96, 32, 128, 33, 136, 0.08, (32, 500.0, None)),
    "64": (2, 32, 32, 64, 17, 400, 0.1, (32, 500.0, None)),
}


@pytest.mark.parametrize("name", sorted(SHAPES))
@pytest.mark.parametrize("expand", [4, 0])
def test_keys_and_values_made_from_latents(name, expand, monkeypatch):
    from mrun_b200.parts import latent_attention
    monkeypatch.setattr(latent_attention, "EXPAND_ROWS", expand)
    monkeypatch.setitem(zasesun.MIXERS, name, SHAPES[name])
    part, rt, tensors, settings = zasesun.build_mixer(name, "bfloat16")
    assert part.expandable
    made = []
    monkeypatch.setattr(part, "_expanded", lambda *a, inner=part._expanded: made.append(a[-1]) or inner(*a))
    total = 700
    h = torch.randn(total, 72, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
    want = plain.latent_attention(h.double(), tensors, "m", settings, 1e-5, torch.arange(total))
    for portions in ([total], [300, 400], [500, 1, 3, 2, 194], [128, 128, 127, 129, 188], [20, 40, 600, 5] + [1] * 35):
        zasesun.close(zasesun.run_mixer(part, rt, h, portions), want, "bfloat16", f"portions {portions[:6]}")
    assert bool(made) == bool(expand)


@pytest.mark.parametrize("pairing", ["interleaved", "half"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rotation_in_place(pairing, dtype):
    """Within the roundings of one product sum of the rotation in 64 bits, in strided rows, nothing else touched."""
    from mrun_b200.kernels import ops
    heads, dim, rot_dim, rot_dims = 3, 10, 12, 8
    wide = torch.randn(9, heads * (dim + rot_dim) + 5, device=DEV).to(dtype)
    q = wide[:, :heads * (dim + rot_dim)]
    rot = torch.randn(9, rot_dims // 2, 2, device=DEV)
    part = q.double().unflatten(1, (heads, -1))[:, :, dim:dim + rot_dims]
    lanes = (slice(0, None, 2), slice(1, None, 2)) if pairing == "interleaved" else (slice(0, rot_dims // 2), slice(rot_dims // 2, None))
    x, y, c, s = part[:, :, lanes[0]], part[:, :, lanes[1]], rot[:, None, :, 0].double(), rot[:, None, :, 1].double()
    before = wide.clone()
    ops.latent_rotate(q, rot, rot_dims, pairing, heads, dim, rot_dim)
    got = q.double().unflatten(1, (heads, -1))[:, :, dim:dim + rot_dims]
    # two products and a sum in 32 bits (24 significant bits: 2^-24 of a value each), then the result in bfloat16 (8: 2^-8)
    unit = 3 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    for lane, want, size in ((lanes[0], x * c - y * s, (x * c).abs() + (y * s).abs()), (lanes[1], y * c + x * s, (y * c).abs() + (x * s).abs())):
        assert ((got[:, :, lane] - want).abs() <= unit * size).all()
    keep = torch.ones_like(wide, dtype=torch.bool)
    keep[:, :heads * (dim + rot_dim)].unflatten(1, (heads, -1))[:, :, dim:dim + rot_dims] = False
    assert torch.equal(wide[keep], before[keep])
