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
    """The same bits as the rotation into query rows, in strided rows, nothing else touched."""
    from mrun_b200.kernels import ops
    heads, dim, rot_dim, rot_dims = 3, 10, 12, 8
    wide = torch.randn(9, heads * (dim + rot_dim) + 5, device=DEV).to(dtype)
    q = wide[:, :heads * (dim + rot_dim)]
    rot = torch.randn(9, rot_dims // 2, 2, device=DEV)
    rows = torch.empty(9, heads, 4 + rot_dim, dtype=dtype, device=DEV)
    ops.latent_query(q, rot, rot_dims, pairing, rows, heads, dim, rot_dim, 4)
    want = wide.clone()
    want[:, :heads * (dim + rot_dim)].unflatten(1, (heads, -1))[:, :, dim:] = rows[:, :, 4:]
    ops.latent_rotate(q, rot, rot_dims, pairing, heads, dim, rot_dim)
    assert (wide.float() - want.float()).abs().max() <= (1e-6 if dtype == torch.float32 else 0.04)     # one rounding apart at most
    keep = torch.ones_like(wide, dtype=torch.bool)
    keep[:, :heads * (dim + rot_dim)].unflatten(1, (heads, -1))[:, :, dim:dim + rot_dims] = False
    assert torch.equal(wide[keep], want[keep])
