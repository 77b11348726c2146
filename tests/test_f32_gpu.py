"""The 32-bit products at the edges of their tiles: against 64 bits, and bit for bit the same whichever
kernel or tile takes a row."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rows(m, k, seed):
    return torch.randn(m, k, generator=torch.Generator().manual_seed(seed)).to(DEV)


@pytest.mark.parametrize("n,k", [(1, 4), (31, 64), (33, 128), (130, 132), (64, 516), (200, 130), (513, 1000), (16400, 36)])
def test_products_of_every_row_count_agree_in_bits(n, k):
    """K in and out of the 16-byte copies, N around the blocks' 16, 32, 64 and 128 rows of weights; M on both
    sides of every choice of kernel."""
    from mrun_b200.kernels import ops
    x, w = rows(300, k, 1), rows(n, k, 2)
    whole = ops.gemm_f32_nt(x, w)
    want = x.double() @ w.double().T
    # one rounding a term of a chain of k: k * 2^-24 of the terms' size at worst, its root on average
    assert (whole.double() - want).abs().max() <= 2.0 ** -24 * 6 * math.sqrt(k) * (x.double().abs() @ w.double().abs().T).max()
    for m in (1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 33, 64, 65, 129):
        assert torch.equal(ops.gemm_f32_nt(x[:m].contiguous(), w), whole[:m]), m
    wide = rows(21, k + 3, 3)                      # rows that do not start on 16 bytes
    for m in (1, 4, 21):
        assert torch.equal(ops.gemm_f32_nt(wide[:m, 3:], w), ops.gemm_f32_nt(wide[:m, 3:].contiguous(), w)), m


@pytest.mark.parametrize("m", [1, 5, 16, 40])
def test_batched_products(m):
    from mrun_b200.kernels import ops
    x, w = rows(m, 6 * 72, 4).view(m, 6, 72), rows(6 * 40, 72, 5).view(6, 40, 72)
    out = torch.full((m, 6, 48), 7.0, device=DEV)
    ops.gemm_f32_nt_batched(x.transpose(0, 1), w, out[:, :, :40].transpose(0, 1))
    for b in range(6):
        assert torch.equal(out[:, b, :40], ops.gemm_f32_nt(x[:, b].contiguous(), w[b].contiguous()))
    assert (out[:, :, 40:] == 7.0).all()
