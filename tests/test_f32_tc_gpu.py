"""32-bit products on the tensor cores: at the edges of their tiles, boxes and ranges, bit for bit the same for every way of
cutting the work, and against 64 bits."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TILES = (16, 32, 64, 96, 112, 128, 144, 160, 176, 192)


def rows(m, k, seed):
    return torch.randn(m, k, generator=torch.Generator().manual_seed(seed)).to(DEV)


def bound(k):
    """Worst case over the sum of the terms' sizes: what the six products leave out (2^-24), the tensor core's 24 additions
    of a 64-k sum, each cut at 2^-23, and the 32-bit additions of the sums and ranges."""
    return 2.0 ** -24 + 24 * 2.0 ** -23 + (k / 64 + 8) * 2.0 ** -24


@pytest.mark.parametrize("n,k", [(64, 2048), (127, 2052), (129, 4100), (1000, 2080), (6200, 2048)])
def test_every_row_count(n, k):
    """N around the tile's 128 rows, K in and out of the boxes' 32 and 64; rows around every tile of tokens; rows of x that do
    not start on 16 bytes."""
    from mrun_b200.kernels import ops
    x, w = rows(400, k, 1), rows(n, k, 2)
    whole = ops.gemm_f32_nt(x, w)
    want = x.double() @ w.double().T
    assert (whole.double() - want).abs().max() <= bound(k) * (x.double().abs() @ w.double().abs().T).max()
    assert (whole.double() - want).norm() <= 6e-7 * want.norm()        # measured: 3.5e-7, whatever K
    for m in (1, 15, 16, 17, 32, 33, 64, 65, 97, 112, 113, 177, 200, 385):
        assert torch.equal(ops.gemm_f32_nt(x[:m].contiguous(), w), whole[:m]), m
    wide = torch.cat([x[:, :3], x], dim=1)
    for m in (1, 5, 40):
        assert torch.equal(ops.gemm_f32_nt(wide[:m, 3:], w), whole[:m]), m
    ops.tc5_check()


@pytest.mark.parametrize("m,n,k", [(13, 200, 2052), (300, 300, 1100)])
@pytest.mark.parametrize("ranges", [1, 2, 3, 8])
def test_tiles_and_clusters_agree_in_bits(m, n, k, ranges):
    """Ranges of k that differ by a block, as the blocks of a cluster and one after the other."""
    from mrun_b200.kernels import ops
    x, w = rows(m, k, 3), rows(n, k, 4)
    results = [ops.gemm_f32_tc(x, w, ranges=ranges, tile=tile, cluster=cluster) for tile in TILES for cluster in {1, ranges}
               if tile > 32 or (m <= tile and cluster == ranges)]
    ops.tc5_check()
    assert all(torch.equal(got, results[0]) for got in results)


def test_portions_of_long_inputs(monkeypatch):
    from mrun_b200.kernels import ops
    x, w = rows(150, 2048, 5), rows(130, 2048, 6)
    whole = ops.gemm_f32_nt(x, w)
    monkeypatch.setattr(ops, "F32_TC_SCRATCH", 6 * 2048 * 40)
    assert torch.equal(ops.gemm_f32_nt(x, w), whole)
    out = torch.empty(0, 130, device=DEV)
    assert ops.gemm_f32_nt(x[:0], w, out) is out


@pytest.mark.parametrize("m", [20, 150])
def test_values_without_parts(m):
    """Infinities, values that are no numbers and sums out of range come out as a chain of multiply-adds has them; what is
    tiny, or beside such a value, keeps its digits."""
    from mrun_b200.kernels import ops
    k, inf, nan = 2048, float("inf"), float("nan")
    x, w = rows(m, k, 7), rows(200, k, 8)
    x[3, 5], x[4, 7], w[9, 100] = inf, nan, -inf
    x[5, 0], x[5, 1], w[12] = inf, -inf, 0.0
    x[6] *= 1e30
    w[11] *= 1e12                                         # sums beyond the largest value
    x[7, 3] = 3.4028e38                                   # rounds up to infinity in bfloat16
    x[8] *= 1e-30
    got, want = ops.gemm_f32_nt(x, w), x.double() @ w.double().T
    fits = want.abs() < 3.4e38
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isposinf(got) | torch.isneginf(got), ~fits & ~torch.isnan(want))
    assert torch.equal(got[~fits & ~torch.isnan(want)] > 0, want[~fits & ~torch.isnan(want)] > 0)
    size = (x.double().abs() @ w.double().abs().T)[fits]
    assert ((got.double() - want)[fits].abs() <= bound(k) * size).all()
