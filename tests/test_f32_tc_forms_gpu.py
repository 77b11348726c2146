"""32-bit products on the tensor cores: every combination of tile, cluster and ranges that is accepted has the same bits."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rows(m, k, seed):
    return torch.randn(m, k, generator=torch.Generator().manual_seed(seed)).to(DEV)


@pytest.mark.parametrize("ranges", [2, 8])
@pytest.mark.parametrize("m,tile,cluster", [(5, 0, 1), (32, 0, 1), (64, 16, 0), (64, 32, 0), (200, 16, 0), (64, 0, 1), (64, 64, 0)])
def test_what_is_left_to_choose_is_chosen_well(m, tile, cluster, ranges):
    """A cluster of one for few rows, a small tile for many: the part that is not given has to fit the part that is."""
    from mrun_b200.kernels import ops
    x, w = rows(m, 4096, 1), rows(4096, 4096, 2)
    want = ops.gemm_f32_tc(x, w, ranges=ranges, tile=64, cluster=ranges)
    assert torch.equal(ops.gemm_f32_tc(x, w, ranges=ranges, tile=tile, cluster=cluster), want)
    ops.tc5_check()


@pytest.mark.parametrize("tile", [16, 32])
def test_small_tiles_take_one_range_a_block(tile):
    from mrun_b200.kernels import ops
    with pytest.raises(ops.KernelError, match="cluster of 1 for 2 ranges"):
        ops.gemm_f32_tc(rows(5, 4096, 1), rows(256, 4096, 2), ranges=2, tile=tile, cluster=1)


@pytest.mark.parametrize("m", [3, 150])
@pytest.mark.parametrize("low,high", [(-112, 100), (-120, 100), (-126, 100), (-135, 100), (100, -120), (100, -135), (-70, -50)])
def test_tiny_operands_keep_their_digits(m, low, high):
    """Operands down to values with few significant bits of their own, beside large ones, so that the results are ordinary numbers;
    and results near the least normal value, where a rounding is up to 2^-150 of each of the ranges' sums."""
    from mrun_b200.kernels import ops
    k = 2048
    x, w = rows(m, k, 3) * 2.0 ** low, rows(200, k, 4) * 2.0 ** high
    if m > 100:
        x[:, ::7] *= 2.0 ** 20 if low < 0 else 2.0 ** -20             # beside each other in a row
    got, want = ops.gemm_f32_nt(x, w).double(), x.double() @ w.double().T
    ops.tc5_check()
    assert (got - want).norm() <= 6e-7 * want.norm() + (m * 200) ** 0.5 * 9 * 2.0 ** -150


@pytest.mark.parametrize("k", [2048, 12288])
@pytest.mark.parametrize("kind", ["positive", "close to one"])
def test_rows_of_one_sign(k, kind):
    """The tensor core cuts its additions, an error of one sign, which shows where the terms have one sign too: measured 2.5e-7 of
    a result whatever K; a chain of K rounded additions is 7e-7 off at K = 2,048 and 1.5e-6 at 12,288."""
    from mrun_b200.kernels import ops
    x, w = rows(40, k, 5), rows(300, k, 6)
    x, w = (x.abs(), w.abs()) if kind == "positive" else (1 + 0.01 * x, 1 + 0.01 * w)
    want = x.double() @ w.double().T
    got = ops.gemm_f32_nt(x, w)
    ops.tc5_check()
    assert (got.double() - want).norm() <= 5e-7 * want.norm()
