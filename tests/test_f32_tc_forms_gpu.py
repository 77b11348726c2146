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
