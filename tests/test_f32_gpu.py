"""The 32-bit products and the tiled 32-bit attention at the edges of their tiles: against 64 bits, and bit for bit
the same whichever kernel or tile takes a row."""
from __future__ import annotations

import math

import pytest
import torch

from test_attention_gpu import Case

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


def test_products_of_more_rows_than_small_tiles_reach():
    """Few columns would choose tiles of 32 rows, of which a grid holds 65,535."""
    from mrun_b200.kernels import ops
    m = 65535 * 32 + 5
    x, w = torch.randn(m, 4, generator=torch.Generator(device=DEV).manual_seed(6), device=DEV), rows(8, 4, 7)
    got, want = ops.gemm_f32_nt(x, w), x.double() @ w.double().T
    assert (got.double() - want).abs().max() <= 2.0 ** -24 * 4 * (x.double().abs() @ w.double().abs().T).max()


@pytest.mark.parametrize("m", [1, 5, 16, 40])
def test_batched_products(m):
    from mrun_b200.kernels import ops
    x, w = rows(m, 6 * 72, 4).view(m, 6, 72), rows(6 * 40, 72, 5).view(6, 40, 72)
    out = torch.full((m, 6, 48), 7.0, device=DEV)
    ops.gemm_f32_nt_batched(x.transpose(0, 1), w, out[:, :, :40].transpose(0, 1))
    for b in range(6):
        assert torch.equal(out[:, b, :40], ops.gemm_f32_nt(x[:, b].contiguous(), w[b].contiguous()))
    assert (out[:, :, 40:] == 7.0).all()


@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size", [(8, 8, 64, 32), (32, 8, 128, 16), (32, 2, 64, 16), (16, 1, 128, 4),
                                                               (16, 1, 64, 16), (6, 2, 128, 1), (8, 2, 128, 24), (9, 3, 64, 8)])
@pytest.mark.parametrize("window", [0, 37, 64])
def test_tiled_attention_against_plain(heads, kv_heads, head_dim, page_size, window):
    segments = [(0, 70), (129, 1), (63, 2), (300, 1), (15, 33), (0, 1), (64, 64)]
    scale = head_dim ** -0.5
    case = Case(segments, heads, kv_heads, head_dim, page_size, torch.float32, seed=head_dim + window, window=window)
    want = case.reference(scale)
    got = case.run(scale)
    assert (got - want).abs().max() <= 2e-5 * want.abs().max()
    # the sums' order differs from the kernel with a block a token and head, nothing else does
    assert (got - case.run(scale, force_generic=True)).abs().max() <= 4e-6 * want.abs().max()


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(4, 4, 64), (8, 2, 128), (16, 1, 128), (32, 2, 64)])
@pytest.mark.parametrize("window", [0, 50, -48])
def test_tiled_attention_is_the_same_in_bits_for_every_cutting(heads, kv_heads, head_dim, window):
    """A request's last tokens alone and in portions of any size, under a window and under chunks."""
    scale, total = head_dim ** -0.5, 150
    whole = Case([(0, total)], heads, kv_heads, head_dim, 16, torch.float32, seed=3, window=window)
    want = whole.run(scale)
    for start, n in ((149, 1), (64, 1), (128, 22), (63, 3), (100, 17), (1, 70)):
        part = Case([(start, n)], heads, kv_heads, head_dim, 16, torch.float32, seed=3, window=window)
        part.kd, part.vd, part.table = whole.kd, whole.vd, whole.table
        part.group.block_tables, part.group.max_blocks = whole.group.block_tables, whole.group.max_blocks
        part.ctx.token_slot = whole.ctx.token_slot[start:start + n].contiguous()
        part.qd = whole.qd[start:start + n].contiguous()
        assert torch.equal(part.run(scale), want[start:start + n]), (start, n)


def test_what_a_row_does_not_see_does_not_enter_its_sums():
    """Later keys and values of a tile that are infinite or no numbers leave the earlier rows alone."""
    case = Case([(0, 40)], 4, 2, 64, 16, torch.float32, seed=9)
    want = case.run(0.125)
    page, at = case.seg_pages[0][30 // 16], 30 % 16
    case.kd[page, :, at] = float("nan")
    case.vd[page, :, at] = float("inf")
    got = case.run(0.125)
    assert torch.equal(got[:30], want[:30]) and not torch.isfinite(got[30:]).all()


def test_tiled_attention_leaves_unaligned_outputs_to_the_general_kernel():
    """Outputs, keys or values that do not start on 16 bytes are taken as before."""
    from mrun_b200.kernels.attention import paged_attention
    case = Case([(0, 20), (30, 1)], 4, 2, 64, 16, torch.float32, seed=10)
    want = case.run(0.125)
    shifted = lambda t: torch.empty(t.numel() + 1, device=DEV)[1:].view(t.shape).copy_(t)
    for which in range(3):
        cache, out = Case.Cache(), torch.empty(case.tokens, 4 * 64, device=DEV)
        cache.k, cache.v = case.kd, case.vd
        if which == 0:
            out = shifted(out)
        elif which == 1:
            cache.k = shifted(case.kd)
        else:
            cache.v = shifted(case.vd)
        paged_attention(case.qd, case.qd.stride(0), out, cache, case.group, case.ctx, 4, 0.125, 0)
        assert (out.cpu() - want).abs().max() <= 4e-6 * want.abs().max()


@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size", [(8, 8, 64, 32), (32, 8, 128, 16), (32, 2, 64, 16), (16, 1, 128, 4),
                                                               (6, 2, 128, 1), (9, 3, 64, 8), (10, 2, 128, 16)])
@pytest.mark.parametrize("window", [0, 37])
def test_tiles_of_every_size_give_the_same_bits(heads, kv_heads, head_dim, page_size, window, monkeypatch):
    """Portions and single tokens, contexts within and beyond the first quarter of a tile, in tiles of 64, 16 and 4 rows."""
    from mrun_b200.kernels import attention
    segments = [(0, 70), (129, 1), (63, 2), (300, 1), (15, 33), (0, 1), (0, 17), (9, 1), (64, 64)]
    scale = head_dim ** -0.5
    case = Case(segments, heads, kv_heads, head_dim, page_size, torch.float32, seed=head_dim + window, window=window)
    want = case.reference(scale)
    results = []
    for rows in attention.F32_TILE_ROWS:
        case.ctx.shared.clear()
        monkeypatch.setattr(attention, "f32_tile_rows", lambda *a: rows)
        results.append(case.run(scale))
    assert (results[0] - want).abs().max() <= 2e-5 * want.abs().max()
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])
