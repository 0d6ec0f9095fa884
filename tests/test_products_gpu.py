"""Matrix products at the edges of their kernels' ranges: rows around the tiles' heights, columns around their widths, k around
the blocks, unaligned rows, strided operands; against 64-bit sums."""
import pytest
import torch

from friday_inference_engine_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


# up to 8 / 16 rows a warp per columns, then tiles of 32 to 64 rows; one column and four per warp meet at 2,368 columns,
# narrow and wide results at 8,192; k = 4 (one 16-byte piece), around 32 and 128, long enough for every split
@pytest.mark.parametrize("m", [1, 2, 3, 5, 8, 9, 16, 17, 33, 57, 129, 333])
@pytest.mark.parametrize("n,k", [(1, 4), (65, 36), (129, 128), (2371, 260), (8195, 100), (3584, 4100)])
def test_float32_product(m, n, k):
    a, w, bias, res = rnd((m, k), 1), rnd((n, k), 2, 0.05), rnd((n,), 3), rnd((m, n), 4)
    want = a.double() @ w.double().T + bias.double() + res.double()
    # any order of k + 2 roundings of a sum errs by at most (k + 2) units of the sum of the terms' sizes
    bound = (k + 2) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T + bias.double().abs() + res.double().abs())
    out = res.clone()
    ops.backend()._linear_simt(a, w, bias, out, out)
    assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("m", [3, 12, 40])
@pytest.mark.parametrize("shift", [0, 1, 4])
def test_float32_product_strided_operands(m, shift):
    """Rows with a stride of their own; a start off the 16-byte boundary takes the general kernel."""
    n, k = 70, 64
    big_a, big_w = rnd((m, k + 8), 5), rnd((n, k + 12), 6)
    a, w = big_a[:, shift:shift + k], big_w[:, shift:shift + k]
    out = torch.empty((m, n), device=DEV)
    ops.backend()._linear_simt(a, w, None, None, out)
    bound = (k + 2) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((out.double() - a.double() @ w.double().T).abs() <= bound).all())


# pairs of SMs take the row tiles in groups: one group, two alike (17 and 33 row tiles of 256, wide), unequal ones, columns so
# few that a group has many row tiles, a last row tile of one row
@pytest.mark.parametrize("m,n,k", [(257, 512, 64), (4097, 9488, 64), (8449, 9600, 72), (3300, 272, 136), (5121, 4608, 64), (2561, 1040, 200)])
def test_row_groups_on_pairs(m, n, k):
    a, w, res = (rnd(s, i, c).bfloat16() for i, (s, c) in enumerate((((m, k), 1.0), ((n, k), 0.1), ((m, n), 1.0))))
    out = ops.linear(a, w, None, res)
    want = a.double() @ w.double().T + res.double()
    size = a.double().abs() @ w.double().abs().T + res.double().abs()
    # the product of two bf16 numbers is exact in 32 bits; k + 1 sums that may cut instead of round, then bf16's rounding
    assert bool(((out.double() - want).abs() <= (k + 1) * 2.0 ** -23 * size + 2.0 ** -8 * want.abs()).all())


# few rows and a small matrix: around 8 and 16 rows, columns around the blocks of 16, k around a warp's 32 and 256 and a block's
# 2,048 (one turn, several, sixteen warps), every epilogue; beyond these sizes the other kernel
@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("n,k", [(16, 8), (30, 264), (64, 2048), (2058, 72), (250, 2056), (96, 6152), (4096, 2304), (6000, 2048)])
def test_few_rows_small_matrix(m, n, k):
    big = rnd((m, k + 8), 1).bfloat16()
    a, w = big[:, :k], rnd((n, k), 2, k ** -0.5).bfloat16()
    bias, res32, res16 = rnd((n,), 3), rnd((m, n), 4), rnd((m, n), 5).bfloat16()
    z, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    slack = (k + 3) * 2.0 ** -23
    out = res32.clone()
    ops.backend()._linear_tc(a, w, bias, out, out)
    assert bool(((out.double() - (z + bias.double() + res32.double())).abs() <= slack * (size + bias.abs() + res32.abs())).all())
    out = torch.empty_like(res16)
    ops.backend()._linear_tc(a, w, None, res16, out, swap=-2)
    want = z + res16.double()
    assert bool(((out.double() - want).abs() <= slack * (size + res16.abs()) + 2.0 ** -8 * want.abs()).all())
    half = torch.empty((m, n // 2), dtype=torch.bfloat16, device=DEV)
    ops.backend()._linear_tc(a, w, None, None, half, act=1)
    gate, up = z[:, 0::2], z[:, 1::2]
    want = gate * torch.sigmoid(gate) * up
    wide = 2 * slack * (size[:, 0::2] * (up.abs() + 1.0) + size[:, 1::2] * (gate.abs() + 1.0))
    assert bool(((half.double() - want).abs() <= wide + 2.0 ** -8 * want.abs() + 1e-6).all())
    squared = torch.empty((m, n), dtype=torch.bfloat16, device=DEV)
    ops.backend()._linear_tc(a, w, None, None, squared, act=4)
    want = z.clamp(min=0.0) ** 2
    assert bool(((squared.double() - want).abs() <= 3 * slack * size * (z.abs() + 1.0) + 2.0 ** -8 * want + 1e-6).all())
