"""The sums of squares that a product leaves for the norm of its result: a tile's columns are added one after another, whichever
kernel and however many warps finish the tile, so that a row's norm does not depend on them."""
import numpy as np
import pytest
import torch

from friday_inference_engine_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16().to(DEV)


# pairs of SMs: one row tile and many, widths of an even and an odd number of 16-column groups, a last tile that is narrower;
# fewer rows: single SMs
@pytest.mark.parametrize("m,n,k", [(257, 512, 64), (300, 1040, 200), (2561, 1040, 72), (513, 3584, 64), (4097, 2320, 64), (160, 272, 136)])
def test_squares_are_added_column_by_column(m, n, k):
    x, w, gain, res = rnd((m, k), 1), rnd((n, k), 2, 0.2), rnd((n,), 3), rnd((m, n), 4)
    out, normed = ops.linear_norm(x, w, gain, 1e-6, None, res)
    assert isinstance(normed, ops.DeferredNorm)
    parts = normed.ssq.shape[0]
    rows, sums = out.float().cpu().numpy(), normed.ssq.cpu().numpy()
    width = ops.backend().plan(m, n, k)[1]
    assert parts == (n + width - 1) // width
    for part in range(parts):
        want = np.zeros(m, dtype=np.float32)
        for c in range(part * width, min(n, (part + 1) * width)):
            want = want + rows[:, c] * rows[:, c]          # a bf16 number's square is exact in 32 bits
        assert np.array_equal(sums[part], want)
