"""Products of few rows with few columns and a long k, or many columns and a short k, on both sides of the lines where the kernel for
small matrices ends."""
import pytest
import torch

from friday_inference_engine_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(64, 65536), (127, 24584), (128, 24576), (128, 24584), (200, 32768), (256, 36864), (256, 36872), (384, 16384), (384, 16392), (384, 24576), (384, 24584),
                                 (4608, 64), (4616, 64), (6145, 256), (12288, 1024), (12304, 1024)])
def test_few_rows_at_the_lines(m, n, k):
    g = torch.Generator().manual_seed(m * n)
    x, w = (torch.randn(s, generator=g).bfloat16().to(DEV) for s in ((m, k), (n, k)))
    got = ops.linear(x, w, out_dtype=torch.float32)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # the products are exact in 32 bits; k sums that may cut instead of round
    assert bool(((got.double() - want).abs() <= k * 2.0 ** -23 * size).all())
