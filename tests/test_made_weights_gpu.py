"""Products whose second operand is the result of the kernel just before: that kernel lets its successor start at its own top, so a
product that read weights before waiting for it would read what lay there earlier."""
import pytest
import torch

from friday_inference_engine_b200 import ops
from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
P, I = lib.P, lib.I


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def made(source, gain, out):
    """out = the rows of `source`, normed: written after the next kernel may have started; NaN until then."""
    out.fill_(float("nan"))
    ops.rmsnorm(source, gain, 1e-6, out=out)


# 32-bit: one row to two blocks of rows, one column and four per warp, then tiles; bf16: the kernel for small matrices (32-bit
# results), weights on the M side, rows on the M side, pairs of SMs
@pytest.mark.parametrize("dtype,out_dtype,m,n,k", [
    (torch.float32, torch.float32, 1, 4096, 4096), (torch.float32, torch.float32, 7, 2048, 4096), (torch.float32, torch.float32, 16, 4096, 2048),
    (torch.float32, torch.float32, 40, 4096, 2048), (torch.bfloat16, torch.float32, 5, 4096, 4096), (torch.bfloat16, torch.float32, 16, 2048, 4096),
    (torch.bfloat16, torch.bfloat16, 8, 12288, 4096), (torch.bfloat16, torch.bfloat16, 200, 4096, 4096), (torch.bfloat16, torch.bfloat16, 600, 4096, 4096)])
def test_product_of_made_weights(dtype, out_dtype, m, n, k):
    x, source, gain = rnd((m, k), 1).to(dtype), rnd((n, k), 2).to(dtype), (1.0 + rnd((k,), 3, 0.1)).to(dtype)
    w = torch.empty_like(source)
    made(source, gain, w)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    store = 2.0 ** -8 if out_dtype == torch.bfloat16 else 0.0
    for _ in range(5):
        made(source, gain, w)
        got = ops.linear(x, w, out_dtype=out_dtype).double()
        # k sums that may cut instead of round, then the result's own rounding; a NaN fails
        assert bool(((got - want).abs() <= k * 2.0 ** -23 * size + store * want.abs()).all())


@pytest.mark.parametrize("layout", [0, 1])
def test_head_product_of_made_weights(layout):
    rows, heads, k, n = 8, 16, 128, 512
    f = lib.family("attention_latent")
    f.declare("attention_latent_head_linear", [P, I, I, I, I, P, I, I, P, I, I, I, P, I, I, P, I, I, I, I, P])
    shape = (heads * k, n) if layout == 0 else (heads * n, k)
    x, source, gain = rnd((rows, heads * k), 4).bfloat16(), rnd(shape, 5).bfloat16(), (1.0 + rnd((shape[1],), 6, 0.1)).bfloat16()
    w, out = torch.empty_like(source), torch.empty((rows, heads * n), device=DEV)
    seq = torch.zeros(rows, dtype=torch.int32, device=DEV)
    made(source, gain, w)
    parts = w.double().reshape(heads, k, n) if layout == 0 else w.double().reshape(heads, n, k).transpose(1, 2)
    a = x.double().reshape(rows, heads, k).transpose(0, 1)
    want, size = a @ parts, a.abs() @ parts.abs()
    for _ in range(5):
        made(source, gain, w)
        f.call("attention_latent_head_linear", x.data_ptr(), 1, heads * k, 0, k, w.data_ptr(), 1, layout, out.data_ptr(), 0, heads * n, n, None, 0, 0,
               seq.data_ptr(), rows, heads, k, n, 0)
        got = out.double().reshape(rows, heads, n).transpose(0, 1)
        assert bool(((got - want).abs() <= (k + 8) * 2.0 ** -23 * size).all())
