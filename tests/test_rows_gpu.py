"""The row norms of 32-bit streams at the edges of their kernels' widths, against 64-bit arithmetic."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


# rows of four-number groups, one to four per thread, partial ones; other widths take the older kernel
@pytest.mark.parametrize("width", [4, 100, 1024, 1028, 2048, 4092, 4096, 4100, 1030])
@pytest.mark.parametrize("dtypes", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
def test_row_norms(width, dtypes):
    r = lib.family("residual")
    P, I, F = lib.P, lib.I, lib.F
    r.declare("residual_layernorm_cast", [P, I, P, P, I, P, I, I, I, F, P])
    r.declare("residual_norm_cast", [P, I, P, I, F, P, I, I, I, F, P])
    code = {torch.float32: 0, torch.bfloat16: 1}
    ti, to = dtypes
    x = (rnd((5, width), 1, 2.0) + 3.0).to(ti)
    w, b = rnd((width,), 2).bfloat16(), rnd((width,), 3).bfloat16()
    st = torch.cuda.current_stream().cuda_stream
    eps = 1e-5
    y = torch.empty((5, width), dtype=to, device=DEV)
    r.call("residual_layernorm_cast", x.data_ptr(), code[ti], w.data_ptr(), b.data_ptr(), 1, y.data_ptr(), code[to], 5, width, eps, st)
    d = x.double() - x.double().mean(-1, keepdim=True)
    dev = torch.sqrt((d * d).mean(-1, keepdim=True) + eps)
    want = d / dev * w.double() + b.double()
    store = 2.0 ** -8 if to == torch.bfloat16 else 0.0
    # the mean errs by some units of the row's largest number, everything after it by a few units of its own
    near = 2.0 ** -20 * (want.abs() + w.double().abs() * (d.abs() + x.double().abs().amax()) / dev + 1.0)
    assert bool(((y.double() - want).abs() <= near + store * want.abs()).all())
    r.call("residual_norm_cast", x.data_ptr(), code[ti], w.data_ptr(), 1, 1.0, y.data_ptr(), code[to], 5, width, eps, st)
    want = x.double() / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + eps) * (1.0 + w.double())
    # 1 + w is formed in 32 bits: its rounding stays where the two nearly cancel
    assert bool(((y.double() - want).abs() <= 2.0 ** -20 * want.abs() + 2.0 ** -22 * x.double().abs() + store * want.abs()).all())
