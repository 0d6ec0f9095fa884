"""Attention over a cached latent, few rows: the kernel whose blocks have all heads of a row, and the products per head in 16-byte
pieces, against 64-bit arithmetic."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
P, I, F = lib.P, lib.I, lib.F
PAGE = 64


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


# one to four heads per warp with idle warps, latents and rotated parts from one group of eight to the largest, keys around a round
# of 16 and a page of 64, one split, several, more splits than keys; 17 columns of a table; a dead row
@pytest.mark.parametrize("heads", [1, 8, 11, 16, 32])
@pytest.mark.parametrize("rank,rot", [(8, 8), (512, 64), (104, 128), (520, 8)])
@pytest.mark.parametrize("splits", [1, 3, 40])
def test_latent_rows(heads, rank, rot, splits):
    f = lib.family("attention_latent")
    f.declare("attention_latent", [P, P, P, P, P, I, I, P, P, P, I, I, I, I, I, F, I, P, I, P])
    f.declare("attention_latent_splits", [I] * 6)
    lens = [1, 16, 17, 64, 130, 1000]
    rows, width = len(lens) + 1, 17
    c, r = rnd((110, PAGE, rank), 1).bfloat16(), rnd((110, PAGE, rot), 2).bfloat16()
    table = torch.randperm(110, generator=torch.Generator().manual_seed(3))[:6 * width].reshape(6, width).to(torch.int32).to(DEV)
    seq = torch.tensor([3, 1, 0, 5, 4, 2, -1], dtype=torch.int32, device=DEV)
    pos = torch.tensor([n - 1 for n in lens] + [5], dtype=torch.int32, device=DEV)
    q, sink = rnd((rows, heads, rank + rot), 4), rnd((heads,), 5, 2.0)
    out = torch.full((rows, heads, rank), 9.0, device=DEV)
    scratch = torch.empty(rows * heads * splits * (rank + 2), device=DEV)
    scale = (rank + rot) ** -0.5
    args = (q.data_ptr(), out.data_ptr(), c.data_ptr(), r.data_ptr(), table.data_ptr(), width, PAGE, seq.data_ptr(), pos.data_ptr(), sink.data_ptr(), 0,
            rows, heads, rank, rot, scale, splits, scratch.data_ptr(), 1, torch.cuda.current_stream().cuda_stream)
    if rank > 512:
        with pytest.raises(lib.KernelError):
            f.call("attention_latent", *args)
        return
    assert 1 <= f.cdll.attention_latent_splits(rows, heads, 1000, rank, rot, 1) <= 63
    f.call("attention_latent", *args)
    for i, n in enumerate(lens):
        pages = table[int(seq[i])].long()
        keys = torch.cat([c[pages].reshape(-1, rank)[:n], r[pages].reshape(-1, rot)[:n]], dim=1).double()
        z = (q[i].double() @ keys.T) * scale
        w = torch.softmax(torch.cat([z, sink.double()[:, None]], dim=1), dim=1)[:, :n]
        want = w @ keys[:, :rank]
        # scores err by (rank + rot) units of their terms' size, weights by that much again, sums by n units
        slack = ((rank + rot + 20) * 2.0 ** -22 * ((q[i].double().abs() @ keys.abs().T) * scale).amax() + (n + 20) * 2.0 ** -22) * keys.abs().amax()
        assert bool(((out[i].double() - want).abs() <= slack).all())
    assert float(out[-1].abs().max()) == 0.0


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("rows,heads,k,n", [(1, 1, 8, 8), (8, 16, 128, 512), (9, 3, 136, 128), (17, 2, 512, 136), (5, 4, 600, 24), (3, 2, 20, 36)])
@pytest.mark.parametrize("dtypes", [(torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16)])
def test_head_products(layout, rows, heads, k, n, dtypes):
    f = lib.family("attention_latent")
    f.declare("attention_latent_head_linear", [P, I, I, I, I, P, I, I, P, I, I, I, P, I, I, P, I, I, I, I, P])
    tx, to = dtypes
    code = {torch.float32: 0, torch.bfloat16: 1}
    x, w = rnd((rows, heads * (k + 3) + 5), 6).to(tx), rnd((heads * k, n) if layout == 0 else (heads * n, k), 7, k ** -0.5).bfloat16()
    gate = rnd((rows, heads + 2), 8).to(to)
    seq = torch.zeros(rows, dtype=torch.int32, device=DEV)
    seq[rows // 2] = -1
    out = torch.full((rows, heads * (n + 1)), 9.0, dtype=to, device=DEV)
    f.call("attention_latent_head_linear", x.data_ptr(), code[tx], x.shape[1], 5, k + 3, w.data_ptr(), 1, layout, out.data_ptr(), code[to], heads * (n + 1),
           n + 1, gate.data_ptr(), heads + 2, 1, seq.data_ptr(), rows, heads, k, n, torch.cuda.current_stream().cuda_stream)
    for h in range(heads):
        a = x[:, 5 + h * (k + 3):5 + h * (k + 3) + k].double()
        m = w[h * k:(h + 1) * k].double() if layout == 0 else w[h * n:(h + 1) * n].double().T
        g = torch.sigmoid(gate[:, 1 + h].double())[:, None]
        want, size = (a @ m) * g, (a.abs() @ m.abs()) * g
        got = out[:, h * (n + 1):h * (n + 1) + n].double()
        live = seq >= 0
        store = 2.0 ** -8 if to == torch.bfloat16 else 0.0
        assert bool(((got - want).abs() <= (k + 8) * 2.0 ** -23 * size + store * want.abs())[live].all())
        assert bool((got[~live] == 9.0).all())
