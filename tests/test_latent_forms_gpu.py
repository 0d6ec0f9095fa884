"""Latent attention: both forms (a block with all heads of a row, a warp per head) on the same calls, on both sides of the rule that
chooses between them, and the products per head on both sides of theirs; against 64-bit arithmetic."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
P, I, F = lib.P, lib.I, lib.F
PAGE = 64


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def family():
    f = lib.family("attention_latent")
    f.declare("attention_latent_form", [P, P, P, P, P, I, I, P, P, P, I, I, I, I, I, F, I, P, I, I, P])
    f.declare("attention_latent_splits", [I] * 6)
    f.declare("attention_latent_head_linear", [P, I, I, I, I, P, I, I, P, I, I, I, P, I, I, P, I, I, I, I, P])
    return f


def test_which_form():
    splits = family().cdll.attention_latent_splits
    for rows, heads, keys, taken in [(8, 16, 500, True), (8, 1, 8000, True), (64, 1, 512, True), (64, 1, 513, False), (65, 1, 20, True), (257, 4, 20, False),
                                     (64, 4, 2048, True), (64, 4, 2049, False), (256, 4, 128, True), (1000, 5, 600, True), (32, 8, 20, True), (33, 8, 47, False), (33, 8, 48, True),
                                     (8, 16, 63, False), (8, 16, 64, True), (1000, 16, 600, True), (8, 32, 127, False), (8, 32, 128, True),
                                     (8, 17, 600, True), (9, 17, 600, False), (64, 22, 256, True), (64, 22, 255, False), (65, 32, 600, False), (8, 33, 600, False)]:
        assert (splits(rows, heads, keys, 512, 64, 1) > 0) == taken, (rows, heads, keys)
        assert splits(rows, heads, keys, 512, 64, 0) == 0            # 32-bit rows: always a warp per head


@pytest.mark.parametrize("all_heads", [0, 1])
@pytest.mark.parametrize("heads", [1, 4, 9, 17, 32])
@pytest.mark.parametrize("rank,rot", [(40, 8), (512, 64)])
@pytest.mark.parametrize("splits", [1, 5])
def test_both_forms(all_heads, heads, rank, rot, splits):
    f = family()
    lens = [1, 2, 17, 32, 33, 200]
    rows, width = len(lens), 4
    c, r = rnd((30, PAGE, rank), 1).bfloat16(), rnd((30, PAGE, rot), 2).bfloat16()
    table = torch.randperm(30, generator=torch.Generator().manual_seed(3))[:rows * width].reshape(rows, width).to(torch.int32).to(DEV)
    seq, pos = torch.arange(rows, dtype=torch.int32, device=DEV), torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    q, sink, out = rnd((rows, heads, rank + rot), 4), rnd((heads,), 5, 2.0), torch.full((rows, heads, rank), 9.0, device=DEV)
    scratch, scale = torch.empty(rows * heads * splits * (rank + 2), device=DEV), (rank + rot) ** -0.5
    f.call("attention_latent_form", q.data_ptr(), out.data_ptr(), c.data_ptr(), r.data_ptr(), table.data_ptr(), width, PAGE, seq.data_ptr(), pos.data_ptr(),
           sink.data_ptr(), 0, rows, heads, rank, rot, scale, splits, scratch.data_ptr(), 1, all_heads, torch.cuda.current_stream().cuda_stream)
    for i, n in enumerate(lens):
        at = table[i].long()
        keys = torch.cat([c[at].reshape(-1, rank)[:n], r[at].reshape(-1, rot)[:n]], dim=1).double()
        z = (q[i].double() @ keys.T) * scale
        want = torch.softmax(torch.cat([z, sink.double()[:, None]], dim=1), dim=1)[:, :n] @ keys[:, :rank]
        # scores err by (rank + rot) units of their terms' size, weights by that much again, sums by n units
        slack = ((rank + rot + 20) * 2.0 ** -22 * ((q[i].double().abs() @ keys.abs().T) * scale).amax() + (n + 20) * 2.0 ** -22) * keys.abs().amax()
        assert bool(((out[i].double() - want).abs() <= slack).all())


# blocks of 8 rows x heads x columns on both sides of the lines: layout 0, k of 24, 64, 128 and 192; layout 1, k of 128 and 512
@pytest.mark.parametrize("layout,rows,heads,k,n", [(0, 9, 2, 24, 64), (0, 9, 2, 32, 64), (0, 85, 31, 64, 40), (0, 88, 31, 64, 40), (0, 340, 8, 128, 512),
                                                   (0, 345, 8, 128, 512), (0, 400, 8, 192, 136), (1, 130, 16, 128, 136), (1, 64, 32, 512, 128), (1, 65, 32, 512, 128)])
def test_head_products_at_the_lines(layout, rows, heads, k, n):
    f = family()
    x, w = rnd((rows, heads * k), 6).bfloat16(), rnd((heads * k, n) if layout == 0 else (heads * n, k), 7, k ** -0.5).bfloat16()
    seq, out = torch.zeros(rows, dtype=torch.int32, device=DEV), torch.full((rows, heads * n), 9.0, device=DEV)
    f.call("attention_latent_head_linear", x.data_ptr(), 1, heads * k, 0, k, w.data_ptr(), 1, layout, out.data_ptr(), 0, heads * n, n, None, 0, 0, seq.data_ptr(),
           rows, heads, k, n, torch.cuda.current_stream().cuda_stream)
    a = x.double().reshape(rows, heads, k).transpose(0, 1)
    m = w.double().reshape(heads, k, n) if layout == 0 else w.double().reshape(heads, n, k).transpose(1, 2)
    got = out.double().reshape(rows, heads, n).transpose(0, 1)
    assert bool(((got - a @ m).abs() <= (k + 8) * 2.0 ** -23 * (a.abs() @ m.abs())).all())
