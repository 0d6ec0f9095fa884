"""Latent attention of one row over thousands of keys: as many splits as the launcher asks for (more than the 256 that the merge takes
in one round), and counts around the rounds, some of them splits without a key; against 64-bit arithmetic."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
P, I, F = lib.P, lib.I, lib.F
PAGE = 64


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


@pytest.mark.parametrize("keys,splits", [(6000, None), (6000, 255), (6000, 256), (6000, 257), (300, 512), (300, 513), (5000, 700)])
@pytest.mark.parametrize("rank,rot,heads", [(512, 64, 3), (40, 8, 17)])
def test_many_splits(keys, splits, rank, rot, heads):
    f = lib.family("attention_latent")
    f.declare("attention_latent", [P, P, P, P, P, I, I, P, P, P, I, I, I, I, I, F, I, P, I, P])
    f.declare("attention_latent_splits", [I] * 6)
    if splits is None:
        splits = f.cdll.attention_latent_splits(1, heads, keys, rank, rot, 1)
        assert splits > 256
    pages = (keys + PAGE - 1) // PAGE
    c, r = rnd((pages + 3, PAGE, rank), 1).bfloat16(), rnd((pages + 3, PAGE, rot), 2).bfloat16()
    table = torch.randperm(pages + 3, generator=torch.Generator().manual_seed(3))[:pages].to(torch.int32).to(DEV)
    seq, pos = torch.zeros(1, dtype=torch.int32, device=DEV), torch.full((1,), keys - 1, dtype=torch.int32, device=DEV)
    q, sink = rnd((1, heads, rank + rot), 4), rnd((heads,), 5, 2.0)
    out, scratch = torch.full((1, heads, rank), 9.0, device=DEV), torch.full((heads * splits * (rank + 2),), float("nan"), device=DEV)
    scale = 2.0 * (rank + rot) ** -0.5
    f.call("attention_latent", q.data_ptr(), out.data_ptr(), c.data_ptr(), r.data_ptr(), table.data_ptr(), pages, PAGE, seq.data_ptr(), pos.data_ptr(),
           sink.data_ptr(), 0, 1, heads, rank, rot, scale, splits, scratch.data_ptr(), 1, torch.cuda.current_stream().cuda_stream)
    at = table.long()
    rows = torch.cat([c[at].reshape(-1, rank)[:keys], r[at].reshape(-1, rot)[:keys]], dim=1).double()
    z = (q[0].double() @ rows.T) * scale
    want = torch.softmax(torch.cat([z, sink.double()[:, None]], dim=1), dim=1)[:, :keys] @ rows[:, :rank]
    # scores err by (rank + rot) units of their terms' size, weights by that much again, sums by a unit per key
    slack = ((rank + rot + 20) * 2.0 ** -22 * ((q[0].double().abs() @ rows.abs().T) * scale).amax() + (keys + splits) * 2.0 ** -23) * rows.abs().amax()
    assert bool(((out[0].double() - want).abs() <= slack).all())
