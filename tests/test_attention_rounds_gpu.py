"""CUDA-core attention at the edges of its rounds of keys: heads at the ends of a lane's 1, 2, 4 and 8 dimensions, keys around rounds
of 4, 8 and 16 and their remainders, values of another size than keys, windows with kept keys, splits; against 64-bit arithmetic."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
P, I, F = lib.P, lib.I, lib.F
PAGE = 8
KEYS = [1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 37, 64, 100]


def rnd(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd,vd", [(8, 8), (32, 32), (33, 20), (64, 64), (24, 65), (128, 128), (129, 128), (192, 200), (256, 256), (100, 256)])
@pytest.mark.parametrize("window,keep,splits,copies", [(0, 0, 1, 1), (24, 3, 1, 1), (0, 0, 3, 1), (0, 0, 1, 40)])
def test_rounds_of_keys(dtype, hd, vd, window, keep, splits, copies):
    f = lib.family("attention_simt")
    f.declare("attention_simt_masked", [P, I, P, P, P, P, I, I, P, P, I, I, I, I, I, I, I, F, F, I, P, I, P])
    nq, nkv, scale = 6, 2, hd ** -0.5
    lens = KEYS * copies                          # many copies: more blocks than two per SM
    rows, width = len(lens) + 1, (max(KEYS) + PAGE - 1) // PAGE
    pages = len(KEYS) * width
    k, v = rnd((pages, PAGE, nkv, hd), 1).to(dtype), rnd((pages, PAGE, nkv, vd), 2).to(dtype)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(3)).reshape(len(KEYS), width).to(torch.int32).to(DEV)
    seq = torch.tensor([i % len(KEYS) for i in range(len(lens))] + [-1], dtype=torch.int32, device=DEV)
    pos = torch.tensor([n - 1 for n in lens] + [7], dtype=torch.int32, device=DEV)
    q, out = rnd((rows, nq * hd), 4).to(dtype), torch.full((rows, nq * vd), 9.0, dtype=dtype, device=DEV)
    scratch = torch.empty(rows * nq * splits * (vd + 2), device=DEV)
    f.call("attention_simt_masked", q.data_ptr(), nq * hd, out.data_ptr(), k.data_ptr(), v.data_ptr(), table.data_ptr(), width, PAGE, seq.data_ptr(),
           pos.data_ptr(), rows, nq, nkv, hd, vd, window, keep, scale, 1.0, splits, scratch.data_ptr(), 1 if dtype == torch.bfloat16 else 0,
           torch.cuda.current_stream().cuda_stream)
    for i, n in enumerate(lens):
        first = max(0, n - window) if window else 0
        seen = list(range(min(keep, first))) + list(range(first, n))
        at = table[i % len(KEYS)].long()
        ks, vs = (x[at].reshape(-1, nkv, x.shape[-1])[seen].double().repeat_interleave(nq // nkv, dim=1) for x in (k, v))
        z = torch.einsum("hd,khd->hk", q[i].reshape(nq, hd).double(), ks) * scale
        want = torch.einsum("hk,khd->hd", torch.softmax(z, dim=1), vs)
        # scores err by hd units of their terms' size, weights by that much and a few units more, sums by a unit per key; then the store
        size = torch.einsum("hd,khd->hk", q[i].reshape(nq, hd).double().abs(), ks.abs()).amax() * scale
        slack = ((hd + 8) * 2.0 ** -23 * size + (len(seen) + 16) * 2.0 ** -23) * 2 * vs.abs().amax()
        store = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
        assert bool(((out[i].reshape(nq, vd).double() - want).abs() <= slack + store * want.abs()).all()), n
    assert float(out[-1].abs().max()) == 0.0
