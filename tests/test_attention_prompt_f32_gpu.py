"""fp32 prompts' attention in tiles, against 64-bit arithmetic: edges of tiles of rows and keys, windows, continued prompts, shared heads,
a sequence that is over, values that are not finite behind the mask."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
P, I, F = lib.P, lib.I, lib.F


class Case:
    def __init__(self, lens, pos0, nq, nkv, hd, window, page=64, seed=0, poison=None):
        g = torch.Generator(device=DEV).manual_seed(seed)
        self.lens, self.pos0, self.sizes, self.window, self.page = lens, pos0, (nq, nkv, hd), window, page
        n, rows, total = len(lens), sum(lens), [a + b for a, b in zip(lens, pos0)]
        self.width = max(-(-t // page) for t in total)
        self.table = torch.randperm(n * self.width + 1, device=DEV)[:n * self.width].int().view(n, self.width).contiguous()
        self.kp, self.vp = (torch.full((n * self.width + 1, page, nkv, hd), float("nan"), device=DEV) for _ in range(2))
        self.k, self.v = ([torch.randn(t, nkv, hd, device=DEV, generator=g) for t in total] for _ in range(2))
        if poison is not None:
            self.k[0][poison], self.v[0][poison] = float("nan"), float("inf")
        for s, t in enumerate(total):
            for j in range(0, t, page):
                at = self.table[s, j // page].long()
                m = min(page, t - j)
                self.kp[at, :m], self.vp[at, :m] = self.k[s][j:j + m], self.v[s][j:j + m]
        self.q = torch.randn(rows, (nq + 2 * nkv) * hd, device=DEV, generator=g)
        self.start = [sum(lens[:i]) for i in range(n)]

    def run(self, over=()):
        fam = lib.family("attention_simt")
        fam.declare("attention_simt_prompt", [P, I, P, P, P, P, I, I, P, P, P, P, I, I, I, I, I, I, F, P])
        nq, nkv, hd = self.sizes
        t = [torch.tensor(v, dtype=torch.int32, device=DEV) for v in
             ([-1 if i in over else i for i, m in enumerate(self.lens) for _ in range(m)], self.start, self.lens, self.pos0)]
        out = torch.full((sum(self.lens), nq * hd), 7.0, device=DEV)
        fam.call("attention_simt_prompt", self.q.data_ptr(), self.q.stride(0), out.data_ptr(), self.kp.data_ptr(), self.vp.data_ptr(), self.table.data_ptr(),
                 self.width, self.page, t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(), len(self.lens), max(self.lens), nq, nkv, hd,
                 self.window, hd ** -0.5, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return out

    def exact(self):
        nq, nkv, hd = self.sizes
        outs = []
        for s, m in enumerate(self.lens):
            q = self.q[self.start[s]:self.start[s] + m, :nq * hd].double().view(m, nq, hd)
            k, v = (x[s].double().repeat_interleave(nq // nkv, 1) for x in (self.k, self.v))
            i, j = torch.arange(m, device=DEV)[:, None] + self.pos0[s], torch.arange(m + self.pos0[s], device=DEV)[None]
            hidden = (j > i) | (j <= i - self.window if self.window else j < 0)
            w = (torch.einsum("thd,khd->htk", q, k) * hd ** -0.5).masked_fill(hidden, -float("inf")).softmax(-1)
            outs.append(torch.einsum("htk,khd->thd", w, v).reshape(m, -1))
        return torch.cat(outs)


@pytest.mark.parametrize("lens,pos0,nq,nkv,hd,window", [([9, 1, 70], [0, 5, 0], 28, 4, 128, 0), ([65, 33], [0, 0], 3, 1, 32, 24), ([100, 7], [5, 64], 6, 3, 20, 9),
                                                        ([130], [70], 64, 1, 96, 0), ([40, 40], [0, 31], 2, 2, 64, 1), ([300], [0], 8, 4, 4, 100),
                                                        ([70] * 10, [0] * 10, 64, 64, 36, 24)])
@pytest.mark.parametrize("page", [64, 16])
def test_prompt(lens, pos0, nq, nkv, hd, window, page):
    c = Case(lens, pos0, nq, nkv, hd, window, page)
    # scores of 128 terms and exponentials in fp32: some 2^-20 of the values, which are below 5
    assert (c.run().double() - c.exact()).abs().max() <= 5 * 2.0 ** -18


def test_sequence_that_is_over_and_what_lies_behind_the_mask():
    c = Case([50, 20, 33], [0, 3, 0], 4, 2, 64, 0)
    clean = c.run()
    over = c.run(over=(1,))
    assert (over[50:70] == 0).all() and torch.equal(over[:50], clean[:50]) and torch.equal(over[70:], clean[70:])
    bad = Case([50, 20, 33], [0, 3, 0], 4, 2, 64, 0, poison=21).run()
    assert torch.equal(bad[:21], clean[:21]) and not torch.isfinite(bad[21:50]).any() and torch.equal(bad[50:], clean[50:])
