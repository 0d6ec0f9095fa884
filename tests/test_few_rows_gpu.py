"""The 32-bit product of few rows with the norm of its input, a gated unit, the rotation and the cache write, against 64-bit arithmetic."""
import ctypes
import math

import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
P, I, F = lib.P, lib.I, lib.F


class Fusion(ctypes.Structure):
    _fields_ = [("norm_w", P), ("norm_w_dtype", I), ("eps", F), ("act", I), ("act_limit", F), ("act_slope", F), ("row_seq", P), ("row_pos", P),
                ("denom", P), ("k_pool", P), ("v_pool", P), ("table", P), ("rot", I), ("nq", I), ("nkv", I), ("hd", I), ("table_width", I),
                ("page", I), ("fixed_weights", I)]


def call(x, w, out, f, bias=None, residual=None):
    fam = lib.family("gemm_simt")
    fam.declare("gemm_simt_few", [P, P, P, P, I, P, I, I, I, I, I, I, P, P])
    fam.call("gemm_simt_few", x.data_ptr(), w.data_ptr(), out.data_ptr(), bias.data_ptr() if bias is not None else None, 0,
             residual.data_ptr() if residual is not None else None, x.shape[0], w.shape[0], x.shape[1], x.stride(0), w.stride(0), out.stride(0),
             ctypes.byref(f), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return out


def inputs(m, n, k, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randn(s, device=DEV, generator=g) for s in ((m, k), (n, k), (n,), (k,))]


def normed(x, gain, eps):
    x = x.double()
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * gain.double()


def near(got, ref, scale):
    # k products and sums in fp32 (k / 2^24 of the sum of their magnitudes at most, far less where signs mix), a handful of roundings after
    assert (got.double() - ref).abs().max() <= 2.0 ** -18 * scale


@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (2, 7, 96), (3, 1000, 132), (4, 96, 256), (8, 2369, 128), (13, 33, 3584)])
@pytest.mark.parametrize("gain", [None, torch.float32, torch.bfloat16])
def test_norm_bias_and_residual(m, n, k, gain):
    x, w, b, g = inputs(m, n, k, m + n)
    f = Fusion(eps=1e-5)
    if gain is not None:
        g = g.to(gain)
        f.norm_w, f.norm_w_dtype = g.data_ptr(), 0 if gain == torch.float32 else 1
    h = normed(x, g, 1e-5) if gain is not None else x.double()
    r = torch.randn(m, n, device=DEV)
    ref = h @ w.double().T + b.double() + r.double()
    out = r.clone()
    near(call(x, w, out, f, b, out), ref, math.sqrt(k) * 4)


@pytest.mark.parametrize("act", [1, 2, 3])
@pytest.mark.parametrize("m,inner", [(1, 5), (4, 256), (7, 1200)])
def test_gated(act, m, inner):
    k = 96
    x, w, _, g = inputs(m, 2 * inner, k, act)
    w *= 0.3
    f = Fusion(norm_w=g.data_ptr(), eps=1e-6, act=act, act_limit=2.0, act_slope=1.7)
    z = normed(x, g, 1e-6) @ w.double().T
    a, u = z[:, 0::2], z[:, 1::2]
    if act == 1:
        ref = a * torch.sigmoid(a) * u
    elif act == 2:
        ref = torch.nn.functional.gelu(a, approximate="tanh") * u
    else:
        a, u = a.clamp(max=2.0), u.clamp(-2.0, 2.0)
        ref = a * torch.sigmoid(1.7 * a) * (u + 1.0)
    near(call(x, w, torch.empty(m, inner, device=DEV), f), ref, 4 * max(1.0, float(ref.abs().max())))


@pytest.mark.parametrize("nq,nkv,hd,rot", [(3, 1, 32, 32), (4, 2, 64, 16), (2, 2, 6, 0), (28, 4, 128, 128)])
@pytest.mark.parametrize("m", [1, 4, 9])
def test_rotary_and_cache(nq, nkv, hd, rot, m):
    k, n = 96, (nq + 2 * nkv) * hd
    x, w, b, g = inputs(m, n, k, nq + m)
    page, width, pages = 16, 5, 60
    denom = torch.tensor([10000.0], device=DEV) ** (2.0 * torch.arange(max(rot // 2, 1), device=DEV) / max(rot, 2))
    pos = torch.randint(0, page * width, (m,), dtype=torch.int32, device=DEV)
    seq = torch.arange(m, dtype=torch.int32, device=DEV)
    if m > 2:
        seq[1] = -1                                              # this one is over
    table = torch.randperm(pages, device=DEV)[:m * width].int().view(m, width).contiguous()
    kp, vp = (torch.full((pages, page, nkv, hd), 9.0, device=DEV) for _ in range(2))
    f = Fusion(norm_w=g.data_ptr(), eps=1e-5, row_seq=seq.data_ptr(), row_pos=pos.data_ptr(), denom=denom.data_ptr() if rot else None,
               k_pool=kp.data_ptr(), v_pool=vp.data_ptr(), table=table.data_ptr(), rot=rot, nq=nq, nkv=nkv, hd=hd, table_width=width, page=page)
    ref = (normed(x, g, 1e-5) @ w.double().T + b.double()).view(m, nq + 2 * nkv, hd)
    if rot:
        angle = (pos.float()[:, None] / denom[None]).double()[:, None]
        c, s, half = torch.cos(angle), torch.sin(angle), rot // 2
        turned = ref.clone()
        u, v = ref[:, :nq + nkv, :half], ref[:, :nq + nkv, half:rot]
        turned[:, :nq + nkv, :half], turned[:, :nq + nkv, half:rot] = u * c - v * s, v * c + u * s
        ref = torch.where((seq < 0)[:, None, None], ref, turned)
    got = call(x, w, torch.empty(m, n, device=DEV), f, b).view(m, nq + 2 * nkv, hd)
    near(got, ref, math.sqrt(k) * 8)
    want_k, want_v = (torch.full((pages, page, nkv, hd), 9.0, device=DEV) for _ in range(2))
    for i in range(m):
        if seq[i] >= 0:
            at = int(table[i, int(pos[i]) // page]), int(pos[i]) % page
            want_k[at], want_v[at] = got[i, nq:nq + nkv], got[i, nq + nkv:]
    assert torch.equal(kp, want_k) and torch.equal(vp, want_v)
