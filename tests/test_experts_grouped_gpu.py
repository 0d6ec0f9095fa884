"""Experts over gathered rows (Ops::experts_grouped) in every form that it takes: bf16 in 16-byte pieces (one launch per product),
32-bit, sizes and weights off the 16 bytes, weights with a row stride of their own; with and without the counts; against 64-bit sums."""
import ctypes
import os
from ctypes import POINTER, byref, c_char_p, c_float, c_int, c_longlong

import pytest
import torch

from friday_inference_engine_b200 import build_plugin, native, ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    lib = ctypes.CDLL(build_plugin(os.path.join(HERE, "cpp", "experts_probe.cu"), str(tmp_path_factory.mktemp("experts") / "libexperts_probe.so")))
    T = POINTER(native.Tensor)
    lib.probe_error.restype = c_char_p
    lib.probe_experts_grouped.argtypes = [T, T, T, T, T, T, POINTER(c_int), c_int, c_int, c_int, c_int, c_float, c_float, T, POINTER(c_longlong)]
    return lib


def rnd(shape, seed, scale=1.0):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale


# (dtype, rows, experts, width, inner, what lies off the 16 bytes)
FORMS = [(torch.bfloat16, 300, 5, 64, 40, None), (torch.bfloat16, 70, 256, 16, 8, None), (torch.bfloat16, 300, 5, 64, 40, "stride"),
         (torch.bfloat16, 90, 3, 64, 40, "start"), (torch.bfloat16, 90, 4, 20, 24, None), (torch.bfloat16, 90, 4, 24, 12, None),
         (torch.float32, 130, 4, 36, 20, None), (torch.float32, 40, 3, 7, 5, None)]


@pytest.mark.parametrize("dtype,rows,experts,width,inner,off", FORMS)
@pytest.mark.parametrize("known", [False, True])
@pytest.mark.parametrize("act", [1, 3])
def test_every_form_of_grouped_experts(probe, dtype, rows, experts, width, inner, off, known, act):
    top, limit, slope = 2, 2.0, 1.702
    ids = torch.randint(-1, experts, (rows, top), generator=torch.Generator().manual_seed(1), dtype=torch.int32)
    h, weights, residual = rnd((rows, width), 2).to(dtype).to(DEV), torch.rand((rows, top), generator=torch.Generator().manual_seed(3)).to(DEV), rnd((rows, width), 4).to(DEV)

    def laid(n, k, seed):
        w = rnd((n, k), seed, k ** -0.5).to(dtype).to(DEV)
        if off == "stride":                        # rows further apart than they are long
            wide = torch.full((n, k + 24), 9.0, dtype=dtype, device=DEV)
            wide[:, :k] = w
            return wide[:, :k]
        if off == "start":
            flat = torch.zeros(n * k + 1, dtype=dtype, device=DEV)
            flat[1:] = w.flatten()
            return flat[1:].view(n, k)
        return w
    gu, down = laid(experts * 2 * inner, width, 5), laid(width, experts * inner, 6)
    out = torch.empty_like(residual)
    counts = (c_int * experts)(*[int((ids == e).sum()) for e in range(experts)])
    launches = c_longlong()
    dids = ids.to(DEV)
    rc = probe.probe_experts_grouped(ops._t(h), ops._t(dids), ops._t(weights), ops._t(gu), ops._t(down), ops._t(residual), counts if known else None, experts,
                                     top, inner, act, limit, slope, ops._t(out), byref(launches))
    assert rc == 0, probe.probe_error().decode()
    if dtype == torch.bfloat16 and off != "start" and width % 8 == 0 and inner % 8 == 0:
        assert launches.value == 5                 # the sort, the gather, a launch per product, the sum

    want, size = residual.double(), residual.double().abs()
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22
    for e in range(experts):
        rows_of, choice = (ids == e).nonzero(as_tuple=True)
        if not len(rows_of):
            continue
        z = h[rows_of.to(DEV)].double() @ gu[e * 2 * inner:(e + 1) * 2 * inner].double().T
        g, u = z[:, 0::2], z[:, 1::2]
        a = g * torch.sigmoid(g) * u if act == 1 else g.clamp(max=limit) * torch.sigmoid(slope * g.clamp(max=limit)) * (u.clamp(-limit, limit) + 1.0)
        d = down[:, e * inner:(e + 1) * inner].double().T
        share = weights.double()[rows_of.to(DEV), choice.to(DEV)][:, None]
        want.index_add_(0, rows_of.to(DEV), share * (a @ d))
        size.index_add_(0, rows_of.to(DEV), share * ((a.abs() + (g.abs() + 1.0) * (u.abs() + 1.0)) @ d.abs()))
    # the unit is rounded once to the rows' dtype (and its arguments to 32 bits), then 32-bit sums
    assert bool(((out.double() - want).abs() <= (2 * eps + (width + inner + 8) * 2.0 ** -23) * size + 1e-6).all())
