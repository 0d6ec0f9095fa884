"""The experts' products alone: the streamed form for few rows at the edges of its pieces and groups, against 64-bit sums."""
from ctypes import c_float, c_int, c_longlong, c_void_p

import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
P, I, F, L = c_void_p, c_int, c_float, c_longlong


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16().to(DEV)


def ptr(t):
    return None if t is None else t.data_ptr()


def stream():
    return torch.cuda.current_stream().cuda_stream


def silu(x):
    return x * torch.sigmoid(x)


# choices: spread over the experts, some of them none (-1); all rows one expert (a full group of 16 pairs); an expert that every
# row names twice (more pairs than a group)
@pytest.mark.parametrize("rows,top,experts,spread", [(1, 2, 8, "any"), (5, 3, 40, "any"), (8, 2, 8, "any"), (16, 4, 256, "any"), (13, 1, 3, "one"), (16, 2, 5, "one")])
@pytest.mark.parametrize("width,inner", [(8, 8), (520, 1032), (2048, 24), (1030 * 8, 520)])
def test_streamed_experts(rows, top, experts, spread, width, inner):
    r = lib.family("routed")
    r.declare("routed_gate_up", [P, P, P, P, I, I, I, I, I, I, F, F, I, P])
    r.declare("routed_down_combine", [P, P, P, P, I, P, P, I, I, I, I, I, I, P, I, P])
    r.declare("routed_down_scratch_floats", [I, I, I, I, I], L)
    if experts * width * inner > 1 << 27:
        experts = 8
    ids = torch.randint(-1, experts, (rows, top), generator=torch.Generator().manual_seed(1), dtype=torch.int32) if spread == "any" else torch.full((rows, top), experts - 1, dtype=torch.int32)
    ids = ids.to(DEV)
    h, gu, down = rnd((rows, width), 2), rnd((experts * 2 * inner, width), 3, width ** -0.5), rnd((width, experts * inner), 4, inner ** -0.5)
    act = torch.zeros((rows * top, inner), dtype=torch.bfloat16, device=DEV)
    r.call("routed_gate_up", ptr(h), ptr(ids), ptr(gu), ptr(act), rows, top, experts, width, inner, 1, 0.0, 1.0, 1, stream())
    want = torch.zeros((rows * top, inner), dtype=torch.float64, device=DEV)
    for pair, e in enumerate(ids.flatten().tolist()):
        if e >= 0:
            z = gu[e * 2 * inner:(e + 1) * 2 * inner].double() @ h[pair // top].double()
            want[pair] = silu(z[0::2]) * z[1::2]
    # rounded once to bf16 (2^-9 of the value); the sums' own rounding is far below
    assert bool(((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())

    weights, residual = torch.rand((rows, top), device=DEV), torch.randn((rows, width), device=DEV)
    floats = r.cdll.routed_down_scratch_floats(rows, top, width, inner, 1)
    assert floats == rows * top * width
    scratch, out = torch.empty(floats, device=DEV), torch.empty((rows, width), device=DEV)
    r.call("routed_down_combine", ptr(act), ptr(ids), ptr(weights), ptr(down), experts * inner, ptr(residual), ptr(out), 0, rows, top, experts, width,
           inner, ptr(scratch), 1, stream())
    total, size = residual.double(), residual.double().abs()
    for pair, e in enumerate(ids.flatten().tolist()):
        if e >= 0:
            w = down[:, e * inner:(e + 1) * inner].double()
            total[pair // top] += weights.flatten()[pair].double() * (w @ act[pair].double())
            size[pair // top] += weights.flatten()[pair].double() * (w.abs() @ act[pair].double().abs())
    assert bool(((out.double() - total).abs() <= (inner + 2 * top + 2) * 2.0 ** -24 * size).all())
