"""The experts' products alone: the streamed form for few rows and the grouped form for many, at the edges of their pieces,
tiles and groups, against 64-bit sums."""
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


# groups: none, one row, around 256 rows, several tiles, rows beyond the last group; columns and k around the tiles; matrices
# side by side (the next one's numbers lie where this one's k ends) and one after another
@pytest.mark.parametrize("sizes", [[0, 1, 256, 257, 0], [700], [3] * 40, [255, 512, 0, 130]])
@pytest.mark.parametrize("n,k,act", [(16, 8, 0), (272, 72, 0), (4096, 200, 1), (520, 64, 3)])
@pytest.mark.parametrize("side_by_side", [False, True])
def test_grouped_product(sizes, n, k, act, side_by_side):
    g = lib.family("gemm_tc")
    g.declare("gemm_tc_grouped", [P, L, P, L, P, I, P, I, I, I, I, I, I, I, I, I, F, F, P, I, P])
    groups, used = len(sizes), sum(sizes)
    rows = used + 5
    x = rnd((rows, k), 7)
    if side_by_side:
        w = rnd((n, groups * k), 8, 0.3)
        parts, ldw, step = [w[:, e * k:(e + 1) * k] for e in range(groups)], groups * k, k
    else:
        w = rnd((groups * n, k), 8, 0.3)
        parts, ldw, step = [w[e * n:(e + 1) * n] for e in range(groups)], k, n * k
    offsets = torch.tensor([sum(sizes[:e]) for e in range(groups + 1)], dtype=torch.int32, device=DEV)
    out = torch.full((rows, n // 2 if act else n), 7.0, dtype=torch.bfloat16 if act else torch.float32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if side_by_side and not act:
        parts[0].fill_(float("nan"))           # reaches no other group's sums
    g.call("gemm_tc_grouped", ptr(x), 0, ptr(w), step, ptr(out), 1 if act else 0, ptr(offsets), groups, rows, n, k, k, ldw, out.shape[1],
           sum((s + 255) // 256 for s in sizes), act, 2.0, 1.702, ptr(status), sms, stream())
    assert int(status) == 0
    assert bool((out[used:] == 7.0).all())
    at = 0
    for e, size in enumerate(sizes):
        a, b = x[at:at + size].double(), parts[e].double()
        got, z, mag = out[at:at + size].double(), a @ b.T, a.abs() @ b.abs().T
        at += size
        if side_by_side and not act and e == 0:
            assert bool(torch.isnan(got).all())
        elif act:
            gate, up = z[:, 0::2], z[:, 1::2]
            want = silu(gate) * up if act == 1 else gate.clamp(max=2.0) * torch.sigmoid(1.702 * gate.clamp(max=2.0)) * (up.clamp(-2.0, 2.0) + 1.0)
            # bf16's rounding, and the sums' errors (k 2^-23 of the terms' size) times what the unit makes of them
            slack = k * 2.0 ** -23 * (mag[:, 0::2] * (up.abs() + 1.0) * 2.0 + mag[:, 1::2] * (gate.abs() + 1.0))
            assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + slack + 1e-6).all())
        else:
            assert bool(((got - z).abs() <= k * 2.0 ** -23 * mag).all())


# groups of equal size whose rows lie side by side (heads), no offsets: rows and columns around the tiles, k around the blocks
@pytest.mark.parametrize("groups,size,n,k", [(1, 1, 8, 8), (3, 40, 520, 192), (16, 257, 264, 24), (5, 600, 128, 72)])
def test_grouped_product_of_planes(groups, size, n, k):
    g = lib.family("gemm_tc")
    g.declare("gemm_tc_grouped", [P, L, P, L, P, I, P, I, I, I, I, I, I, I, I, I, F, F, P, I, P])
    x, w = rnd((size, groups * k + 8), 9), rnd((n, groups * k), 10, 0.3)
    out = torch.empty((groups * size, n), device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g.call("gemm_tc_grouped", ptr(x), k, ptr(w), k, ptr(out), 0, None, groups, groups * size, n, k, groups * k + 8, groups * k, n,
           groups * ((size + 255) // 256), 0, 0.0, 0.0, ptr(status), sms, stream())
    assert int(status) == 0
    for e in range(groups):
        a, b = x[:, e * k:(e + 1) * k].double(), w[:, e * k:(e + 1) * k].double()
        assert bool(((out[e * size:(e + 1) * size].double() - a @ b.T).abs() <= k * 2.0 ** -23 * (a.abs() @ b.abs().T)).all())


# The down product's sums are fp32 multiply-adds that round: a lane adds k / 64 terms in each of two sums, whose partial sums grow like
# the square root of their number, each addition off by 2^-24 / sqrt(3) (root mean square) of the sum so far at most; over all sums that is
# 2^-24 / sqrt(3) * sqrt(k / 128) of the result's norm.  (An accumulator that drops bits is two to five times as far off.)
@pytest.mark.parametrize("rows,top", [(1, 8), (8, 2), (16, 3)])
@pytest.mark.parametrize("inner", [1024, 2048, 4096])
def test_streamed_experts_sums_round(rows, top, inner):
    r = lib.family("routed")
    r.declare("routed_down_combine", [P, P, P, P, I, P, P, I, I, I, I, I, I, P, I, P])
    width, experts = 512, 8
    ids = torch.stack([torch.randperm(experts, generator=torch.Generator().manual_seed(i))[:top] for i in range(rows)]).int().to(DEV)
    act, down = rnd((rows * top, inner), 5), rnd((width, experts * inner), 6)
    weights, scratch, out = torch.ones((rows, top), device=DEV), torch.empty(rows * top * width, device=DEV), torch.empty((rows, width), device=DEV)
    r.call("routed_down_combine", ptr(act), ptr(ids), ptr(weights), ptr(down), experts * inner, None, ptr(out), 0, rows, top, experts, width, inner,
           ptr(scratch), 1, stream())
    want = torch.stack([down[:, e * inner:(e + 1) * inner].double() @ act[pair].double() for pair, e in enumerate(ids.flatten().tolist())])
    error = (scratch.view(rows * top, width).double() - want).norm() / want.norm()
    assert float(error) <= 2.0 ** -24 / 3 ** 0.5 * (inner / 128) ** 0.5
