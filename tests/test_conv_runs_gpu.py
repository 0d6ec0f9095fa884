"""Prompts' short convolution with unit heads, several rows per warp, and the heads' gated norm in pieces of four: against 64-bit arithmetic."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
P, I, F, L = lib.P, lib.I, lib.F, lib.c_longlong


def ulp(dtype):
    return 2.0 ** -18 if dtype == torch.float32 else 2.0 ** -8


# runs of 16 rows that end inside sequences, sequences shorter than the taps, one that is over, heads of fewer than 128 channels, a value
# segment that is not whole
@pytest.mark.parametrize("lens", [[64], [1, 2, 70, 3, 17, 16], [33, 40]])
@pytest.mark.parametrize("groups,dk,values,taps", [(1, 128, 128, 4), (2, 20, 132, 3), (3, 64, 4, 2), (1, 4, 256, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_conv(lens, groups, dk, values, taps, dtype):
    fam = lib.family("delta")
    fam.declare("delta_conv_prepare", [P, I, I, I, I, P, I, P, P, L, P, P, P, I, I, I, I, I, F, F, I, I, P])
    g = torch.Generator(device=DEV).manual_seed(dk + taps)
    rows, channels, n = sum(lens), 2 * groups * dk + values, len(lens)
    x = torch.randn(rows, channels + 8, device=DEV, generator=g).to(dtype)
    w = torch.randn(channels, taps, device=DEV, generator=g).to(dtype)
    state = torch.randn(n + 1, (taps - 1) * channels + 5, device=DEV, generator=g)
    start = [sum(lens[:i]) for i in range(n)]
    over = n - 1 if n > 1 else -1
    t = [torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([-1 if i == over else i for i, m in enumerate(lens) for _ in range(m)], start, range(n, 0, -1))]
    out = torch.full((rows, channels), 7.0, device=DEV)
    qk = groups * dk
    fam.call("delta_conv_prepare", x.data_ptr(), x.stride(0), 4, 4 + qk, 4 + 2 * qk, w.data_ptr(), 0 if dtype == torch.float32 else 1, out.data_ptr(),
             state.data_ptr(), state.stride(0), t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), rows, groups, dk, values, taps, 0.25, 1e-6, 0,
             0 if dtype == torch.float32 else 1, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for i, m in enumerate(lens):
        got = out[start[i]:start[i] + m]
        if i == over:
            assert (got == 7.0).all()
            continue
        before = state[n - i, :(taps - 1) * channels].view(taps - 1, channels).double()
        full = torch.cat([before, x[start[i]:start[i] + m, 4:4 + channels].double()])
        y = sum(full[j:j + m] * w[:, j].double() for j in range(taps))
        y = y * torch.sigmoid(y)
        heads = y[:, :2 * qk].view(m, 2 * groups, dk)
        heads = heads / torch.sqrt((heads * heads).sum(-1, keepdim=True) + 1e-6)
        heads[:, :groups] *= 0.25
        ref = torch.cat([heads.reshape(m, -1), y[:, 2 * qk:]], dim=1)
        assert (got.double() - ref).abs().max() <= 2.0 ** -18 * max(1.0, float(ref.abs().max()))


# as many inputs as make the runs the faster way
@pytest.mark.parametrize("lens,groups,dk,values,taps", [([1, 2, 300, 3, 17, 200], 8, 128, 2052, 4), ([5500], 16, 20, 132, 3), ([3000, 1, 2, 8000], 3, 64, 4, 2),
                                                        ([16000, 33], 1, 4, 256, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_conv_in_runs(lens, groups, dk, values, taps, dtype):
    assert lib.family("delta").declare("delta_conv_runs_pay", [I, I, I, I])(sum(lens), groups, dk, values) == 1
    test_conv(lens, groups, dk, values, taps, dtype)


@pytest.mark.parametrize("rows,heads,dv", [(1, 1, 4), (5, 3, 64), (33, 16, 128), (7, 2, 100)])
@pytest.mark.parametrize("act,per_head", [(0, 0), (1, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_head_norm_gate(rows, heads, dv, act, per_head, dtype):
    fam = lib.family("recurrence")
    fam.declare("recurrence_head_norm_gate", [P, P, I, P, P, I, I, P, I, I, I, F, F, I, I, P])
    g = torch.Generator(device=DEV).manual_seed(rows + dv)
    o, z = torch.randn(rows, heads, dv, device=DEV, generator=g), torch.randn(rows, heads * dv + 4, device=DEV, generator=g).to(dtype)
    w = torch.randn(heads if per_head else 1, dv, device=DEV, generator=g)
    seq = torch.arange(rows, dtype=torch.int32, device=DEV)
    if rows > 1:
        seq[1] = -1
    out = torch.full((rows, heads * dv), 7.0, dtype=dtype, device=DEV)
    fam.call("recurrence_head_norm_gate", o.data_ptr(), z.data_ptr() + 4 * z.element_size(), z.stride(0), out.data_ptr(), w.data_ptr(), 0, per_head, seq.data_ptr(),
             rows, heads, dv, 1e-5, 0.5, act, 0 if dtype == torch.float32 else 1, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    a = z[:, 4:].double().view(rows, heads, dv)
    a = torch.sigmoid(a) if act else a * torch.sigmoid(a)
    x = o.double()
    ref = (0.5 * x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double() * a).view(rows, -1)
    live = seq >= 0
    assert (out[~live] == 7.0).all()
    assert ((out.double() - ref).abs() <= ulp(dtype) * ref.abs() + 2.0 ** -18)[live].all()
