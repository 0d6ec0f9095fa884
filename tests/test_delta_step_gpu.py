"""One token of the gated delta rule in one kernel, against 64-bit arithmetic: what it returns and what it leaves in the state."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(g, *shape, scale=1.0):
    return torch.randn(shape, generator=g) * scale


def silu(x):
    return x * torch.sigmoid(x)


# heads on one query/key head alone, two, eight (a cluster each); matrices from one group of four columns to the largest that
# fit a thread's registers, threads without a column, no history, the longest one; a sequence that is over
@pytest.mark.parametrize("heads,groups,dk,dv,taps", [(1, 1, 4, 4, 1), (4, 2, 16, 24, 4), (8, 1, 40, 12, 8), (3, 3, 128, 128, 4), (16, 8, 128, 128, 4),
                                                     (2, 2, 256, 64, 2), (2, 1, 64, 256, 3), (5, 5, 10, 20, 5)])
@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_delta_step(heads, groups, dk, dv, taps, per_channel, dtype):
    d = lib.family("delta")
    P, I, F = lib.P, lib.I, lib.F
    L = lib.c_longlong
    d.declare("delta_step_supports", [I, I, I, I, I, L])
    d.declare("delta_step", [P, I, I, I, I, P, I, P, I, P, I, P, P, I, P, I, I, P, I, F, F, P, P, L, P, P, P, P] + [I] * 6 + [F, F, I, I, P])
    g = torch.Generator().manual_seed(heads * 1000 + dk + dv + per_channel)
    qk, hv = groups * dk, heads * dv
    channels, seqs = 2 * qk + hv, 5
    hist = (taps - 1) * channels
    stride = (hist + heads * dk * dv + 3) // 4 * 4
    assert d.cdll.delta_step_supports(heads, groups, dk, dv, taps, stride) == (hist % 4 == 0)
    if hist % 4:
        return
    proj = rnd(g, seqs, channels + hv).to(dtype)                            # q, k, v, gate
    w = rnd(g, channels, taps, scale=0.5).to(dtype)
    a_raw, b_raw = rnd(g, seqs, heads * dk if per_channel else heads), rnd(g, seqs, heads + 3)
    a_log, bias = rnd(g, heads, scale=0.3), rnd(g, heads * dk if per_channel else heads)
    norm = 1.0 + rnd(g, dv, scale=0.1)
    state = rnd(g, seqs + 2, stride)
    slots, order = [6, 0, 3, 2, 5], [2, 0, 1, 4, 3]                         # sequence -> slot, sequence -> row
    row_seq = torch.full((seqs,), -1, dtype=torch.int32)
    for s_, r_ in enumerate(order):
        row_seq[r_] = s_
    row_seq[order[3]] = -1                                                  # this one is over
    c = [t.to(DEV).contiguous() for t in (proj, w, a_raw, b_raw, a_log, bias, norm, state, row_seq)]
    start, ones, where = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in (order, [1] * seqs, slots))
    y = torch.full((seqs, hv), 9.0, dtype=dtype, device=DEV)
    code = 0 if dtype == torch.float32 else 1
    scale, eps = dk ** -0.5, 1e-5
    d.call("delta_step", c[0].data_ptr(), channels + hv, 0, qk, 2 * qk, c[1].data_ptr(), code, c[2].data_ptr(), a_raw.shape[1], c[3].data_ptr(),
           heads + 3, c[4].data_ptr(), c[5].data_ptr(), 0, c[0].data_ptr() + channels * c[0].element_size(), channels + hv, 1 if per_channel else 0,
           c[6].data_ptr(), 0, eps, 0.5, y.data_ptr(), c[7].data_ptr(), stride, c[8].data_ptr(), start.data_ptr(), ones.data_ptr(), where.data_ptr(),
           seqs, heads, groups, dk, dv, taps, scale, 1e-6, 1 if per_channel else 0, code, torch.cuda.current_stream().cuda_stream)
    got_y, got = y.cpu().double(), c[7].cpu().double()
    want = state.double().clone()
    for s_ in (0, 1, 2, 4):
        row, slot = order[s_], slots[s_]
        past, x = want[slot, :hist].reshape(taps - 1, channels).clone(), proj[row].double()
        window = torch.cat([past, x[None, :channels]])
        z = silu((window * w.double().T).sum(0))
        want[slot, :hist] = window[1:].reshape(-1)
        q, k, v = z[:qk].reshape(groups, dk), z[qk:2 * qk].reshape(groups, dk), z[2 * qk:].reshape(heads, dv)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * scale
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        q, k = q.repeat_interleave(heads // groups, 0), k.repeat_interleave(heads // groups, 0)
        decay = torch.exp(-torch.exp(a_log.double()).reshape(heads, 1) * torch.nn.functional.softplus((a_raw[row].double() + bias.double()).reshape(heads, -1)))
        S = want[slot, hist:hist + heads * dk * dv].reshape(heads, dk, dv) * decay[:, :, None]
        u = torch.sigmoid(b_raw[row, :heads].double())[:, None] * (v - torch.einsum("hkv,hk->hv", S, k))
        S = S + k[:, :, None] * u[:, None, :]
        want[slot, hist:hist + heads * dk * dv] = S.reshape(-1)
        o = torch.einsum("hkv,hk->hv", S, q)
        gate = x[channels:].reshape(heads, dv)
        act = torch.sigmoid(gate) if per_channel else silu(gate)
        ref = o * 0.5 / torch.sqrt((o * o).mean(-1, keepdim=True) + eps) * norm.double() * act
        # sums of dk numbers of size 1 in 32 bits, a norm that may divide by a small root mean square
        slack = (dk + taps + 30) * 2.0 ** -22 * (1.0 + (S.abs().amax() * 0.5 / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)))
        err = (got_y[row].reshape(heads, dv) - ref).abs()
        assert bool((err <= slack * (1.0 + act.abs()) + (2.0 ** -8 if code else 0.0) * ref.abs()).all())
    assert bool((got_y[order[3]] == 9.0).all())
    assert bool(((got - want).abs() <= (dk + taps + 30) * 2.0 ** -22 * (1.0 + want.abs().amax())).all())
    untouched = [i for i in range(seqs + 2) if i not in slots] + [slots[3]]
    assert torch.equal(got[untouched], state.double()[untouched])
