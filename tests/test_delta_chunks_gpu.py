"""The delta rule of prompts in chunks of sixteen tokens, against 64-bit arithmetic token by token: edges of chunks, head sizes that fill a
tile or not, shared keys, both kinds of decays, sequences that are over, values that are not finite."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
P, I, L = lib.P, lib.I, lib.c_longlong
SIGNATURE = [P, P, I, P, I, I, P, P, I, P, P, L, L, P, P, P, P, I, I, I, I, I, I, P]


def inputs(lens, heads, groups, dk, dv, per_channel, dtype, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)

    def rnd(*shape):
        return torch.randn(shape, device=DEV, generator=g)
    rows = sum(lens)
    qkv = rnd(rows, 2 * groups * dk + heads * dv)
    q, k = (qkv[:, i * groups * dk:(i + 1) * groups * dk].view(rows, groups, dk) for i in (0, 1))
    q /= q.norm(dim=-1, keepdim=True) * dk ** 0.5
    k += 0.7 * rnd(1, groups, dk)                                # keys that have much in common
    k /= k.norm(dim=-1, keepdim=True)
    n = heads * dk if per_channel else heads
    return {"lens": lens, "sizes": (heads, groups, dk, dv, per_channel), "qkv": qkv, "a": rnd(rows, n + 2).to(dtype), "b": rnd(rows, heads + 1).to(dtype),
            "a_log": rnd(heads) - 1.0, "bias": rnd(n), "state": rnd(len(lens) + 1, 5 + heads * dk * dv + 3)}


def run(name, c, over=()):
    fam = lib.family("delta")
    chunks = name == "delta_scan_chunks"
    fam.declare(name, SIGNATURE[:-1] + [I, I, P, L, P] if chunks else SIGNATURE)
    heads, groups, dk, dv, per_channel = c["sizes"]
    n, rows = len(c["lens"]), sum(c["lens"])
    starts = [sum(c["lens"][:i]) for i in range(n)]
    start, count, slots = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in (starts, c["lens"], range(n, 0, -1)))
    row_seq = torch.tensor([-1 if i in over else i for i, m in enumerate(c["lens"]) for _ in range(m)], dtype=torch.int32, device=DEV)
    out, state = torch.full((rows, heads * dv), 7.0, device=DEV), c["state"].clone()
    more = []
    if chunks:
        need = fam.declare("delta_scan_chunks_scratch", [P, I, I, I, I, I], L)(c["qkv"].data_ptr(), rows, n, heads, dk, dv)
        scratch = torch.full((need,), 255, dtype=torch.uint8, device=DEV)
        more = [rows, max(c["lens"]), scratch.data_ptr(), need]
    fam.call(name, c["qkv"].data_ptr(), c["a"].data_ptr(), c["a"].stride(0), c["b"].data_ptr(), c["b"].stride(0), 0 if c["a"].dtype == torch.float32 else 1,
             c["a_log"].data_ptr(), c["bias"].data_ptr(), 0, out.data_ptr(), state.data_ptr(), state.stride(0), 5, row_seq.data_ptr(), start.data_ptr(),
             count.data_ptr(), slots.data_ptr(), n, heads, groups, dk, dv, 1 if per_channel else 0, *more,
             torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return out, state


def exact(c):
    heads, groups, dk, dv, per_channel = c["sizes"]
    rate, outs, state, r0 = c["a_log"].double().exp(), [], c["state"].double(), 0
    for i, m in enumerate(c["lens"]):
        S = state[len(c["lens"]) - i, 5:5 + heads * dk * dv].view(heads, dk, dv).clone()
        x = c["qkv"][r0:r0 + m].double()
        q, k = (x[:, j * groups * dk:(j + 1) * groups * dk].view(m, groups, dk).repeat_interleave(heads // groups, 1) for j in (0, 1))
        v = x[:, 2 * groups * dk:].view(m, heads, dv)
        z = torch.nn.functional.softplus(c["a"][r0:r0 + m, :-2].double() + c["bias"].double(), threshold=1e9)
        z = z.view(m, heads, dk) if per_channel else z[:, :, None].expand(m, heads, dk)
        decay, beta = torch.exp(-rate[None, :, None] * z), torch.sigmoid(c["b"][r0:r0 + m, :heads].double())
        for t in range(m):
            S = S * decay[t][:, :, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None]
            outs.append(torch.einsum("hkv,hk->hv", S, q[t]).reshape(-1))
        state[len(c["lens"]) - i, 5:5 + heads * dk * dv] = S.reshape(-1)
        r0 += m
    return torch.stack(outs), state


@pytest.mark.parametrize("lens,heads,groups,dk,dv", [([16], 1, 1, 128, 64), ([1, 37, 100, 17], 4, 2, 128, 128), ([65, 3, 32], 3, 3, 20, 24),
                                                     ([200], 2, 1, 64, 132), ([33, 15], 2, 2, 4, 4),
                                                     ([20, 50, 20, 50, 1, 90], 26, 13, 16, 8), ([1] * 62 + [17, 3], 4, 1, 8, 4)])
@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_delta_chunks(lens, heads, groups, dk, dv, per_channel, dtype):
    c = inputs(lens, heads, groups, dk, dv, per_channel, dtype)
    out, state = run("delta_scan_chunks", c)
    ref, ref_state = exact(c)
    # sums of up to 200 tokens and 128 channels in fp32: each addition rounds by 2^-24 of values that stay within a few times the
    # largest; 2^-17 is 128 of them, all in one direction
    assert (out.double() - ref).abs().max() <= 2.0 ** -17 * ref.abs().max()
    assert (state.double() - ref_state).abs().max() <= 2.0 ** -17 * ref_state.abs().max()


def test_sequence_that_is_over_and_values_that_are_not_finite():
    c = inputs([40, 20, 33], 2, 1, 128, 128, False, torch.float32)
    out, state = run("delta_scan_chunks", c, over=(1,))
    assert (out[40:60] == 7.0).all() and torch.equal(state[2], c["state"][2])
    c["qkv"][21, 256:] = float("inf")
    bad, _ = run("delta_scan_chunks", c, over=(1,))
    scan, _ = run("delta_scan", c, over=(1,))
    assert torch.isfinite(bad[:21]).all() and torch.equal(torch.isfinite(bad).all(1), torch.isfinite(scan).all(1))
    assert (bad[:21] - out[:21]).abs().max() <= 2.0 ** -17 * out.abs().max() and torch.equal(bad[60:], out[60:])


# An error that is no larger than that of the walk token by token, which rounds every addition: the same inputs through both, against 64 bits.
# The mean of three seeds; a fiftieth for what seeds leave open (measured: outputs 0.69 to 0.97 of it, states 0.91 to 1.00).  Keys that are nearly
# parallel (`common`): U0 and W S0 round by themselves and are larger than their difference, the corrections; half of 2^-24 more of each, beside
# the 2^-24 of the state's own sums, is a tenth in a root of squares (measured: states 1.02).
@pytest.mark.parametrize("rate,common", [(-2.0, 0.0), (0.0, 0.0), (1.0, 0.0), (2.0, 0.0), (1.0, 1.0)])
@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64)])
@pytest.mark.parametrize("per_channel", [False, True])
def test_errors_are_those_of_rounded_sums(rate, common, dk, dv, per_channel):
    errors = {"delta_scan": [0.0, 0.0], "delta_scan_chunks": [0.0, 0.0]}
    for seed in range(3):
        c = inputs([400, 77, 33], 8, 4, dk, dv, per_channel, torch.bfloat16, seed)
        c["a_log"] += rate
        k = c["qkv"][:, 4 * dk:8 * dk].view(-1, 4, dk)
        k += common * torch.randn(1, 4, dk, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))
        k /= k.norm(dim=-1, keepdim=True)
        c["state"] *= 0.1
        ref, ref_state = exact(c)
        for name, total in errors.items():
            out, state = run(name, c)
            for i, (got, want) in enumerate([(out, ref), (state, ref_state)]):
                total[i] += float((got.double() - want).norm() / want.norm())
    for i in (0, 1):
        assert errors["delta_scan_chunks"][i] <= (1.1 if common else 1.02) * errors["delta_scan"][i]
        assert errors["delta_scan_chunks"][i] / 3 <= 1e-6             # losing a third bf16 number of any operand is 1.5e-6 and more


# more heads than the scratch holds at a time: two rounds of 34 and 33, whose chunks lie at other places of it
@pytest.mark.parametrize("per_channel", [False, True])
def test_heads_in_uneven_rounds(per_channel):
    c = inputs([700, 33, 267], 67, 1, 8, 4, per_channel, torch.float32)
    need = lib.family("delta").declare("delta_scan_chunks_scratch", [P, I, I, I, I, I], L)(c["qkv"].data_ptr(), 1000, 3, 67, 8, 4)
    one = lib.family("delta").declare("delta_scan_chunks_scratch", [P, I, I, I, I, I], L)(c["qkv"].data_ptr(), 1000, 3, 1, 8, 4)
    assert need == 34 * one
    out, state = run("delta_scan_chunks", c)
    ref, ref_state = exact(c)
    assert (out.double() - ref).norm() <= 1e-6 * ref.norm() and (state.double() - ref_state).norm() <= 1e-6 * ref_state.norm()
