"""32-bit products on the tensor cores, every operand as three bf16 numbers: edges of tiles, splits of k, rows in portions, weights
with and without low bits, values that cannot be split."""
import pytest
import torch

from friday_inference_engine_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def product(x, w, bias=None, residual=None, scratch_bytes=38 << 20):
    fam = lib.family("gemm_simt")
    m, k, n = x.shape[0], x.shape[1], w.shape[0]
    out = residual.clone() if residual is not None else torch.full((m, n), float("nan"), device=DEV)
    scratch = torch.empty(scratch_bytes, dtype=torch.uint8, device=DEV)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    fam.call("gemm_simt_split", x.data_ptr(), w.data_ptr(), out.data_ptr(), bias.data_ptr() if bias is not None else None, 0,
             out.data_ptr() if residual is not None else None, m, n, k, x.stride(0), w.stride(0), n, 0, scratch.data_ptr(), scratch_bytes,
             status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert status[0] == 0
    return out


def check(out, x, w, extra=0.0):
    # an accumulator drops less than 2^-23 of the sum at each of its additions (sixteen in a part of k at most, all of them in its
    # small products, which are 2^-8 of the sum), adding a part or a split rounds by 2^-24, what the six products leave out is 2^-25
    k = x.shape[1]
    bound = (16 + 6 * k / 16 / 256 + k / 128 + 8) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    bound = bound + 2.0 ** -22 * (abs(extra) + 1e-30)
    ref = x.double() @ w.double().T + extra
    assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("m,n,k", [(9, 128, 32), (17, 130, 36), (16, 1, 4), (176, 257, 160), (177, 384, 2048), (352, 128, 1028), (40, 96, 18944),
                                   (353, 600, 3072), (1, 5000, 520)])
@pytest.mark.parametrize("weights", ["bf16", "fp32", "some"])
def test_split_product(m, n, k, weights):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    if weights != "fp32":
        w = w.bfloat16().float()
    if weights == "some":
        w[n // 2, k // 2] *= 1.001                             # one block of one quarter has low bits
    check(product(x, w), x, w)
    b, r = torch.randn(n, device=DEV, generator=g), torch.randn(m, n, device=DEV, generator=g)
    check(product(x, w, b, r), x, w, b.double() + r.double())


def test_rows_in_portions_and_padded_rows():
    g = torch.Generator(device=DEV).manual_seed(5)
    big, wide = torch.randn(500, 260, device=DEV, generator=g), torch.randn(200, 264, device=DEV, generator=g)
    x, w = big[:, :252], wide[:, 4:256]
    few = 180 * (6 * 256 + 4) + 16                             # scratch for 176 rows at a time
    got = product(x, w, scratch_bytes=few)
    check(got, x, w)
    assert torch.equal(got, torch.cat([product(x[a:a + 176], w) for a in (0, 176, 352)]))


@pytest.mark.parametrize("k", [64, 4096])
def test_values_that_cannot_be_split(k):
    g = torch.Generator(device=DEV).manual_seed(6)
    x, w = torch.randn(20, k, device=DEV, generator=g), torch.randn(150, k, device=DEV, generator=g)
    clean = product(x, w)
    x[3, 1], x[4, k - 1], x[5, 7], w[140, 5] = float("inf"), float("nan"), 3.4e38, float("-inf")
    got = product(x, w)
    rows, cols = [i for i in range(20) if i not in (3, 4, 5)], [i for i in range(150) if i != 140]
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])
    ref = x.double() @ w.double().T
    assert torch.equal(got[[3, 4]].isnan(), ref[[3, 4]].isnan()) and got[4].isnan().all()
    inf = ref[3].isinf()
    assert inf.any() and torch.equal(got[3].isinf(), inf) and torch.equal(got[3][inf].sign().double(), ref[3][inf].sign())
    assert torch.equal(got[rows][:, 140], ref[rows][:, 140].float())
    fits = ref[5][cols].abs() < 0.99 * torch.finfo(torch.float32).max
    assert fits.any() and ((got[5][cols][fits].double() - ref[5][cols][fits]).abs() <= 1e-4 * ref[5][cols][fits].abs() + 1e32).all()


# Values so small that three bf16 numbers do not hold their 24 bits: rows of x as a whole (and beside ordinary ones), and weight rows, bf16 numbers or
# not.  2^-21 of a row's norm is three times what k = 4,096 was measured at for ordinary values, and above what sums of 64 rounded terms come to
# (sqrt(64 / 2) 2^-24 / sqrt(3), a fifth more for adding 64 of them); without care it is 2^-13 here.
@pytest.mark.parametrize("m,n,k", [(20, 150, 64), (40, 130, 4096), (300, 128, 1028)])
@pytest.mark.parametrize("exponent", [-120, -100, -140])
def test_rows_of_very_small_values(m, n, k, exponent):
    g = torch.Generator(device=DEV).manual_seed(m)
    x, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)

    def small(rows):
        return torch.ldexp(rows.double(), torch.tensor(exponent, device=DEV)).float()

    def rows_close(out, a, b):
        ref = a.double() @ b.double().T
        assert ((out.double() - ref).norm(dim=1) <= 2.0 ** -21 * ref.norm(dim=1)).all()
    for some in (slice(None), slice(3, None, 2)):
        tiny = x.clone()
        tiny[some] = small(tiny[some])
        big = w * 2.0 ** 60                                      # (results well within the normal numbers)
        rows_close(product(tiny, big), tiny, big)
    for weights in (w, w.bfloat16().float()):
        tiny = weights.clone()
        tiny[1::3] = small(tiny[1::3])
        big = x * 2.0 ** 60
        rows_close(product(big, tiny).T, tiny, big)
    zero = x.clone()
    zero[2] = 0.0
    assert (product(zero, w)[2] == 0).all()


# What the products are split for: an error of the size of fp32 sums' at any k, measured at 1.2e-7 to 2.4e-7 of the norm.  Any one of the partial products
# that reach 2^-18 left out comes to 2.3e-6 and more with 32-bit weights (a lost lo plane of x with weights that are bf16 numbers 1.6e-6), whatever k is.
@pytest.mark.parametrize("m,n,k", [(40, 130, 32), (176, 257, 160), (177, 384, 2048), (352, 128, 1028), (40, 96, 18944), (353, 600, 3072), (20, 5000, 520)])
@pytest.mark.parametrize("weights", ["bf16", "fp32", "some"])
def test_split_product_keeps_its_bits(m, n, k, weights):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    full = w.clone()
    if weights != "fp32":
        w = w.bfloat16().float()
    if weights == "some":
        w[n // 2] = full[n // 2]                                 # one column of the result, whose rows of weights alone have low bits
    out, ref = product(x, w).double(), x.double() @ w.double().T
    assert (out - ref).norm() <= 8e-7 * ref.norm()
    assert (out - ref)[:, n // 2].norm() <= 8e-7 * ref[:, n // 2].norm()
