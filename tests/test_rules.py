"""Which kernel a call goes to, asked of the built libraries on the host: on both sides of each line, at sizes that were timed."""
import pytest

from friday_inference_engine_b200.ops import lib

SCRATCH = lib.c_longlong(2 * 148 * 128 * 256 * 4)          # what Ops gives a product


def ask(family, name, *args):
    try:
        fam = lib.family(family)
    except Exception as e:           # no compiler, or no CUDA runtime library to load against
        pytest.skip("the %s library is not available here: %s" % (family, e))
    fn = getattr(fam.cdll, name)
    fn.argtypes = [lib.P if a is None else type(a) if isinstance(a, lib.c_longlong) else lib.I for a in args]
    return fn(*args)


# (lengths, heads, dk, dv), a decay per head, a decay per channel: whether chunks of sixteen tokens were the faster way
@pytest.mark.parametrize("lens,heads,dk,dv,per_head,per_channel", [
    ([2048], 16, 128, 128, 1, 1), ([256], 4, 128, 128, 1, 1), ([64], 16, 128, 128, 0, 1), ([32], 16, 128, 128, 0, 1), ([31], 16, 128, 128, 0, 0),
    ([64, 512, 300, 128, 400, 90, 230, 480], 16, 128, 128, 1, 1), ([64, 512, 300, 128, 400, 90, 230, 480], 32, 128, 128, 1, 1),
    ([300] * 16, 32, 128, 128, 0, 1), ([300] * 16, 4, 128, 128, 1, 1), ([33] * 64, 16, 128, 128, 0, 1), ([128] + [1] * 63, 16, 128, 128, 0, 1),
    ([512] + [17] * 31, 16, 128, 128, 1, 1), ([2048], 16, 64, 64, 0, 0), ([2048], 16, 16, 128, 0, 0), ([300] * 8, 16, 128, 16, 0, 0),
    ([1000] * 4, 16, 128, 64, 0, 1), ([96] + [33] * 20, 32, 128, 128, 0, 1),
])
def test_delta_rule_in_chunks(lens, heads, dk, dv, per_head, per_channel):
    for flag, want in ((0, per_head), (1, per_channel)):
        assert ask("delta", "delta_scan_chunks_pays", sum(lens), len(lens), max(lens), heads, dk, dv, flag) == want


# two kernels per round of heads (50 heads' chunks fit at a time), per portion of rows (341 rows of 18,944 fit, and go 176 at a time then)
def test_launches_of_calls_that_go_in_parts():
    assert [ask("delta", "delta_scan_chunks_launches", 1000, 3, heads, 64) for heads in (1, 50, 51, 101)] == [2, 2, 4, 6]
    assert ask("delta", "delta_scan_chunks_launches", 100000, 1, 4, 64) == 0
    assert [ask("gemm_simt", "gemm_simt_split_launches", m, 18944, SCRATCH) for m in (17, 341, 342, 600)] == [2, 2, 4, 8]


# end: 0 a product alone, 1 a gated unit, 2 rotary columns; with the norm of the input unless said otherwise
@pytest.mark.parametrize("m,n,k,end,norm,want", [
    (1, 152064, 896, 0, 1, 1), (1, 37888, 3584, 1, 0, 1), (2, 4608, 3584, 2, 1, 1), (2, 8192, 1024, 0, 1, 1), (2, 9728, 896, 0, 1, 0), (2, 152064, 896, 1, 1, 0),
    (2, 1024, 4096, 0, 1, 0), (2, 2048, 4096, 2, 1, 1), (3, 1000, 96, 0, 1, 1), (4, 512, 256, 0, 1, 0), (4, 4864, 896, 1, 1, 1), (4, 2048, 2048, 1, 1, 0),
    (4, 37888, 3584, 1, 1, 0), (4, 6144, 2048, 2, 1, 1), (4, 8192, 1024, 2, 1, 0), (5, 512, 96, 1, 1, 1), (16, 160, 96, 2, 1, 1), (5, 512, 96, 0, 1, 0),
    (5, 512, 96, 1, 0, 0), (8, 4608, 3584, 2, 1, 0), (16, 3584, 18944, 1, 1, 0),
])
def test_few_rows_with_their_neighbours(m, n, k, end, norm, want):
    assert ask("gemm_simt", "gemm_simt_few_pays", m, n, k, end, norm) == want


def splits_of(rows, heads, keys):          # of the keys where a warp has a row and head
    return max(1, min(148 * 16 // (rows * heads), (keys + 63) // 64, 64)) if rows * heads < 148 * 16 and keys > 128 else 1


# new tokens, keys before them, heads, kv heads, their size, window: whether the tiles were the faster way
@pytest.mark.parametrize("lens,before,nq,nkv,hd,window,want", [
    ([16], 0, 28, 4, 128, 0, 0), ([16], 8000, 28, 4, 128, 0, 0), ([20], 300, 28, 4, 128, 0, 0), ([48], 1000, 28, 4, 128, 0, 1), ([333], 0, 28, 4, 128, 0, 1),
    ([333], 8000, 28, 4, 128, 0, 1), ([64], 8000, 8, 8, 128, 0, 0), ([200], 8000, 8, 8, 128, 0, 1), ([100], 8000, 3, 1, 32, 0, 0), ([333], 8000, 3, 1, 32, 0, 1),
    ([16] * 8, 1000, 28, 4, 128, 0, 1), ([16] + [1] * 31, 500, 16, 16, 64, 0, 0), ([300, 33], 0, 28, 4, 128, 0, 1), ([16], 4000, 28, 4, 128, 512, 0),
    ([300], 4000, 28, 4, 128, 512, 1), ([1] * 64 + [100], 2000, 16, 16, 64, 0, 0), ([256] * 8, 0, 3, 1, 32, 0, 1), ([64] * 16, 2000, 64, 1, 128, 0, 1), ([15] * 64, 2000, 28, 4, 128, 0, 0),
    ([16] * 64, 2000, 28, 4, 128, 0, 1),
])
def test_fp32_attention_of_prompts(lens, before, nq, nkv, hd, window, want):
    keys = max(lens) + before
    assert ask("attention_simt", "attention_simt_prompt_pays", sum(lens), len(lens), max(lens), keys, nq, nkv, hd, window, splits_of(sum(lens), nq, keys)) == want


@pytest.mark.parametrize("m,n,k,want", [
    (333, 37888, 3584, 1), (333, 3584, 18944, 1), (353, 3584, 18944, 1), (17, 3584, 3584, 1), (16, 3584, 3584, 0), (48, 2048, 1024, 1), (47, 2048, 1024, 0), (65, 1024, 1024, 1),
    (64, 1024, 1024, 0), (96, 640, 2048, 0), (128, 640, 2048, 1), (1024, 512, 1024, 0), (96, 200000, 64, 0), (128, 128, 18944, 0), (1024, 128, 18944, 0), (96, 300, 4096, 0),
    (333, 300, 4096, 1), (520, 256, 18944, 0), (48, 512, 8192, 1),
])
def test_32_bit_products_on_the_tensor_cores(m, n, k, want):
    assert ask("gemm_simt", "gemm_simt_split_pays", None, None, m, n, k, k, k, SCRATCH) == want


@pytest.mark.parametrize("rows,qk_heads,dk,values,want", [
    (64, 8, 128, 2048, 0), (256, 8, 128, 2048, 0), (512, 8, 128, 2048, 1), (2304, 8, 128, 2048, 1), (512, 4, 128, 1024, 0), (1024, 4, 128, 1024, 1),
    (256, 16, 128, 4096, 1), (100, 32, 128, 8192, 0), (2304, 1, 128, 128, 0), (1024, 8, 64, 1024, 0), (2048, 8, 64, 1024, 1), (2304, 2, 32, 128, 0),
])
def test_convolutions_sixteen_rows_per_warp(rows, qk_heads, dk, values, want):
    assert ask("delta", "delta_conv_runs_pay", rows, qk_heads, dk, values) == want
