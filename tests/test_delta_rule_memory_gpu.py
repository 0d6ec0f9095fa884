"""What the delta rule's prompts take of the working memory beside their result."""
import ctypes
import os

import pytest

from friday_inference_engine_b200 import build_plugin

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    return ctypes.CDLL(build_plugin(os.path.join(HERE, "cpp", "delta_memory_probe.cu"), str(tmp_path_factory.mktemp("probe") / "libdelta_memory_probe.so"))).probe_delta_scan


def scan(probe, rows, heads, dv):
    held, launches = ctypes.c_longlong(), ctypes.c_longlong()
    assert probe(rows, heads, dv, ctypes.byref(held), ctypes.byref(launches)) == 0
    return held.value, launches.value


@pytest.mark.parametrize("rows,heads,dv", [(600, 4, 128), (1000, 64, 64)])
def test_chunks_are_not_the_arenas(probe, rows, heads, dv):
    # (64 heads go in two rounds of two kernels)  The arena holds the result, of which every layer's arena keeps one, and at most as much again from growing in blocks
    held, launches = scan(probe, rows, heads, dv)
    assert launches == (2 if heads == 4 else 4) and held <= 2 * 4 * rows * heads * dv + (1 << 20)


def test_a_head_that_does_not_fit_goes_token_by_token(probe):
    assert scan(probe, 60000, 1, 64)[1] == 1
