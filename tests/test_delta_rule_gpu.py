"""When the delta rule's one-token kernel is taken: it reads the recurrent state while the kernel before still runs, which is only
sound for the program entry that writes the state's cache entry."""
import ctypes
import os

import pytest

from friday_inference_engine_b200 import build_plugin

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_only_the_entry_that_writes_the_state(tmp_path):
    ok = ctypes.CDLL(build_plugin(os.path.join(HERE, "cpp", "delta_probe.cu"), str(tmp_path / "libdelta_probe.so"))).probe_delta_step_ok
    assert ok(4, 2, 16, 24, 4, 1, 1) == 1
    assert ok(4, 2, 16, 24, 4, 1, 0) == 0          # an entry that only reads: the kernels that wait
    assert ok(4, 2, 16, 24, 4, 0, 1) == 0          # not a step of one token per sequence
    assert ok(4, 2, 16, 22, 4, 1, 1) == 0          # a size that the kernel does not take
