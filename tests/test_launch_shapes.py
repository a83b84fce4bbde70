"""The rules that choose lanes per chain (csrc/launch_shape.h): that every
choice is reached and fits the GPU (CPU), and that calls which reach each of
them decode the same samples (GPU)."""
import ctypes
import os

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148


@pytest.fixture(scope="module")
def hc():
    lib = ctypes.CDLL(os.path.join(ROOT, "cuopus_b200", "lib", "libcuopus_hostcheck.so"))
    lib.hc_server_wave_width.argtypes = [ctypes.c_size_t, ctypes.c_int, ctypes.c_int]
    return lib


def _file():
    with open(os.path.join(ROOT, "tests", "golden", "streams", "mixed_stereo_b.opus"), "rb") as f:
        return f.read()   # seven chains


def test_server_waves_reach_every_width_and_fit(hc):
    """A 32-lane wave has a group for each chain and an SM holds eight of them."""
    widths = [hc.hc_server_wave_width(load, SMS, 8) for load in range(1, 48 * SMS)]
    assert sorted(widths, reverse=True) == widths and set(widths) == {32, 16, 8}
    assert widths.count(32) <= 8 * SMS
    assert hc.hc_server_wave_width(10 ** 6, SMS, 8) == 8


@pytest.mark.gpu
@pytest.mark.parametrize("files", [60, 200, 620])
def test_server_waves_of_every_width_decode_the_same(cuda, files):
    """One wave in flight: the first takes the requests that are there, the
    next the other 420, 1,400 or 4,340 chains, at 32, 16 and 8 lanes."""
    from cuopus_b200 import cuopus_native as cn
    from cuopus_b200.serving import Server
    data = _file()
    (t, ch), = cn.decode_ogg_to_int16([data])
    want = t.cpu().numpy()
    with Server(budget_bytes=2 << 30, max_inflight=1) as srv:
        ids = [srv.submit(data) for _ in range(files)]
        for rid in ids:
            out, channels, _ = srv.wait(rid)
            assert channels == ch and np.array_equal(out, want)
