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


def _shape(hc, cost, want=0):
    c = np.sort(np.asarray(cost, np.float64))[::-1].copy()
    v = hc.hc_choose_shape(ctypes.c_void_p(c.ctypes.data), len(c), want, SMS, 8, 12)
    return v // 100, v % 100


@pytest.mark.parametrize("chains,shape", [(1, (32, 4)), (592, (32, 4)), (593, (32, 5)), (740, (32, 5)), (741, (32, 4)),
                                          (1184, (16, 4)), (1185, (16, 6)), (1776, (16, 6)), (1777, (16, 4)),
                                          (2486, (16, 6)), (2641, (8, 8)), (4736, (8, 8)), (4737, (8, 0)), (20000, (8, 0))])
def test_every_launch_shape_is_reached(hc, chains, shape):
    """Equal chains: the counts at which a shape's groups run out."""
    assert _shape(hc, np.ones(chains)) == shape


def test_launch_shape_follows_the_longest_chain(hc):
    """Short chains behind one long one: the widest shape, whatever their number."""
    assert _shape(hc, [4000.0] + [1.0] * 5000) == (32, 4)
    for want in (8, 16, 32):
        assert _shape(hc, np.ones(3000), want)[0] == want
    assert _shape(hc, np.ones(3000), 4) == (0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("files,width", [(1, 32), (60, 32), (160, 16), (420, 16), (700, 8), (1100, 8)])
def test_file_calls_take_the_shape_and_decode_the_same(cuda, hc, files, width):
    """7 to 7,700 chains: the call's width is the rule's."""
    from cuopus_b200 import cuopus_native as cn
    from oracle import ogg_port
    data = _file()
    ix = ogg_port.demux(data)
    cost = [2.0 * sum(ogg_port.decode_capacity48(p) for p in ix["packets"][c[0]:c[0] + c[1]])
            for c in ogg_port.build_chains(ix, 1.0, 250.0)]
    assert _shape(hc, cost * files)[0] == width
    (want, ch), = cn.decode_ogg_to_int16([data])
    got = cn.decode_ogg_to_int16([data] * files)
    assert cn.last_stats()["width"] == width
    assert all(c == ch and cuda.equal(t, want) for t, c in got)


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
