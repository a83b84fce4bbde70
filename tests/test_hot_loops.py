"""The decoder's register-resident loops against plain restatements of the
same recursions (CPU only, the host build of the decoder sources): inputs at
and past the values where the operators saturate, which encoded streams hardly
ever reach."""
import ctypes
import os

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HOSTCHECK = os.path.join(ROOT, "cuopus_b200", "lib", "libcuopus_hostcheck.so")


@pytest.fixture(scope="module")
def hc():
    if not os.path.exists(HOSTCHECK):
        pytest.fail("libcuopus_hostcheck.so must be built (python -m cuopus_b200.build)")
    return ctypes.CDLL(HOSTCHECK)


def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def _wrap(x):
    return (x + (1 << 31)) % (1 << 32) - (1 << 31)


def _sat(x):
    return max(-(1 << 31), min((1 << 31) - 1, x))


def _lpc(order, hist, a, exc):
    """silk/decode_core.c: v = ADD_SAT32(exc, LSHIFT_SAT32(pred, 4)), wrapping tap sums."""
    w, out = [int(x) for x in hist], []
    for e in exc:
        p = order >> 1
        for j in range(order):
            p = _wrap(p + (w[-1 - j] * int(a[j]) >> 16))
        p4 = max(-(1 << 27), min((1 << 27) - 1, p)) << 4
        out.append(_sat(int(e) + p4))
        w = w[1:] + [out[-1]]
    return out, w


@pytest.mark.parametrize("order", [10, 16])
@pytest.mark.parametrize("n", [40, 60, 80])
@pytest.mark.parametrize("loud", [14, 26, 29, 31])
def test_lpc_synthesis_saturates_as_the_serial_recursion(hc, order, n, loud):
    rng = np.random.default_rng(1000 * order + 10 * n + loud)
    top = (1 << loud) - 1
    hist = rng.integers(-top, top, 16).astype(np.int32)
    exc = rng.integers(-top, top, n).astype(np.int32)
    exc[::7] = rng.choice([top, -top - 1, 0], len(exc[::7]))
    a = rng.integers(-32768, 32768, 16).astype(np.int16)
    want, wwin = _lpc(order, hist, a, exc)
    v = np.zeros(n, np.int32)
    hc.hc_silk_lpc_synth(order, _ptr(hist), _ptr(a), _ptr(exc), _ptr(v), n)
    assert v.tolist() == want
    assert hist.tolist() == wwin
