"""The block-parallel comb filter against the serial one (CPU, the host build)."""
import ctypes
import os

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("n", [120, 240, 480, 960])
def test_blocks_equal_the_serial_recursion(n):
    """Lags from the shortest (blocks of 13) to the longest, equal and unequal
    on the two sides, gains of zero among them."""
    hc = ctypes.CDLL(os.path.join(ROOT, "cuopus_b200", "lib", "libcuopus_hostcheck.so"))
    rng = np.random.default_rng(n)
    for _ in range(200):
        lag, gain, tap = ([int(rng.choice(v)) for _ in "01"] for v in ([15, 16, 100, 700, 1022], [0, 3072, 9000, 20000],
                                                                       [0, 1, 2]))
        if rng.random() < 0.2:
            lag[1], gain[1], tap[1] = lag[0], gain[0], tap[0]
        x = rng.integers(-2 ** 27, 2 ** 27, 1100 + n + 8).astype(np.int32)
        out = []
        for lanes in (0, 1):
            y = x.copy()
            hc.hc_comb_filter(ctypes.c_void_p(y.ctypes.data), 1100, *lag, n, *gain, *tap, lanes)
            out.append(y)
        assert np.array_equal(*out), (lag, gain, tap)
