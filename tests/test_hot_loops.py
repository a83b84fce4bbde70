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


@pytest.fixture(scope="module")
def ls():
    path = os.path.join(ROOT, "cuopus_b200", "lib", "libcuopus_lanesim.so")
    if not os.path.exists(path):
        pytest.fail("libcuopus_lanesim.so must be built (python -m cuopus_b200.build)")
    return ctypes.CDLL(path)


@pytest.mark.parametrize("width,max_run", [(4, 0), (8, 0), (8, 3), (16, 5), (32, 0)])
@pytest.mark.parametrize("order,n", [(10, 16), (16, 40), (10, 60), (16, 320)])
@pytest.mark.parametrize("loud", [14, 26, 30, 31])
def test_lpc_synthesis_on_lanes_saturates_as_the_serial_recursion(ls, width, max_run, order, n, loud):
    rng = np.random.default_rng(7000 * width + 100 * order + n + loud)
    top = (1 << loud) - 1
    hist = rng.integers(-top, top, 16).astype(np.int32)
    exc = rng.integers(-top, top, n).astype(np.int32)
    exc[::7] = rng.choice([top, -top - 1, 0], len(exc[::7]))
    a = rng.integers(-32768, 32768, 16).astype(np.int16)
    want, wwin = _lpc(order, hist, a, exc)
    v = np.zeros(n, np.int32)
    assert ls.ls_silk_lpc_synth(order, _ptr(hist), _ptr(a), _ptr(exc), _ptr(v), n, width, max_run,
                                ctypes.c_uint64(loud)) == 0
    assert v.tolist() == want
    assert hist.tolist() == wwin


@pytest.mark.parametrize("width,max_run", [(1, 0), (8, 0), (8, 1), (32, 0), (32, 2)])
@pytest.mark.parametrize("n,shift", [(1, 1), (7, 3), (63, 120), (64, 1), (257, 8), (2168, 120), (2168, 960)])
def test_history_shift_reads_before_it_writes(ls, width, max_run, n, shift):
    buf = np.arange(1, n + shift + 1, dtype=np.int32)
    want = np.concatenate([buf[shift:], buf[n:]])
    assert ls.ls_lshift_copy(_ptr(buf), n, shift, width, max_run, ctypes.c_uint64(n + shift)) == 0
    assert buf.tolist() == want.tolist()


def _pvq_u(n, k, memo={}):
    """Vectors of n integers whose magnitudes sum to k or, for the first nonzero one, half of them."""
    if n == 0 or k == 0:
        return 1 if n == 0 and k == 0 else 0
    if k == 1:
        return 1
    if (n, k) not in memo:
        memo[n, k] = _pvq_u(n - 1, k) + _pvq_u(n, k - 1) + _pvq_u(n - 1, k - 1)
    return memo[n, k]


def _icwrs(y):
    """celt/cwrs.c icwrs: the index of a pulse vector."""
    idx, k = int(y[-1] < 0), abs(int(y[-1]))
    for j in range(len(y) - 2, -1, -1):
        n = len(y) - j
        idx += _pvq_u(n, k)
        k += abs(int(y[j]))
        if y[j] < 0:
            idx += _pvq_u(n, k + 1)
    return idx


@pytest.mark.parametrize("n,k", [(2, 1), (2, 128), (3, 2), (4, 4), (4, 40), (6, 12), (8, 3), (9, 9), (11, 13),
                                 (16, 1), (16, 7), (22, 8), (44, 5), (96, 4), (176, 3), (176, 1)])
def test_codewords_decode_to_their_pulse_vectors(hc, n, k):
    rng = np.random.default_rng(1000 * n + k)
    for t in range(60):
        y = np.zeros(n, np.int32)
        # all pulses in one place, at either end, or anywhere
        at = [np.full(k, t % n), np.full(k, n - 1 - t % n), rng.integers(0, n, k)][t % 3]
        np.add.at(y, at, 1)
        y *= rng.choice([-1, 1], n).astype(np.int32)
        got = np.full(n, 99, np.int32)
        yy = hc.hc_cwrsi(n, k, ctypes.c_uint32(_icwrs(y)), _ptr(got))
        assert got.tolist() == y.tolist()
        assert yy == int((y.astype(np.int64) ** 2).sum())


@pytest.mark.parametrize("entries", [2, 3, 4, 5, 8, 9, 17, 18])
@pytest.mark.parametrize("flat", [0, 1])
def test_symbol_rows_decode_as_the_plain_search(hc, entries, flat):
    rng = np.random.default_rng(10 * entries + flat)
    for _ in range(20):
        cuts = np.sort(rng.choice(np.arange(1, 256), entries - 1, replace=False))[::-1] if flat else \
            np.array([entries - 1 - i for i in range(entries - 1)])     # likely first symbol, then 1 / 256 each
        icdf = np.concatenate([cuts, [0]]).astype(np.uint8)
        buf = rng.integers(0, 256, 400).astype(np.uint8)
        a, b = np.zeros(601, np.uint32), np.zeros(601, np.uint32)
        hc.hc_icdf(_ptr(buf), 400, _ptr(icdf), entries, 0, 600, _ptr(a))
        hc.hc_icdf(_ptr(buf), 400, _ptr(icdf), entries, 1, 600, _ptr(b))
        assert a.tolist() == b.tolist()


def _up2(S, x):
    """silk/resampler_private_up2_HQ.c, one sample after the other."""
    coef = ((1746, 14986, 39083 - 65536), (6854, 25769, 55542 - 65536))
    out = []
    for v in x:
        for ph in range(2):
            in32 = int(v) << 10
            for s in range(3):
                y = _wrap(in32 - S[3 * ph + s])
                w = y * coef[ph][s] >> 16
                z = _wrap(y + w) if s == 2 else _wrap(w)
                o = _wrap(S[3 * ph + s] + z)
                S[3 * ph + s] = _wrap(in32 + z)
                in32 = o
            out.append(max(-32768, min(32767, (in32 >> 9) + 1 >> 1)))
    return out


@pytest.mark.parametrize("n", [0, 1, 2, 3, 9, 10, 11, 17, 18, 40, 160])
@pytest.mark.parametrize("loud", [200, 32767])
def test_up_sampling_at_every_remainder(hc, n, loud):
    rng = np.random.default_rng(n + loud)
    S = rng.integers(-loud << 10, loud << 10, 6)
    x = rng.integers(-loud, loud + 1, max(n, 1)).astype(np.int16)
    st, out = S.astype(np.int32), np.zeros(2 * n + 2, np.int16)
    want_st = [int(v) for v in S]
    want = _up2(want_st, x[:n])
    hc.hc_silk_up2(_ptr(st), _ptr(out), _ptr(x), n)
    assert out[:2 * n].tolist() == want and not out[2 * n:].any()
    assert st.tolist() == want_st


def _rotation(x, stride, c, s):
    """celt/vq.c exp_rotation1."""
    n = len(x)
    order = list(range(n - stride)) + list(range(n - 2 * stride - 1, -1, -1))
    i16 = lambda v: (v + 32768) % 65536 - 32768
    for i in order:
        x1, x2 = x[i], x[i + stride]
        x[i + stride] = i16(c * x2 + s * x1 + 16384 >> 15)
        x[i] = i16(c * x1 - s * x2 + 16384 >> 15)


@pytest.mark.parametrize("n,stride", [(2, 1), (3, 1), (4, 2), (6, 2), (7, 3), (9, 1), (10, 2), (13, 3), (16, 4), (24, 5),
                                      (48, 6), (88, 9), (176, 13), (176, 1)])
@pytest.mark.parametrize("top", [600, 32767])
def test_rotation_by_residue_classes(hc, n, stride, top):
    rng = np.random.default_rng(n + stride + top)
    for c, s in ((32767, 0), (30274, 12540), (23170, 23170), (12540, 30274), (-32768, 1)):
        x = rng.integers(-top, top + 1, n).astype(np.int16)
        want = [int(v) for v in x]
        _rotation(want, stride, c, s)
        hc.hc_exp_rotation_pass(_ptr(x), n, stride, c, s)
        assert x.tolist() == want


@pytest.mark.parametrize("width,max_run", [(1, 0), (2, 0), (8, 0), (8, 2), (32, 0)])
@pytest.mark.parametrize("n,channels", [(120, 1), (120, 2), (480, 2), (960, 1), (960, 2)])
@pytest.mark.parametrize("accum,top", [(0, 1 << 20), (1, 1 << 27), (0, 300000000)])
def test_deemphasis_by_recursion_and_lanes(ls, width, max_run, n, channels, accum, top):
    rng = np.random.default_rng(n + channels + top)
    x = rng.integers(-top, top, (channels, n)).astype(np.int32)
    pcm = rng.integers(-32768, 32768, n * channels).astype(np.int16)
    mem = rng.integers(-top, top, 2).astype(np.int32)
    want, want_mem = pcm.astype(np.int64), [int(v) for v in mem]
    for c in range(channels):
        m = want_mem[c]
        for j in range(n):
            v = _wrap(int(x[c, j]) + m)
            m = _wrap(27853 * v >> 15)      # celt/celt_decoder.c, coef0 = .85 in 15 bits
            s = max(-32768, min(32767, v + 2048 >> 12))
            q = j * channels + c
            want[q] = max(-32768, min(32767, s + int(want[q]))) if accum else s
        want_mem[c] = m
    assert ls.ls_deemphasis(_ptr(x), _ptr(pcm), n, channels, _ptr(mem), accum, width, max_run, ctypes.c_uint64(n)) == 0
    assert pcm.tolist() == want.tolist()
    assert mem.tolist() == want_mem
