"""No lane of a group reads group memory that another lane is writing (CPU
only).

test_lanes.py runs the decoder's lanes in many orders and compares samples; a
value that passes through another one on its way (a store of zero, then of the
final value) hides from it when no switch falls between the two.  Here every
load and store is seen: lanesim.cpp is compiled with -fsanitize=thread against
tests/lane_race_hooks.cpp, which records what each lane does to the decoder slot
between two __syncwarp barriers and counts the bytes whose outcome depends on
the order.  Shuffles hold lanes together but order no memory, and count as no
barrier."""
import ctypes
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_host_parity import host_decode
from test_lanes import _golden, _lossy, lane_decode, ls  # noqa: F401 (ls is a fixture)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cuopus_b200", "csrc")


@pytest.fixture(scope="module")
def hc():
    return ctypes.CDLL(os.path.join(ROOT, "cuopus_b200", "lib", "libcuopus_hostcheck.so"))


@pytest.fixture(scope="module")
def race(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ is not installed")
    d = tmp_path_factory.mktemp("race")
    run = lambda *cmd: subprocess.run(cmd, check=True, capture_output=True)  # noqa: E731
    common = ["g++", "-g", "-std=c++17", "-fPIC", "-w", "-I", CSRC, "-c"]
    run(*common, "-O1", "-DCUO_LANE_SIM", "-DCUO_LANE_RACE", "-fsanitize=thread", "-Dmemset=lanerace_memset",
        "-include", "string.h", os.path.join(CSRC, "lanesim.cpp"), "-o", str(d / "lanesim.o"))
    run(*common, "-O2", os.path.join(ROOT, "tests", "lane_race_hooks.cpp"), "-o", str(d / "hooks.o"))
    run("g++", "-shared", "-o", str(d / "librace.so"), str(d / "lanesim.o"), str(d / "hooks.o"), "-lpthread", "-ldl",
        "-Wl,-Bsymbolic")
    lib = ctypes.CDLL(str(d / "librace.so"))
    lib.ls_decode_chains.restype = ctypes.c_longlong
    lib.ls_decode_chains.argtypes = [ctypes.c_void_p] * 6 + [ctypes.c_int] + [ctypes.c_void_p] * 8 + \
        [ctypes.c_int] * 4 + [ctypes.c_uint64, ctypes.c_int, ctypes.POINTER(ctypes.c_ulonglong)]
    return lib


def _same(got, want):
    return got[3] == want[3] and all(np.array_equal(got[k], want[k]) for k in range(3))


@pytest.mark.parametrize("name", ["plain_a", "plain_b", "mixed_mono_a", "mixed_mono_b", "long_hybrid", "code3_120ms",
                                  "mixed_stereo_a"])
@pytest.mark.parametrize("width,fec", [(2, 1), (8, 0)])
def test_lossy_streams_have_no_lane_race(race, hc, name, width, fec):
    """Lost and DTX packets: concealment, comfort noise and the recoveries."""
    ix, chains = _golden(name)
    pk = _lossy(ix["packets"], 5, 0.1, 0.05)
    chains = [c[:2] for c in chains]
    got, _, races = lane_decode(race, pk, chains, ix["channels"], width, 0, 1, fec=fec)
    assert races == 0
    assert all(_same(g, w) for g, w in zip(got, host_decode(hc, pk, chains, ix["channels"], fec=fec)))


def _with_random_packets(packets, seed, n):
    rng = np.random.default_rng(seed)
    pk, chains = [], []
    for _ in range(n):
        a, good = int(rng.integers(0, len(packets) - 6)), int(rng.integers(0, 5))
        chains.append((len(pk), 2 * good + 2))
        pk += packets[a:a + good]
        pk.append(rng.integers(0, 256, int(rng.integers(1, 400)), dtype=np.uint8).tobytes())
        pk += packets[a:a + good] + [b""]
    return pk, chains


@pytest.mark.parametrize("name,channels,width", [("mixed_stereo_a", 2, 32), ("mixed_mono_b", 1, 4), ("plain_b", 2, 8)])
def test_random_packets_have_no_lane_race(race, hc, name, channels, width):
    pk, chains = _with_random_packets(_golden(name)[0]["packets"], width, 40)
    got, _, races = lane_decode(race, pk, chains, channels, width, 0, 3)
    assert races == 0
    assert all(_same(g, w) for g, w in zip(got, host_decode(hc, pk, chains, channels)))


@pytest.mark.parametrize("name,width,max_run", [("plain_b", 2, 3), ("mixed_mono_b", 4, 3), ("long_hybrid", 8, 8),
                                                ("short_stereo_300ms", 16, 8)])
def test_concealment_under_random_interleavings(ls, hc, name, width, max_run):  # noqa: F811
    """Random switches inside every stretch; the one-lane build's samples."""
    ix, chains = _golden(name)
    pk = _lossy(ix["packets"], width, 0.2, 0.05)
    chains = [c[:2] for c in chains]
    for fec in (0, 1):
        got, _, _ = lane_decode(ls, pk, chains, ix["channels"], width, max_run, 50 + width, fec=fec)
        assert all(_same(g, w) for g, w in zip(got, host_decode(hc, pk, chains, ix["channels"], fec=fec)))
