"""The decoder kernel against libopus without a reference tree: the golden
streams (per-packet sample counts, final ranges and SHA-256 of every chain's
samples, made by libopus 1.5.2 fixed point), and the one-lane host build, which
the CPU tests hold to the same fixtures, on lost and random packets."""
import ctypes
import hashlib
import json
import os

import numpy as np
import pytest

from oracle import ogg_port

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLD = os.path.join(ROOT, "tests", "golden")
with open(os.path.join(GOLD, "decode.json")) as _f:
    DECODE = json.load(_f)
with open(os.path.join(GOLD, "index.json")) as _f:
    INDEX = json.load(_f)


def _golden(name):
    with open(os.path.join(GOLD, "streams", name + ".opus"), "rb") as f:
        ix = ogg_port.demux(f.read())
    return ix["packets"], [tuple(c) for c in INDEX[name]["chains_1_250"]], ix["channels"]


@pytest.mark.gpu
@pytest.mark.parametrize("width", [1, 2, 4, 8, 16, 32])
def test_golden_streams_at_every_width(cuda, width):
    from gpu_util import run_batch
    names = sorted(DECODE)
    g = [_golden(n) for n in names]
    got, _ = run_batch([p for p, _, _ in g], [[c[:2] for c in ch] for _, ch, _ in g], [c for _, _, c in g], width=width,
                       schedule=1)
    want = [(n, i, w) for n in names for i, w in enumerate(DECODE[n])]
    assert len(got) == len(want)
    for r, (name, i, w) in zip(got, want):
        assert r["stop"] == w["status"], (name, i)
        assert r["nsamp"].tolist() == w["nsamp"] and r["rng"].tolist() == w["rng"], (name, i)
        assert hashlib.sha256(r["pcm"].astype("<i2").tobytes()).hexdigest() == w["pcm_sha256"], (name, i)


def _damaged(packets, rng, n, p_lost, p_random):
    """n chains of up to 24 packets, some lost, some DTX, some of random bytes."""
    pk, chains = [], []
    for _ in range(n):
        a, k = int(rng.integers(0, len(packets))), int(rng.integers(1, 25))
        run = []
        for p in packets[a:a + k]:
            u = rng.random()
            if u < p_lost:
                p = b""
            elif u < p_lost + 0.05 and (p[0] & 3) == 0:
                p = p[:1]
            elif u > 1 - p_random:
                p = rng.integers(0, 256, int(rng.integers(1, 400)), dtype=np.uint8).tobytes()
            run.append(p)
        chains.append((len(pk), len(run)))
        pk += run
    return pk, chains


@pytest.mark.gpu
@pytest.mark.parametrize("width", [4, 8, 16, 32])
@pytest.mark.parametrize("p_lost,p_random,fec", [(0.15, 0.0, 0), (0.15, 0.0, 1), (0.0, 0.2, 0)])
def test_damaged_chains_equal_the_host_build(cuda, width, p_lost, p_random, fec):
    """400 chains a case (4,800 in all, 1,600 of them with random packets), as
    mono and as stereo output."""
    from gpu_util import run_batch
    from test_host_parity import host_decode
    hc = ctypes.CDLL(os.path.join(ROOT, "cuopus_b200", "lib", "libcuopus_hostcheck.so"))
    rng = np.random.default_rng(1000 * width + 10 * fec + int(10 * p_random))
    names = ["mixed_stereo_b", "mixed_stereo_a", "mixed_mono_b", "long_hybrid", "plain_b"]
    sets = [_damaged(_golden(n)[0], rng, 80, p_lost, p_random) + (1 + i % 2,) for i, n in enumerate(names)]
    got, _ = run_batch([s[0] for s in sets], [s[1] for s in sets], [s[2] for s in sets], width=width, schedule=1, fec=fec)
    k = 0
    for name, (pk, chains, ch) in zip(names, sets):
        for c, (pcm, ns, rg, stop, samples) in enumerate(host_decode(hc, pk, chains, ch, fec=fec)):
            r = got[k]
            k += 1
            assert r["stop"] == stop and r["samples"] == samples, (name, c)
            done = ns.nonzero()[0].size if stop else len(ns)   # packets before the one that stopped the chain
            assert np.array_equal(r["nsamp"][:done], ns[:done]) and np.array_equal(r["rng"][:done], rg[:done]), (name, c)
            assert np.array_equal(r["pcm"][:len(pcm)], pcm), (name, c)
