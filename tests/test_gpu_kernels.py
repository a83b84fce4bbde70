"""The resampler and the cost model's kernels on the GPU at the sizes where
their tiles and lane splits end, against the CPU restatements."""
import ctypes
import os

import numpy as np
import pytest

from oracle import mlp_port, ogg_port, pipeline

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TILE, SMALL = 2304, 768   # outputs per block of k_resample48to16: long inputs, short ones
LONG = 2 * 148 * TILE     # the shortest input of the long form on 148 SMs


@pytest.mark.gpu
@pytest.mark.parametrize("skew", [0, 1, 3, 7])
@pytest.mark.parametrize("n_out", [1, 2, SMALL // 2 - 1, SMALL // 2 + 1, SMALL, SMALL + 1, 3 * SMALL + 5, LONG - 1, LONG,
                                   LONG + TILE // 2 + 1, LONG + TILE - 1])
def test_resampler_tiles(cuda, n_out, skew):
    """Exactly the restatement's sums (taps in order, one fused multiply-add
    each) at every tile edge, input alignment and number of samples left
    behind the last output."""
    from cuopus_b200 import cuopus_native as cn
    rng = np.random.default_rng(100 * skew + n_out)
    for avail in (3 * n_out - 2, 3 * n_out + 24, 3 * n_out + 200):
        x = rng.integers(-32768, 32768, avail).astype(np.int16)
        x[:: 5] = rng.choice([-32768, 32767], len(x[::5]))
        d = cuda.zeros(avail + 16, dtype=cuda.int16, device="cuda")
        d[skew:skew + avail] = cuda.from_numpy(x).cuda()
        for lead in (0, 1):   # output on a 16-byte boundary, or one float past it
            y = cuda.full((n_out + 2 * lead + 4,), 7.0, dtype=cuda.float32, device="cuda")
            rc = cn.lib().cuopus_resample48to16(ctypes.c_void_p(d.data_ptr() + 2 * skew), avail, n_out,
                                                ctypes.c_void_p(y.data_ptr() + 4 * lead),
                                                ctypes.c_void_p(cuda.cuda.current_stream().cuda_stream), None, 0)
            assert rc == 0
            got = y.cpu().numpy()
            assert np.array_equal(got[lead:lead + n_out], pipeline.resample(x, n_out))
            assert np.all(got[:lead] == 7.0) and np.all(got[lead + n_out:] == 7.0)


@pytest.mark.gpu
def test_features_of_chains_around_a_warp(cuda):
    """Chains of 1, 31, 32, 33 and 100 packets, lost packets among them."""
    from cuopus_b200 import costmodel
    from gpu_util import device_batch
    with open(os.path.join(ROOT, "tests", "golden", "streams", "mixed_stereo_b.opus"), "rb") as f:
        packets = list(ogg_port.demux(f.read())["packets"])
    for k in (5, 40, 41, 200):
        packets[k] = b""
    chains = [(0, 1), (3, 31), (20, 32), (39, 33), (150, 100)]
    b, keep_alive, _ = device_batch([packets], [chains], [2])
    got = costmodel.chain_features(b).cpu().numpy()
    want = mlp_port.features(packets, chains, 2)
    assert np.allclose(got, want, rtol=1e-6, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 15, 16, 17, 300])
def test_predictions_around_a_block(cuda, n):
    from cuopus_b200 import costmodel
    rng = np.random.default_rng(n)
    m = costmodel.CostModel(seed=3)
    x = rng.standard_normal((n, 16)).astype(np.float32)
    y = m.predict_raw(cuda.from_numpy(x).cuda()).cpu().numpy()
    want = mlp_port.forward(m.params.cpu().numpy().astype(np.float64), x.astype(np.float64))
    assert np.allclose(y, want, rtol=1e-4, atol=1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("files", [1, 60, 110, 420])
def test_launch_shapes_decode_the_same(cuda, files, monkeypatch):
    """The launch shape follows the number of chains (7 per file: 32, 16 and 8
    lanes, and fewer warps per SM than fit); the samples do not."""
    from cuopus_b200 import cuopus_native as cn
    with open(os.path.join(ROOT, "tests", "golden", "streams", "mixed_stereo_b.opus"), "rb") as f:
        data = f.read()
    (want, ch), = cn.decode_ogg_to_int16([data])
    got = cn.decode_ogg_to_int16([data] * files)
    assert all(c == ch and cuda.equal(t, want) for t, c in got)
    for width in ("8", "16", "32"):
        monkeypatch.setenv("CUOPUS_STRIDE", width)
        (t, _), = cn.decode_ogg_to_int16([data])
        assert cn.last_stats()["width"] == int(width) and cuda.equal(t, want)
