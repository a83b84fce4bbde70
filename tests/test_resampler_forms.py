"""The two forms of the resampler's kernel where one takes over from the other."""
import ctypes

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n_out", [4 * 148 * 2304 - 1, 4 * 148 * 2304, 4 * 148 * 2304 + 1153])
def test_resampler_where_its_forms_meet(cuda, n_out):
    """Exactly the restatement's sums on both sides of the line between the two
    forms of k_resample48to16 (148 SMs), from an input off the word boundary."""
    from cuopus_b200 import cuopus_native as cn
    from oracle import pipeline
    x = np.random.default_rng(n_out).integers(-32768, 32768, 3 * n_out + 24).astype(np.int16)
    d = cuda.zeros(len(x) + 1, dtype=cuda.int16, device="cuda")
    d[1:] = cuda.from_numpy(x).cuda()
    y = cuda.zeros(n_out, dtype=cuda.float32, device="cuda")
    assert cn.lib().cuopus_resample48to16(ctypes.c_void_p(d.data_ptr() + 2), len(x), n_out, ctypes.c_void_p(y.data_ptr()),
                                          ctypes.c_void_p(cuda.cuda.current_stream().cuda_stream), None, 0) == 0
    assert np.array_equal(y.cpu().numpy(), pipeline.resample(x, n_out))


@pytest.mark.gpu
@pytest.mark.parametrize("seconds", [7.0, 100.0])
def test_interleaved_channels_in_both_forms(cuda, seconds):
    """A stereo file to 16 kHz, below and above that line: each channel is the
    restatement's resampling of the int16 decode's channel."""
    from cuopus_b200 import cuopus_native as cn
    from oracle import pipeline
    from perf import cases
    f = cases._files(dict(files=1, min_s=seconds, max_s=seconds, content="stereo"), 3)
    (pcm, ch), = cn.decode_ogg_to_int16(f)
    (got, ch16), = cn.decode_ogg_to_f16k_channels(f)
    assert ch == ch16 == 2
    pcm, got = pcm.cpu().numpy().reshape(-1, 2), got.cpu().numpy().reshape(-1, 2)
    assert len(got) == (len(pcm) - 48) // 3
    for c in range(2):
        assert np.array_equal(got[:, c], pipeline.resample(np.ascontiguousarray(pcm[:, c]), len(got)))
