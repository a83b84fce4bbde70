"""The cost model's chain features where another number of lanes takes a chain
(csrc/costmodel.cu, on 148 SMs), against the restatement."""
import numpy as np
import pytest

SMS = 148


@pytest.mark.gpu
@pytest.mark.parametrize("chains", [1, 31, 33, 32 * SMS, 32 * SMS + 1, 64 * SMS + 1, 128 * SMS + 1, 512 * SMS + 1])
def test_features_at_every_number_of_lanes(cuda, chains):
    """0, 1, 2, 3, 5, 17 and 70 packets a chain in turn, empty packets and every
    framing code among them."""
    from cuopus_b200 import costmodel
    from cuopus_b200 import cuopus_native as cn
    from oracle import mlp_port
    rng = np.random.default_rng(chains)
    pool = [rng.integers(0, 256, int(n), dtype=np.uint8).tobytes() for n in rng.integers(0, 60, 300)]
    lens = np.array([len(p) for p in pool], np.uint32)
    counts = np.array([0, 1, 2, 3, 5, 17, 70], np.uint32)[np.arange(chains) % 7]
    first = rng.integers(0, len(pool) - 70, chains).astype(np.uint32)
    first[np.arange(chains) % 7 != 6] += 35
    kinds = np.arange(chains) % 2 + 1
    on = lambda a, t: cuda.from_numpy(np.ascontiguousarray(a, dtype=t)).cuda()  # noqa: E731
    t = dict(data=on(np.frombuffer(b"".join(pool) + bytes(16), np.uint8), np.uint8),
             off=on(np.concatenate([[0], np.cumsum(lens)[:-1]]), np.uint64), len=on(lens, np.uint32),
             first=on(first, np.uint32), npkts=on(counts, np.uint32), channels=on(kinds, np.uint8))
    b = cn.Batch(**{k: v.data_ptr() for k, v in t.items()})
    b.nchains = chains
    got = costmodel.chain_features(b).cpu().numpy()
    assert got.shape == (chains, 16)
    look = np.unique(np.concatenate([np.arange(min(chains, 200)), rng.integers(0, chains, 300),
                                     np.arange(max(0, chains - 40), chains)]))
    for ch in (1, 2):
        rows = [int(c) for c in look if kinds[c] == ch]
        if rows:
            want = mlp_port.features(pool, [(int(first[c]), int(counts[c])) for c in rows], ch)
            assert np.allclose(got[rows], want, rtol=1e-6, atol=1e-6)
