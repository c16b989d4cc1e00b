"""The detector's parallel statistics have the bits of sums in index order: event
times equal the oracle's on data for which the last bits decide (constant
channels, a large offset, values over many binades, values on a coarse grid), at
chunk and segment edges (512 samples), for one channel and for one timepoint."""
import numpy as np
import pytest

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


def _data(kind, N, M):
    rng = np.random.default_rng(17 * N + M)
    g = rng.standard_normal((N, M))
    if kind == "rounded":
        return (np.floor(g / 1e-4 + 0.5) * 1e-4).astype(np.float32)
    if kind == "constant":
        return np.full((N, M), 0.1, np.float32)
    if kind == "offset":
        return (1000 + g).astype(np.float32)
    if kind == "binades":
        return (g * np.exp(rng.uniform(-10, 10, (N, M)))).astype(np.float32)
    if kind == "coarse":
        return np.floor(g * 8).astype(np.float32)
    if kind == "tiny":
        return (g * 1e-42).astype(np.float32)
    X = g.astype(np.float32)
    X[N // 2, 0] = np.inf
    return X


@pytest.mark.parametrize("kind", ["rounded", "constant", "offset", "binades", "coarse", "tiny", "infinity"])
@pytest.mark.parametrize("N,M,chunk", [(1, 1, 0), (511, 3, 0), (20513, 33, 20000), (60001, 1, 0), (45056, 5, 21024)])
def test_event_times_equal_the_oracles(gpu_lib, ref32, kind, N, M, chunk):
    X = _data(kind, N, M)
    for thr, interval, sign in ((1.0, 3.0, 0), (2.0, 25.5, -1), (0.0, 10.0, 1)):
        got = api.detect_events(X, detect_threshold=thr, detect_interval=interval, detect_sign=sign, chunk_size=chunk)
        ref = ref32.detect_events(X, detect_threshold=thr, detect_interval=interval, detect_sign=sign,
                                  chunk_size=chunk or None)
        for m in range(M):
            np.testing.assert_array_equal(got[m], ref[m])
