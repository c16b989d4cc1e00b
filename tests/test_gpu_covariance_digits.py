"""The int8 digit products of mountainsort_b200/csrc/cov_i8.cu at the edges of
its pipeline: recordings of fewer K blocks (32 timepoints) than the two groups
of converter warps or the three ring stages, odd counts, remainders, several
runs, and one to four channel blocks (diagonal and off-diagonal pairs).

The oracle here restates the fixed-point scheme in exact integers: digits of
v = rint(x 2^(30 - e)) (the last digit held at 127 where it would be 128), the
ten kept digit products per pair of values, the channels' own d2 d2 sums on the
diagonal.  The kernel's class sums are exact, so what may differ is its FP64
arithmetic: four weighted classes and the correction per run, the runs' sum and
one division, each rounded once: fewer than 16 roundings of 2^-53, of terms no
larger than the sum of the classes' magnitudes; 2^-49 of that sum is allowed."""
import numpy as np
import pytest

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


def _digits(X):
    e = np.frexp(np.abs(X).max(axis=0))[1]
    xs = np.ldexp(X, 30 - e)
    h = np.rint(xs / 256.0)
    d3 = np.minimum(np.rint(xs - 256.0 * h), 127.0)
    h = h.astype(np.int64)
    d2 = ((h + 128) & 255) - 128
    h = (h - d2) >> 8
    d1 = ((h + 128) & 255) - 128
    d0 = (h - d1) >> 8
    return e, [d0.astype(np.float64), d1.astype(np.float64), d2.astype(np.float64), d3]


def _model(X, R):
    N, M = X.shape
    S, mag = np.zeros((M, M)), np.zeros((M, M))
    for t0 in range(0, N, R):
        e, d = _digits(X[t0 : t0 + R])
        scale = np.ldexp(1.0, e[:, None] + e[None, :] - 60)
        for c in range(4):
            A = sum(d[k].T @ d[c - k] for k in range(c + 1))  # exact: below 2^53
            S += A * 2.0 ** (48 - 8 * c) * scale
            mag += np.abs(A) * 2.0 ** (48 - 8 * c) * scale
        own = np.diag((d[2] * d[2]).sum(axis=0)) * 2.0**16 * scale
        S += own
        mag += own
    return S / max(1, N - 1), mag / max(1, N - 1)


@pytest.mark.parametrize("M", [128, 132, 256, 260, 512])
@pytest.mark.parametrize("N", [2, 33, 96, 129, 8191, 8225, 40001])
def test_digit_products(gpu_lib, M, N):
    rng = np.random.default_rng(M * 100003 + N)
    X = rng.integers(-(2**23) + 1, 2**23, size=(N, M)).astype(np.float64)
    one = np.arange(M) % 4 == 0
    X[:, one] = rng.integers(-63, 64, size=(N, int(one.sum())))
    C = api.whiten_covariance(X.astype(np.float32))
    np.testing.assert_array_equal(C, C.T)
    ref, mag = _model(X, 8192)
    assert np.all(np.abs(C - ref) <= 2.0**-49 * mag)
