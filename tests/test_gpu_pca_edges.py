"""The register power iteration at the edges of its instances (32, 64, 96, 128
channels in one CTA; 192, 256, 320, 384, 512 in a cluster of 16) and on matrices
whose norms leave the quotient's fast range: the bits of the shared-memory
kernel, which divides with the ordinary operator."""
import os

import numpy as np
import pytest

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


def _matrix(M, kind):
    rng = np.random.default_rng(1000 * M + len(kind))
    if kind == "zero":
        return np.zeros((M, M))
    if kind == "rank_one":
        v = rng.standard_normal((M, 1))
        return v @ v.T
    A = np.eye(M) + 0.3 * rng.standard_normal((M, M)) / np.sqrt(M)
    C = 100.0 * A @ A.T
    if kind == "tiny":
        return C * 1e-200
    if kind == "nan":
        C[0, 0] = np.nan
    return C


@pytest.mark.parametrize("M", [1, 32, 33, 64, 65, 96, 97, 128, 129, 192, 193, 257, 320, 321, 384, 385, 512, 513])
@pytest.mark.parametrize("kind", ["plain", "zero", "rank_one", "tiny", "nan"])
def test_bits_of_the_shared_memory_kernel(gpu_lib, M, kind):
    C = _matrix(M, kind)
    got = api.whitening_matrix(C, return_components=True)
    os.environ["MS3GPU_PCA_KERNEL"] = "smem"
    try:
        want = api.whitening_matrix(C, return_components=True)
    finally:
        del os.environ["MS3GPU_PCA_KERNEL"]
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
