"""The register power iteration with silent channels, whose entries are zero in every
vector: the bits of the shared-memory kernel, which divides with the ordinary operator,
signs of zeros included, and about the time of a matrix without them."""
import numpy as np
import pytest
import torch

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


def _matrix(M, silent):
    rng = np.random.default_rng(M)
    A = np.eye(M) + 0.3 * rng.standard_normal((M, M)) / np.sqrt(M)
    C = 100.0 * A @ A.T
    C[silent], C[:, silent] = 0.0, 0.0
    return C


@pytest.mark.parametrize("M", [65, 96, 128, 200, 384, 512])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_bits_with_silent_channels(gpu_lib, monkeypatch, M, sign):
    C = _matrix(M, [0, M // 2, M - 1])
    C[C == 0] *= sign
    got = api.whitening_matrix(C, return_components=True)
    monkeypatch.setenv("MS3GPU_PCA_KERNEL", "smem")
    want = api.whitening_matrix(C, return_components=True)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(np.asarray(g).view(np.int64), np.asarray(w).view(np.int64))


@pytest.mark.parametrize("M", [128, 384])
def test_time_with_a_silent_channel(gpu_lib, M):
    def ms(C):
        C = torch.from_numpy(C).cuda()
        best = 1e9
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            api.whitening_matrix(C)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    # ordinary divisions in every step: 1.6 times at 128 channels, 2.3 times at 384
    assert ms(_matrix(M, [M // 2])) <= 1.4 * ms(_matrix(M, []))
