"""Artifact masking at the edges of its copies: stretches of 16384 values and 16-byte
pieces (odd channel counts, intervals longer and shorter than a stretch or than the
value-by-value form's limit, an output or input off a 16-byte boundary), tiles of 64
intervals in the channel limits, no whole interval, and an output over the input: the
oracle's output bit for bit."""
import numpy as np
import pytest
import torch

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


def _data(M, N, I):
    rng = np.random.default_rng(M + N)
    X = rng.standard_normal((N, M)).astype(np.float32)
    for i in range(3, max(4, N // I), 41):
        X[i * I:(i + 1) * I] *= 20
    return X


@pytest.mark.parametrize("M,N,I", [(1, 1, 1), (3, 50, 100), (5, 20001, 1), (1, 70000, 2047), (1, 140001, 2049), (7, 9973, 146),
                                   (64, 66 * 300 + 17, 300), (33, 65 * 500, 500), (13, 64 * 1261 + 3, 1261), (128, 12345, 6000)])
@pytest.mark.parametrize("shift", [0, 1])
def test_oracles_bits(gpu_lib, ref32, M, N, I, shift):
    X = _data(M, N, I)
    ref, kept_ref = ref32.mask_out_artifacts(X, threshold=3.0, interval_size=I)
    src = torch.empty(N * M + 8, device="cuda")[shift:shift + N * M].view(N, M)
    src.copy_(torch.from_numpy(X))
    for dst in (torch.full((N * M + 8,), 7.0, device="cuda")[:N * M].view(N, M),
                torch.full((N * M + 8,), 7.0, device="cuda")[3:3 + N * M].view(N, M), src):
        _, kept = api.mask_out_artifacts(src, threshold=3.0, interval_size=I, out=dst, return_kept=True)
        np.testing.assert_array_equal(dst.cpu().numpy(), ref)
        assert kept == kept_ref


@pytest.mark.parametrize("I", [15, 16, 17, 31, 32, 33, 48])
@pytest.mark.parametrize("nint", [1183, 1185])  # 64 channels: either side of 512 norm sums per SM
def test_norm_batches(gpu_lib, ref32, I, nint):
    X = _data(64, nint * I + 3, I)
    ref, kept_ref = ref32.mask_out_artifacts(X, threshold=3.0, interval_size=I)
    out, kept = api.mask_out_artifacts(torch.from_numpy(X).cuda(), threshold=3.0, interval_size=I, return_kept=True)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    assert kept == kept_ref


@pytest.mark.parametrize("M", [1, 33])
@pytest.mark.parametrize("nint", [1, 2, 255, 256, 257])  # either side of the limits' own flags
def test_few_intervals(gpu_lib, ref32, M, nint):
    X = _data(M, nint * 20 + 3, 20)
    ref, kept_ref = ref32.mask_out_artifacts(X, threshold=3.0, interval_size=20)
    out, kept = api.mask_out_artifacts(torch.from_numpy(X).cuda(), threshold=3.0, interval_size=20, return_kept=True)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    assert kept == kept_ref
