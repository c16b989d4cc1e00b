"""The float apply from 11-bit halves: against FP64 for channel counts at the edges of
its tiles (K-blocks of 64, steps of 16, 192 channels per tile, one to three column
tiles) and timepoints at the edges of 128-row tiles and of one tile per SM, on data of
one size and on channels whose gains differ by 10^6; the 1e-4 rounding beyond the FP32
form's range; and rows and columns that hold infinities or NaN."""
import math

import pytest
import torch

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


def _case(M, N, spread, seed=0):
    g = torch.Generator(device="cuda").manual_seed(1000 * M + N + seed)
    A = torch.eye(M, device="cuda", dtype=torch.float64)
    A += 0.3 * torch.randn((M, M), generator=g, device="cuda", dtype=torch.float64) / math.sqrt(M)
    w, v = torch.linalg.eigh(100 * A @ A.T)
    W = (v / w.sqrt()) @ v.T
    X = 10 * torch.randn((N, M), generator=g, device="cuda")
    if spread:
        s = 10 ** (6 * torch.rand(M, generator=g, device="cuda", dtype=torch.float64) - 3)
        X, W = (X.double() * s).float(), W / s[:, None]
    return X, W


@pytest.mark.parametrize("M", [4, 12, 16, 20, 32, 48, 64, 68, 80, 96, 100, 112, 128, 192, 196, 200, 384, 388, 580])
@pytest.mark.parametrize("N", [1, 127, 128, 129, 19000])
@pytest.mark.parametrize("spread", [False, True])
def test_against_fp64(gpu_lib, M, N, spread):
    X, W = _case(M, N, spread)
    ref = X.double() @ W
    size = X.double().abs() @ W.abs()
    for precision in ("plain", "mixed"):
        y = api.whiten_clips(X.reshape(1, N, M), W, precision=precision).reshape(N, M)
        # per term 2^-22 of representation on each side and the rounded sums' 2^-24 per block
        assert ((y - ref).abs() / size).max() <= 1e-6


def test_rounding_beyond_the_fp32_range(gpu_lib):
    M, N = 8, 300
    g = torch.Generator(device="cuda").manual_seed(5)
    scale = 10 ** torch.linspace(-4, 6, N, device="cuda").reshape(N, 1)
    X = (torch.randn((N, M), generator=g, device="cuda") * scale).float()
    W = torch.eye(M, device="cuda", dtype=torch.float64)
    raw = api.whiten_clips(X.reshape(1, N, M), W).reshape(N, M)  # the same sums, unrounded
    want = (torch.floor(raw.double() / 0.0001 + 0.5) * 0.0001).float()
    assert torch.equal(api.apply_whitening_matrix(X, W), want)


def test_infinities_and_nan_stay_in_their_rows_and_columns(gpu_lib):
    M, N = 96, 300
    X, W = _case(M, N, False)
    clean = api.apply_whitening_matrix(X, W)
    for bad in (float("inf"), float("nan")):
        Y = X.clone()
        Y[5, 3], Y[200, 70] = bad, -bad
        out = api.apply_whitening_matrix(Y, W)
        hit = torch.zeros(N, dtype=torch.bool, device="cuda")
        hit[[5, 200]] = True
        assert torch.isnan(out[hit]).all() and torch.equal(out[~hit], clean[~hit])
        V = W.clone()
        V[7, 11] = bad  # input channel 7 into output channel 11
        out = api.apply_whitening_matrix(X, V)
        keep = [m for m in range(M) if m != 11]
        assert torch.isnan(out[:, 11]).all() and torch.equal(out[:, keep], clean[:, keep])
