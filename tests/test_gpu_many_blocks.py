"""More neighbouring blocks of one size than one launch's grid takes in its third extent."""
import pytest
import torch

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


def test_blocks_beyond_the_grids_extent(gpu_lib):
    M, N = 65537, 6
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn((N, M), generator=g, device="cuda")
    y = api.whiten_blocks(X, [[m + 1] for m in range(M)])
    # one channel: W = 1 / sqrt(sum x^2 / (N - 1)); the 1e-4 rounding and the floats'
    x = X.double()
    ref = x / (x.square().sum(0) / (N - 1)).sqrt()
    assert (y.double() - ref).abs().max() <= 5e-5 + 1e-6 * ref.abs().max()
