"""The covariance of up to 32 channels by 4 x 4 blocks (one warp up to 28 channels, two
beyond) and the staged reduction of its slices, at the edges of its stages (32
timepoints), slices and reduction groups: bit-identical to the same channels inside a
wider recording, whose 64 x 64 tiles the general kernel forms in the same order."""
import pytest
import torch

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [4, 8, 24, 28, 32])
@pytest.mark.parametrize("N", [1, 2, 31, 32, 33, 63, 65, 1024, 1057, 37889, 75777, 300001])
def test_bits_of_the_wider_tile(gpu_lib, M, N):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    X = 10 * torch.randn((N, 36), generator=g, device="cuda")
    own = X[:, :M].contiguous()
    C = api.whiten_covariance(own)
    assert torch.equal(C, C.T)
    assert torch.equal(C, api.whiten_covariance(X)[:M, :M])
