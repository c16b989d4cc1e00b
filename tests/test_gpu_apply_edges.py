"""The float apply at the edges of its dispatch, against FP64."""
import pytest
import torch

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu

# per term 2^-22 of representation on each side and the rounded sums' 2^-24 per block
BOUND = 1e-6


@pytest.mark.parametrize("M", [580, 960, 964, 1024, 1056, 1060, 1156, 1232, 1348, 1408, 1540, 1584, 1732, 1760, 1924, 1936, 2816])
@pytest.mark.parametrize("precision", ["plain", "mixed"])
def test_shared_memory_of_every_tiling(gpu_lib, M, precision):
    """Tiles of 176 columns keep two staging boxes per warp: with many column tiles they
    need more shared memory than the widest tile."""
    N = 200
    g = torch.Generator(device="cuda").manual_seed(M)
    X = torch.randn((N, M), generator=g, device="cuda")
    W = torch.eye(M, device="cuda", dtype=torch.float64) + 0.01 + 0.02 * torch.rand((M, M), generator=g, device="cuda", dtype=torch.float64)
    y = api.whiten_clips(X.reshape(1, N, M), W, precision=precision).reshape(N, M)
    size = X.double().abs() @ W.abs()
    assert ((y - X.double() @ W).abs() / size).max() <= BOUND
