"""Per-block whitening: blocks read and written in place in the recording's rows
(adjacent channels at 16-byte boundaries), blocks through gathered copies
(scattered, odd or misaligned ones, an output that overlays the input) and
neighbouring blocks whose matrices are formed side by side all give the bits of
whitening each block's channels on their own."""
import os

import pytest
import torch

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


def _recording(M, N, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.eye(M, device="cuda") + 0.3 * torch.randn((M, M), generator=g, device="cuda") / M ** 0.5
    return 10.0 * torch.randn((N, M), generator=g, device="cuda") @ A


LAYOUTS = {
    "adjacent": (64, [list(range(1, 33)), list(range(33, 65))]),
    "three sizes": (176, [list(range(1, 9)), list(range(9, 17)), list(range(17, 145)), list(range(145, 177))]),
    "beside a scattered one": (12, [[1, 2, 3, 4], [5, 7, 9, 11], [6, 8, 10, 12]]),
    "misaligned": (16, [list(range(1, 7)), list(range(7, 17))]),
    "odd channels": (13, [list(range(1, 5)), list(range(5, 14))]),
    "one block": (8, [[8, 7, 6, 5, 4, 3, 2, 1]]),
    "single channels": (4, [[2], [1], [4], [3]]),
}


@pytest.mark.parametrize("layout", list(LAYOUTS))
@pytest.mark.parametrize("N", [1, 129, 5003])
@pytest.mark.parametrize("precision,q", [("plain", 0.0), ("mixed", 0.0), ("plain", 0.01)])
def test_blocks_equal_their_own_whitening(gpu_lib, layout, N, precision, q):
    M, blocks = LAYOUTS[layout]
    X = _recording(M, N)
    out = api.whiten_blocks(X, blocks, quantization_unit=q, precision=precision)
    for b in blocks:
        cols = [c - 1 for c in b]
        own = api.whiten(X[:, cols].contiguous(), quantization_unit=q, precision=precision)
        assert torch.equal(out[:, cols], own)


def test_output_over_the_input_and_fma_apply(gpu_lib):
    M, blocks = LAYOUTS["adjacent"]
    X = _recording(M, 5003)
    want = api.whiten_blocks(X, blocks)
    Y = X.clone()
    api.whiten_blocks(Y, blocks, out=Y)
    assert torch.equal(Y, want)
    os.environ["MS3GPU_APPLY_FFMA"] = "1"
    try:
        got = api.whiten_blocks(X, blocks)
        own = api.whiten(X[:, :32].contiguous())
    finally:
        del os.environ["MS3GPU_APPLY_FFMA"]
    assert torch.equal(got[:, :32], own)
