"""A wait of the power iteration's exchange that gives up in one warp: the call returns an
error, the context stays usable, and the next call gives the values it gave before."""
import numpy as np
import pytest
import torch

from mountainsort_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [200, 500])  # 4 and 8 warps a CTA
@pytest.mark.parametrize("step", ["first", "middle", "last"])
def test_one_warp_gives_up(gpu_lib, monkeypatch, M, step):
    g = torch.Generator(device="cuda").manual_seed(M)
    X = torch.randn((4 * M, M), generator=g, device="cuda", dtype=torch.float64)
    XXt = X.T @ X / X.shape[0]
    before = api.whitening_matrix(XXt).cpu().numpy()
    monkeypatch.setenv("MS3GPU_PCA_GIVE_UP_STEP", str({"first": 0, "middle": 1000, "last": 11 * M - 1}[step]))
    with pytest.raises(_lib.Ms3GpuError, match="timed out"):
        api.whitening_matrix(XXt)
    monkeypatch.delenv("MS3GPU_PCA_GIVE_UP_STEP")
    np.testing.assert_array_equal(api.whitening_matrix(XXt).cpu().numpy(), before)
