"""The tensor-core covariance beside other recordings' kernels, whose traffic lets its copies
land late and out of order: the bits of the calls made one by one, every time."""
import pytest
import torch

from mountainsort_b200 import api

pytestmark = pytest.mark.gpu


def test_batch_repeats_the_single_calls_bits(gpu_lib):
    g = torch.Generator(device="cuda").manual_seed(3)
    opts = {"samplerate": 30000.0, "freq_min": 300.0, "freq_max": 6000.0, "freq_wid": 1000.0, "num_threads": 16}
    jobs = [{"X": 10 * torch.randn((N, M), generator=g, device="cuda"), **opts}
            for M, N in ((384, 49324), (32, 198375), (16, 680868), (128, 277534), (64, 242047))]
    want = [api.bandpass_whiten(j["X"], 30000.0, 300.0, 6000.0, 1000.0, num_threads=16) for j in jobs]
    for _ in range(60):
        for got, w in zip(api.bandpass_whiten_batch(jobs), want):
            assert torch.equal(got, w)
