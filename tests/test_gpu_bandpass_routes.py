"""The 480 x 500 column transforms' checked-free loads and stores: odd channel counts,
groups with fewer than 16 pairs, int16 input and output, neighbouring groups in turn,
windows inside and at the ends of the recording, misaligned buffers.  Float output
against the oracle; int16 output equal to the float output scaled and truncated; int16
input equal to the same values as floats."""
import numpy as np
import pytest
import torch

from mountainsort_b200 import api
from oracle import oracle64 as o64

pytestmark = pytest.mark.gpu

ARGS = dict(samplerate=30000, freq_min=300, freq_max=6000, freq_wid=1000, num_threads=16)


def _recording(M, N):
    g = torch.Generator(device="cuda").manual_seed(M)
    return torch.round(100 * torch.randn((N, M), generator=g, device="cuda"))


def _shifted(X, by):
    """X's values in a buffer `by` elements off a 256-byte boundary."""
    out = torch.empty(X.numel() + 8, dtype=X.dtype, device=X.device)[by:by + X.numel()].view(X.shape)
    return out.copy_(X)


@pytest.mark.parametrize("M", [12, 13, 31, 32, 33, 40, 62, 63, 66, 97])
def test_forms_agree(gpu_lib, ref32, M):
    N = 400001  # windows at both ends and two inside
    X = _recording(M, N)
    out = api.bandpass_filter(X, **ARGS)
    ref = ref32.bandpass_filter(X.cpu().numpy(), 30000, 300, 6000, 1000, num_threads=16)
    assert o64.rel_l2(out.cpu().numpy(), ref) <= 1e-6  # two FP32 transforms: 4e-7 apart
    X16 = X.to(torch.int16)
    q = 0.25
    scaled = (out.double() * (1.0 / q)).float().to(torch.int32).to(torch.int16)
    for src in (X, _shifted(X, 1), X16, _shifted(X16, 1), _shifted(X16, 2)):
        assert torch.equal(api.bandpass_filter(src, **ARGS), out)
        assert torch.equal(api.bandpass_filter(src, quantization_unit=q, **ARGS), scaled)
        dst = _shifted(torch.zeros_like(scaled), 1)
        assert torch.equal(api.bandpass_filter(src, quantization_unit=q, out=dst, **ARGS), scaled)
    dst = _shifted(torch.zeros_like(out), 1)
    assert torch.equal(api.bandpass_filter(X, out=dst, **ARGS), out)
    sub = api.bandpass_filter(X16, subsample_factor=3, **ARGS)
    assert torch.equal(sub, out[:3 * (N // 3):3])
