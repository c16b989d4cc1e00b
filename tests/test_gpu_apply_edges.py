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


def _bound(M, precision):
    """Of sum |x| |w|: the TF32 form's representation, 2^-22 three times, and its truncated
    additions, twelve to a K-block of 32 or, mixed, three to each 8 channels.  (FP32 FMAs, up
    to 32 channels: half an ulp for each and for W, 33 x 2^-24 at most, below both.)"""
    return 3 * 2.0 ** -22 + (12 if precision == "plain" else 3 * -(-M // 8)) * 2.0 ** -23


def _matrix(kind, M, g):
    dense = 0.1 * torch.randn((M, M), generator=g, device="cuda", dtype=torch.float64) + torch.eye(M, device="cuda", dtype=torch.float64)
    if kind == "identity":
        return torch.eye(M, device="cuda", dtype=torch.float64)
    if kind == "blocks":
        b = torch.arange(M, device="cuda") // 8
        return dense * (b[:, None] == b[None, :])
    if kind == "tiny":
        return torch.eye(M, device="cuda", dtype=torch.float64) + 1e-9 * dense
    if kind == "wide":
        return dense * 2.0 ** (-34 * torch.rand((M, M), generator=g, device="cuda", dtype=torch.float64))
    if kind == "near":  # within the range of the 11-bit halves
        return torch.exp2(-28.5 * torch.rand((M, M), generator=g, device="cuda", dtype=torch.float64)) + torch.eye(M, device="cuda")
    if kind == "silent":  # no weight leads from the loud channel
        loud = min(5, M - 1)
        dense[loud], dense[:, loud] = 0, 0
    return dense


@pytest.mark.parametrize("kind", ["identity", "blocks", "tiny", "wide", "near", "silent"])
@pytest.mark.parametrize("M", [4, 8, 16, 20, 32, 36, 64, 96, 200, 580])
@pytest.mark.parametrize("gain", [1.0, 1e6, 1e12])
def test_one_loud_channel(gpu_lib, kind, M, gain):
    """Each output is as exact as the terms that it sums, whatever a channel that hardly or
    not at all contributes to it holds."""
    N = 300
    g = torch.Generator(device="cuda").manual_seed(M)
    W = _matrix(kind, M, g)
    X = torch.randn((N, M), generator=g, device="cuda")
    loud = min(5, M - 1)
    X[:, loud] *= gain
    ref, size = X.double() @ W, X.double().abs() @ W.abs()
    for precision in ("plain", "mixed"):
        y = api.whiten_clips(X.reshape(1, N, M), W, precision=precision).reshape(N, M)
        assert ((y - ref).abs() <= _bound(M, precision) * size).all()


@pytest.mark.parametrize("M", [8, 64, 96, 200, 2820])
@pytest.mark.parametrize("N", [1, 300])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("kind", ["dense", "blocks"])
def test_tf32_float_output(gpu_lib, M, N, offset, kind):
    """The TF32 kernel's float output, through TMA stores (offset 0: a block matrix of more than
    32 channels, or more than 2816 of any) and straight from registers (off a 16-byte
    boundary); up to 32 channels on a boundary, the FP32 form's."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    W = _matrix(kind, M, g)
    X = torch.randn((N, M), generator=g, device="cuda")
    ref, size = X.double() @ W, X.double().abs() @ W.abs()
    for precision in ("plain", "mixed"):
        room = torch.full((N * M + 8,), 7.0, device="cuda")
        out = room[offset:offset + N * M].view(N, M)
        y = api.apply_whitening_matrix(X, W, out=out, precision=precision)
        # the 1e-4 rounding, and its product's to a float
        assert ((y - ref).abs() <= _bound(M, precision) * size + 5e-5 + 2.0 ** -24 * ref.abs() + 1e-9).all()
        assert (room[:offset] == 7).all() and (room[offset + N * M:] == 7).all()


@pytest.mark.parametrize("M", [4, 12, 16, 20, 28, 32])
@pytest.mark.parametrize("N", [1, 897, 200_001])  # one timepoint, past a group's, several groups a block
def test_fp32_form(gpu_lib, M, N):
    """The FP32 form: an identity gives the values themselves, also in place, and infinities and
    NaN stay in their rows and columns."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    X = torch.randn((N, M), generator=g, device="cuda")
    eye = torch.eye(M, device="cuda", dtype=torch.float64)
    assert torch.equal(api.whiten_clips(X.reshape(1, N, M), eye).reshape(N, M), X)
    want = (torch.floor(X.double() / 0.0001 + 0.5) * 0.0001).float()
    assert torch.equal(api.apply_whitening_matrix(X, eye), want)
    Y = X.clone()
    Y[N // 2, 1], Y[N - 1, M - 1] = float("inf"), float("nan")
    hit = torch.zeros(N, dtype=torch.bool, device="cuda")
    hit[[N // 2, N - 1]] = True
    api.apply_whitening_matrix(Y, eye, out=Y)
    assert torch.isnan(Y[hit]).all() and torch.equal(Y[~hit], want[~hit])
    eye[2, 3] = float("inf")
    keep = [m for m in range(M) if m != 3]
    out = api.apply_whitening_matrix(X, eye)
    assert torch.isnan(out[:, 3]).all() and torch.equal(out[:, keep], want[:, keep])
