"""Window lengths with prime factors from 7 to 61 (few channels: 699050 = 2 5 5 11
31 41 at 4 channels and 16 threads, and others): the general radix pass, whose
outputs a thread forms eight at a time, against the oracle, with channel counts that
leave 1 to 8 signals per transform."""
import numpy as np
import pytest

from mountainsort_b200 import api
from oracle import oracle64 as o64

pytestmark = pytest.mark.gpu


def _factors(n):
    out, p = set(), 2
    while n > 1:
        while n % p == 0:
            out.add(p)
            n //= p
        p += 1
    return out


def _cases():
    """For each channel count up to 11, the first thread counts whose windows have factors in 7..61."""
    cases = []
    for M in range(1, 12):
        hits = [T for T in range(1, 200 // M) if 7 <= max(_factors(api.chunk_size(M, T) + 120000)) <= 61
                and api.chunk_size(M, T) < 600000]
        cases += [(M, T) for T in hits[:2]]
    return cases


@pytest.mark.parametrize("M,T", _cases())
def test_against_the_oracle(gpu_lib, ref32, M, T):
    rng = np.random.default_rng(M * 100 + T)
    X = (30 * rng.standard_normal((api.chunk_size(M, T) // 2 + 1, M))).astype(np.float32)
    ref = ref32.bandpass_filter(X, 30000, 300, 6000, 1000, num_threads=T)
    got = api.bandpass_filter(X, 30000, 300, 6000, 1000, num_threads=T)
    assert o64.rel_l2(got, ref) <= 1e-6  # two FP32 transforms: 4e-7 apart at other lengths
