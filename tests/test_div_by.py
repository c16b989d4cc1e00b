"""The power iteration's quotient by one divisor (mountainsort_b200/csrc/div_by.cuh,
__host__ __device__), run on the CPU through tests/cpp/div_by_driver.cu: it must
equal the ordinary division bit for bit, also for mantissas near 1 and near 2 and
over the whole exponent range it accepts."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("div") / "div_by_driver")
    r = subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-I", os.path.join(ROOT, "mountainsort_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "div_by_driver.cu"), "-o", exe],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("span", [0, 3, 60, 499])
def test_quotients_are_the_divisions_bits(driver, span):
    out = subprocess.run([driver, "3000", str(span)], capture_output=True, text=True, timeout=600, check=True)
    tried, different = map(int, out.stdout.split())
    assert tried > 2_900_000 and different == 0
