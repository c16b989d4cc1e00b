"""The power iteration's quotient of a zero (mountainsort_b200/csrc/div_by.cuh) on the CPU:
the ordinary division's bits, the sign among them."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_zero_over_any_divisor(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "div_zero_driver")
    r = subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-I", os.path.join(ROOT, "mountainsort_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "div_zero_driver.cu"), "-o", exe],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600, check=True)
    tried, different = map(int, out.stdout.split())
    assert tried > 60_000 and different == 0
