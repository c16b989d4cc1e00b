"""The 1e-4 rounding in FP32 operations (mountainsort_b200/csrc/quantize.cuh, __host__
__device__), run on the CPU through tests/cpp/quantize_driver.cpp for every 61st float of
its range, both signs: the bits of the reference's double expression."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bits_of_the_double_expression(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "quantize_driver")
    r = subprocess.run([cxx, "-O2", "-ffp-contract=off", "-frounding-math", "-std=c++17", "-I",
                        os.path.join(ROOT, "mountainsort_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "quantize_driver.cpp"), "-o", exe],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    tried, different = map(int, subprocess.run([exe, "61"], capture_output=True, text=True, timeout=600,
                                               check=True).stdout.split())
    assert tried > 30_000_000 and different == 0
