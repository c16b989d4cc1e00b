"""The deal of the covariance's (run, block pair) items to CTAs
(mountainsort_b200/csrc/cov_share.h), run on the CPU through
tests/cpp/cov_share_driver.cpp: each item once, in range, on level CTAs."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_each_item_once_and_level(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "cov_share_driver")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "mountainsort_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "cov_share_driver.cpp"), "-o", exe],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    tried, bad = map(int, subprocess.run([exe], capture_output=True, text=True, timeout=300, check=True).stdout.split())
    assert tried == 420 and bad == 0
