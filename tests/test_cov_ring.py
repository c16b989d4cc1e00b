"""The converters' waits on the covariance's stage ring (mountainsort_b200/csrc/cov_ring.h), run
on the CPU through tests/cpp/cov_ring_driver.cpp with copies that land late and out of order:
no stage is taken before its tiles have landed and its slot is free.  The same waits in the
other order (a mistake planted in a copy of the header) take some, so the model can see it."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mountainsort_b200", "csrc")


def _run(tmp_path, name, include):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / name)
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-I", include, os.path.join(ROOT, "tests", "cpp", "cov_ring_driver.cpp"),
                        "-o", exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return tuple(map(int, subprocess.run([exe], capture_output=True, text=True, timeout=300, check=True).stdout.split()))


def test_no_stage_is_taken_early(tmp_path):
    assert _run(tmp_path, "ring", CSRC) == (360000, 0, 0)


def test_the_other_order_takes_stages_early(tmp_path):
    text = open(os.path.join(CSRC, "cov_ring.h")).read()
    right = "(g < stages || planes_read(phase ^ 1u)) && tiles_landed(phase)"
    assert right in text
    (tmp_path / "cov_ring.h").write_text(text.replace(right, "tiles_landed(phase) && (g < stages || planes_read(phase ^ 1u))"))
    _, early, _ = _run(tmp_path, "swapped", str(tmp_path))
    assert early > 0


def test_the_kernel_uses_it():
    assert "ok = converter_may_take(" in open(os.path.join(CSRC, "cov_i8.cu")).read()
