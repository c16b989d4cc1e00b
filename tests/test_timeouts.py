"""The timeout checks of a call run together (mountainsort_b200/csrc/timeouts.h), on the CPU:
every sticky flag that was set is cleared before the one error that names them all, so that
none is left for the next call; and the C ABI's calls use it."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mountainsort_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include <stdexcept>
#include "timeouts.h"
struct Err : std::runtime_error {
    int code;
    Err(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};
int flags[3];
void check(int i) {
    if (!flags[i]) return;
    flags[i] = 0;
    throw Err(-2 - i, "flag " + std::to_string(i));
}
int main() {
    for (int set = 0; set < 8; set++) {
        for (int i = 0; i < 3; i++) flags[i] = (set >> i) & 1;
        try {
            ms3gpu::raise_together<Err>([] { check(0); }, [] { check(1); }, [] { check(2); });
            std::printf("0 none");
        } catch (const Err& e) {
            std::printf("%d %s", e.code, e.what());
        }
        std::printf("|%d%d%d\n", flags[0], flags[1], flags[2]);
    }
    return 0;
}
"""


def test_every_flag_is_cleared_and_named(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "drv.cpp"
    src.write_text(DRIVER)
    exe = str(tmp_path / "drv")
    r = subprocess.run([gxx, "-std=c++17", "-I", CSRC, str(src), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lines = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    for s, line in enumerate(lines):
        which = [i for i in range(3) if s >> i & 1]
        want = f"{-2 - which[0]} " + "; ".join(f"flag {i}" for i in which) if which else "0 none"
        assert line == want + "|000"


def test_no_call_checks_one_flag_after_another():
    """Two checks in a row would leave the second flag set when the first throws."""
    check = r"(?:bandpass|covariance|whitening)_(?:check|raise)_timeout\("
    for f in ("capi.cu", "pipeline.cu", "stream.cu", "cov_i8.cu"):
        text = open(os.path.join(CSRC, f)).read()
        assert not re.search(r"^\s*" + check + r"[^\n]*;\n\s*" + check, text, re.M), f
