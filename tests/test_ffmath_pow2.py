"""Correct rounding of sinf_cr, logf_cr and powf_cr (wrf_gb300/csrc/ffmath.h)
next to powers of two, where the rounding test's half ulp differs on the two
sides, and of the sine's float-float series over its whole range: the host
build of the kernels' code against long double."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_rounding_next_to_powers_of_two(tmp_path):
    exe = str(tmp_path / "pow2_check")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-o", exe,
                    os.path.join(HERE, "native", "ffmath_pow2_check.cpp"), "-lm"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
