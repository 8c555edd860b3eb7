"""The integer arithmetic of the FP64 form's gridding (cunfft_gb300/csrc/fixmath.h) on the
CPU against long double: exponential, Gaussian taps, the two products and the conversions
from and to FP64, with the bounds that the header states."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fixed_point_arithmetic_bounds(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "fixmath_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "cunfft_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "fixmath_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=300).stdout
    got = {ln.split()[0]: [float(v) for v in ln.split()[1:] if v != "mean"] for ln in out.splitlines()}
    assert got["exp2neg"][0] <= 0.7            # units of 2^-56
    assert got["gauss"][0] <= 4.0              # 2^-54
    assert -1.0 <= got["mad"][0] and got["mad"][1] <= 1.0 and abs(got["mad"][2]) < 0.01
    assert -0.75 <= got["mad62"][0] and got["mad62"][1] <= 0.75 and abs(got["mad62"][2]) < 0.01
    assert got["roundtrip"][0] <= 1.0          # units of 2^-55 of the value's power of two
    assert got["tofloat"][0] <= 2.0            # one ulp (ties)
