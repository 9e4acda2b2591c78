"""The fixed-point logarithm (csrc/fixlog.cuh) compiled for the host, against
long double.  Bound: the table entry and the series are rounded to 2^-55 once
each (half a unit), the powers of two rounded down (one unit), the series'
seven terms in Q62 and Q68 stay below 2^-59 together, and the terms left out
below t^8 / 8 = 2^-67: 2.2 units of 2^-55, so 0.55 of 2^-53 (of the logarithm
itself where that is above one)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
@pytest.mark.parametrize("seed", [1, 2])
def test_log_against_long_double(tmp_path, seed):
    exe = str(tmp_path / "fixlog_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", ROOT, os.path.join(HERE, "fixlog_check.cpp"), "-o", exe])
    out = subprocess.run([exe, "1000000", str(seed)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    worst, lib = (float(v) for v in out.stdout.split())
    assert worst <= 0.55, (worst, lib)
