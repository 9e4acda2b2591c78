"""The deposit's 9-point weights from one square and their exact products
(csrc/fixmap.cuh) compiled for the host: the same integers as separate squares
and 128-bit products give (tests/tsc_weights_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
@pytest.mark.parametrize("seed", [1, 2])
def test_deposit_weights_are_the_separate_squares(tmp_path, seed):
    exe = str(tmp_path / "tsc_weights_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", ROOT, os.path.join(HERE, "tsc_weights_check.cpp"),
                           "-o", exe])
    out = subprocess.run([exe, "1000000", str(seed)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip() == "0", out.stdout + out.stderr
