"""The integer-pipe binary64 division (sf::div in csrc/softf64.cuh) compiled
for the host and compared bit for bit with the host's IEEE division."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "py-orbit_gb300", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
@pytest.mark.parametrize("seed", [1, 2])
def test_soft_division_matches_ieee(tmp_path, seed):
    exe = str(tmp_path / "softdiv_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
                           os.path.join(HERE, "softdiv_check.cpp"), "-o", exe])
    out = subprocess.run([exe, "2000000", str(seed)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip() == "0", out.stdout + out.stderr
