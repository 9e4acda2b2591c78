"""Which beams the fixed-point maps (csrc/fixmap.cuh, fx::fine_enough) take,
compiled for the host (tests/fixmap_planes_check.cpp): beams whose planes differ
by up to five decades, since one scale serves both planes."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
@pytest.mark.parametrize("seed", [1, 2])
def test_planes_apart(tmp_path, seed):
    exe = str(tmp_path / "fixmap_planes_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", ROOT,
                           os.path.join(HERE, "fixmap_planes_check.cpp"), "-o", exe])
    out = subprocess.run([exe, "6000", str(seed)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    taken, refused, worst, round_share, flat_share = (float(t) for t in out.stdout.split())
    # each coordinate about as close as binary64's.  Both store a double; over a
    # Gaussian beam that rounds by 0.29 x 2.7 of 2^-53 of the geometric mean, and
    # a unit of the fixed point, at most 2^-53 of it, by 0.29.  Where binary64
    # makes no other rounding than the store's, two of a unit before it give
    # sqrt(1 + 2 / 2.7^2) = 1.13; a tenth more for the sample of 400 particles
    assert worst <= 1.13 * 1.1
    # ordinary beams are taken, and a plane a thousand times smaller is not
    assert round_share >= 0.95 and flat_share == 0.0
    assert taken > 2000 and refused > 1000
