"""The fixed-point TEAPOT maps (csrc/fixmap.cuh) compiled for the host and
compared with long double maps over random segments, strengths, beam sizes
and energy spreads (tests/fixmap_check.cpp), beside the same maps in binary64."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
@pytest.mark.parametrize("seed", [1, 2])
def test_fixed_point_maps_against_long_double(tmp_path, seed):
    exe = str(tmp_path / "fixmap_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", ROOT, os.path.join(HERE, "fixmap_check.cpp"), "-o", exe])
    out = subprocess.run([exe, "4000", str(seed)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    v = [float(t) for t in out.stdout.split()]
    segments, fixed, (fx, db) = v[0], v[1], (v[2:8], v[8:14])
    # most random segments have a fixed-point form; the rest mix coordinates
    # too strongly or reach the nonlinear maps' limits
    assert fixed >= 0.3 * segments
    # largest and rms error of x, p and z: no larger than binary64 leaves on
    # the same particles (z ends as a double in both)
    assert all(a <= b for a, b in zip(fx, db)), (fx, db)
