"""Lattice passes of beams that are much smaller in one plane: the smaller
plane's coordinates against extended precision, over drifts whose kicks are too
weak to matter (1e-20 particles of charge each).

Tolerance (max-norm relative): every pass stores y as a double and, with dE = 0
and drifts of 1/2 m, no product before that rounds in binary64: half an ulp a
pass, at most 2^-53 of the largest |y|.  In fixed point a typical coordinate
keeps 2^54 units, so that 3 m of drift add less than that to y and a pass less
than 2^-54 to yp.  Twelve drifts' ends and kicks at most."""
import numpy as np
import pytest

from helpers import rel_err
from test_gpu_parity import gpu_bunch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2000, 100_003])
@pytest.mark.parametrize("ratio", [1.0, 2.0 ** -4, 1e-2, 1e-3, 1e-5])
def test_smaller_plane_keeps_its_digits(n, ratio):
    from orbit_gb300 import workloads as W
    from spacecharge import SpaceChargeCalc2p5D
    soa = np.ascontiguousarray(W.c2_coords(n, seed=5))
    soa[2:4] *= ratio
    soa[5] = 0.0
    b = gpu_bunch(soa, 1e-20)
    lat = W.c1_lattice(SpaceChargeCalc2p5D(32, 32, 8), cells=6)
    assert lat.fusedProgram(b) is not None
    lat.trackBunch(b)
    got = b.getCoordinates()
    t = np.longdouble
    for c in (0, 2):
        want = soa[c].astype(t) + t(3.0) * soa[c + 1].astype(t)
        assert float(np.max(np.abs(got[c].astype(t) - want))) <= 12 * 2.0 ** -53 * float(np.max(np.abs(want)))
        assert rel_err(got[c + 1], soa[c + 1]) <= 12 * 2.0 ** -54
