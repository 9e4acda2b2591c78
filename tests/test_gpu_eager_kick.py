"""The separate kick kernel (kick_direct and kick_rb_direct in
csrc/sc_device.cuh): particles on cell edges and on the grid's limits, outside a
boundary, inside and outside the beam radius of the longitudinal kick, one slice
and several, the potential in shared and in global memory.  Kicks of particles
at rest (so that they are read back unrounded): the transverse ones against the
9-point gradient in extended precision of the potential and line density that
the calculator reports (the oracle's own potential differs by its rounding,
which the gradient amplifies with the number of cells), those inside a boundary
and the longitudinal ones against the oracle.

Tolerances (max-norm relative) as the kicks' elsewhere: 1e-12, and 1e-11 for
the longitudinal kick, whose derivative of the line density cancels."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FIELD, rel_err
from test_gpu_deposit_edges import _coords
from test_gpu_parity import gpu_bunch, oracle_sync_of

pytestmark = pytest.mark.gpu


def _kicks(calc, grid, soa, b, length):
    t, nz = np.longdouble, grid[2]
    g, zg = calc.getPhiGrid(), calc.getLongGrid()
    phi, lam = g.getArray().astype(t), zg.getArray().astype(t)
    val, der, step = [], [], []
    for v, lo, hi, n in ((soa[0], g.getMinX(), g.getMaxX(), grid[0]), (soa[2], g.getMinY(), g.getMaxY(), grid[1])):
        d = (t(hi) - t(lo)) / (n - 1)
        c = (v.astype(t) - t(lo)) / d
        i = np.clip(np.floor(c + t(0.5)).astype(int), 1, n - 2)
        f = c - i
        val.append((i, ((t(0.5) - f) ** 2 / 2, t(0.75) - f * f, (t(0.5) + f) ** 2 / 2)))
        der.append((f - t(0.5), -2 * f, f + t(0.5)))
        step.append(d)
    (ix, wx), (iy, wy) = val
    ex, ey = np.zeros(soa.shape[1], t), np.zeros(soa.shape[1], t)
    for a in range(3):
        for c in range(3):
            q = phi[ix - 1 + a, iy - 1 + c]
            ex += der[0][a] * wy[c] * q
            ey += wx[a] * der[1][c] * q
    dz = (t(zg.getMaxZ()) - t(zg.getMinZ())) / nz
    if nz > 1:
        u = (soa[4].astype(t) - t(zg.getMinZ())) / dz + t(0.5)
        k = np.floor(u).astype(int)
        w = u - k
        line = (1 - w) * lam[(k - 1) % nz] + w * lam[k % nz]
    else:
        line = lam[0]
    s = b.getSyncParticle()
    fac = 2 * t(length) * t(b.classicalRadius()) / (t(s.beta()) ** 2 * t(s.gamma()) ** 3)
    fac /= dz * t(b.macroSize()) * soa.shape[1]
    return {1: -ex / step[0] * line * fac, 3: -ey / step[1] * line * fac}


@pytest.mark.parametrize("n,grid,coords", [
    (2, (16, 16, 1), "plain"),
    (5000, (33, 33, 8), "lattice"),
    (5000, (64, 64, 1), "edges"),
    (20_000, (32, 40, 2), "edges"),
    (20_001, (96, 80, 12), "plain"),
    (60_000, (200, 250, 16), "plain"),
])
def test_kick_in_extended_precision(n, grid, coords):
    from spacecharge import SpaceChargeCalc2p5D
    soa = _coords(n, coords)
    b = gpu_bunch(soa, 1e9)
    calc = SpaceChargeCalc2p5D(*grid)
    calc.trackBunch(b, 0.5)
    got = b.getCoordinates()
    for c, ref in _kicks(calc, grid, soa, b, 0.5).items():
        assert np.abs(ref).max() > 0.0 and np.abs(got[c] - ref).max() <= TOL_FIELD * np.abs(ref).max(), c


def test_kick_inside_a_boundary():
    from spacecharge import Boundary2D, SpaceChargeCalc2p5D
    soa = _coords(30_000, "plain")
    soa[0, ::3] *= 20.0
    b = gpu_bunch(soa, 1e9)
    SpaceChargeCalc2p5D(64, 64, 16).trackBunch(b, 0.5, Boundary2D(128, 10, "Circle", 0.03))
    got, ref = b.getCoordinates(), np.ascontiguousarray(soa.copy())
    assert O.sc_track_bnd(O.OracleSC(64, 64, 16), ref, oracle_sync_of(b), 0.5,
                          O.OracleBoundary(128, 10, "Circle", 0.03), nthreads=8) == 0
    assert np.array_equal(got[1] == 0.0, ref[1] == 0.0)
    for c in (1, 3):
        assert rel_err(got[c], ref[c]) <= TOL_FIELD, c


@pytest.mark.parametrize("n,grid", [(2000, (32, 32, 1)), (2000, (32, 32, 2)), (30_001, (64, 64, 16)),
                                    (30_000, (200, 200, 16))])
def test_longitudinal_kick(n, grid):
    """A dense core and a halo far outside the beam radius."""
    from spacecharge import SpaceChargeCalc2p5Drb
    soa = _coords(n, "plain")
    soa[:4, : 3 * n // 4] *= 0.05
    soa[4] *= np.abs(soa[4]) / 10.0
    b = gpu_bunch(soa, 1e9)
    SpaceChargeCalc2p5Drb(*grid, 1.0).trackBunch(b, 0.5, 0.05)
    got, ref = b.getCoordinates(), np.ascontiguousarray(soa.copy())
    assert O.OracleSCrb(*grid, 1.0).track(ref, oracle_sync_of(b), 0.5, 0.05, nthreads=8) == 0
    for c in (1, 3):
        assert rel_err(got[c], ref[c]) <= TOL_FIELD, c
    if grid[2] > 1:
        assert np.abs(ref[5]).max() > 0.0 and rel_err(got[5], ref[5]) <= 1e-11
    else:
        assert np.array_equal(got[5], ref[5])
