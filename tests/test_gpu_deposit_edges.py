"""The integer deposit (deposit_fast in csrc/sc_device.cuh) at the limits of its
range: particles on cell edges and on the grid's own limits, outside a
boundary's grid, macrosizes from far above the mean down to negative ones, the
smallest bunches that carry macrosizes on it, one and several row bands.
Line densities after one kick against the oracle, densities against the
9-point weights in extended precision on the grid the calculator reports (far
off the axis the oracle's own cell coordinates round by 5e-12 of a cell).

Tolerance (max-norm relative): TOL_FIELD, as every deposit's; a contribution is
rounded to at most 2^-42 of a particle's charge."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL_FIELD, rel_err
from test_gpu_parity import gpu_bunch, oracle_sync_of

pytestmark = pytest.mark.gpu


def _coords(n, kind, seed=7):
    rng = np.random.Generator(np.random.PCG64(seed))
    c = np.zeros((6, n))
    c[[0, 2]] = rng.uniform(-1.0, 1.0, (2, n)) * 1e-2
    c[4] = rng.uniform(-1.0, 1.0, n) * 10.0
    if kind == "lattice":   # cell edges and centres, the limits among them
        c[[0, 2]] = rng.integers(-64, 65, (2, n)) / 64.0
        c[4] = rng.integers(-16, 17, n) / 16.0
        c[0, :2] = c[2, :2] = c[4, :2] = -1.0, 1.0
    if kind == "offset":
        c[0] += 25.0
    if kind == "edges":     # everything within a cell of the limits
        c[[0, 2]] = np.sign(c[[0, 2]]) * (1e-2 - 1e-5 * rng.uniform(0.0, 1.0, (2, n)) ** 4)
        c[4] = np.sign(c[4]) * 10.0
    return c


def _sizes(n, kind):
    if kind is None:
        return None
    m = np.random.Generator(np.random.PCG64(9)).uniform(0.5e9, 1.5e9, n)
    if kind == "spread":
        m *= 10.0 ** np.linspace(-6.0, 4.0, n)
    if kind == "signs":
        m[::3] *= -0.5
        m[1::7] = 0.0
    return m


def _density(calc, grid, soa, w):
    t, g = np.longdouble, calc.getRhoGrid()
    rho = np.zeros(grid[:2], t)
    keep = ((soa[0] >= g.getMinX()) & (soa[0] <= g.getMaxX()) & (soa[2] >= g.getMinY()) & (soa[2] <= g.getMaxY()))
    m = (np.full(soa.shape[1], 1e9) if w is None else w)[keep].astype(t)
    cells = []
    for v, lo, hi, n in ((soa[0], g.getMinX(), g.getMaxX(), grid[0]), (soa[2], g.getMinY(), g.getMaxY(), grid[1])):
        c = (v[keep].astype(t) - t(lo)) * t(n - 1) / (t(hi) - t(lo))
        i = np.clip(np.floor(c + t(0.5)).astype(int), 1, n - 2)
        f = c - i
        cells.append((i, ((t(0.5) - f) ** 2 / 2, t(0.75) - f * f, (t(0.5) + f) ** 2 / 2)))
    (ix, wx), (iy, wy) = cells
    for a in range(3):
        for b in range(3):
            np.add.at(rho, (ix - 1 + a, iy - 1 + b), wx[a] * wy[b] * m)
    return rho.astype(float)


@pytest.mark.parametrize("n,grid,coords,sizes", [
    (2, (16, 16, 1), "plain", None),
    (5000, (33, 33, 8), "lattice", None),
    (5000, (33, 33, 8), "lattice", "plain"),
    (5000, (64, 64, 1), "edges", None),
    (20_000, (32, 40, 2), "edges", "plain"),
    (20_000, (64, 64, 16), "offset", "plain"),
    (511, (32, 32, 4), "plain", "plain"),
    (512, (32, 32, 4), "plain", "plain"),
    (20_000, (32, 32, 8), "plain", "spread"),
    (20_000, (32, 32, 1), "plain", "signs"),
    (60_000, (225, 225, 16), "lattice", None),
    (60_000, (200, 250, 16), "edges", "spread"),
])
def test_densities_against_oracle(n, grid, coords, sizes):
    from spacecharge import SpaceChargeCalc2p5D
    soa, w = _coords(n, coords), _sizes(n, sizes)
    b = gpu_bunch(soa, 1e9)
    if w is not None:
        b.addPartAttr("macrosize")
        b._part_attr["macrosize"][:n, 0] = w
        b._host_modified()
    calc = SpaceChargeCalc2p5D(*grid)
    calc.trackBunch(b, 0.5)
    sc = O.OracleSC(*grid)
    assert sc.track(np.ascontiguousarray(soa.copy()), oracle_sync_of(b), 0.5, msize=w, nthreads=8) == 0
    rho, phi, zg, lim = sc.grids()
    assert rel_err(calc.getRhoGrid().getArray(), _density(calc, grid, soa, w)) <= TOL_FIELD
    assert rel_err(calc.getLongGrid().getArray(), zg) <= TOL_FIELD


@pytest.mark.parametrize("grid", [(64, 64, 16), (256, 256, 16)])
def test_particles_outside_a_boundary(grid):
    """A third of the bunch outside the boundary's grid: no density, but their
    line density counts."""
    from spacecharge import Boundary2D, SpaceChargeCalc2p5D
    soa = _coords(30_000, "plain")
    soa[0, ::3] *= 20.0
    soa[2, 1::5] *= 20.0
    b = gpu_bunch(soa, 1e9)
    calc = SpaceChargeCalc2p5D(*grid)
    calc.trackBunch(b, 0.5, Boundary2D(128, 10, "Circle", 0.03))
    sc = O.OracleSC(*grid)
    assert O.sc_track_bnd(sc, np.ascontiguousarray(soa.copy()), oracle_sync_of(b), 0.5,
                          O.OracleBoundary(128, 10, "Circle", 0.03), nthreads=8) == 0
    rho, phi, zg, lim = sc.grids()
    assert rel_err(calc.getRhoGrid().getArray(), _density(calc, grid, soa, None)) <= TOL_FIELD
    assert rel_err(calc.getLongGrid().getArray(), zg) <= TOL_FIELD
