"""The fixed-point lattice pass (k_pass_fx in csrc/program.cu): which bunches,
grids and lattices take it and which particles or maps leave it for the FP64
routines.  Fused programs against the oracle's program executor.

Tolerance: coordinates are held to 1e-10 over 100 kicks elsewhere; each test
here has at most 20, and rounding adds up no faster than linearly in the kicks
of so short a line, so 2e-11."""
import numpy as np
import pytest

import oracle as O
from helpers import coord_err
from test_gpu_parity import gpu_bunch, oracle_sync_of

pytestmark = pytest.mark.gpu
TOL = 2e-11


def _beam(n, kind):
    from orbit_gb300 import workloads as W
    c = W.c2_coords(max(n, 64), seed=11)[:, :n].copy()
    if kind == "outliers":      # beyond 128 times the typical size, slope and dp/p
        c[0, 0], c[2, 1] = 0.9, -0.8
        c[1, 2], c[3, 3] = 0.3, -0.2
        c[5, 4], c[5, 5] = 0.4, -0.25
    elif kind == "offset":      # far off axis in x, much smaller in y
        c[0] = 0.05 + 1e-2 * c[0]
        c[2] *= 1e-3
        c[3] *= 1e-3
    elif kind == "cold":        # no energy spread, no slopes at first
        c[1] = c[3] = c[5] = 0.0
    elif kind == "wide":        # the dp/p limit of the expansions is passed
        c[5] = 0.25 * np.cos(np.arange(n))
    return np.ascontiguousarray(c)


def _lattice(kind, calc):
    from orbit_gb300 import workloads as W
    if kind == "ring":
        return W.ring_lattice(calc, cells=1)
    if kind == "strong":        # fringes beyond their fixed-point range
        return W.fodo_lattice(calc, cells=2, kq=400.0, lq=0.002, ld=0.8, sc_min=0.1)
    if kind == "drifts":
        return W.c1_lattice(calc, cells=6)
    return W.fodo_lattice(calc, cells=2)


@pytest.mark.parametrize("n,beam,lattice,grid,turns", [
    (2, "plain", "fodo", (16, 16, 1), 1),
    (33, "plain", "drifts", (16, 24, 2), 1),
    (1023, "outliers", "fodo", (32, 32, 8), 1),
    (100_003, "outliers", "drifts", (64, 64, 16), 1),
    (100_003, "plain", "ring", (64, 48, 16), 2),
    (20_000, "outliers", "ring", (32, 32, 8), 1),
    (20_000, "offset", "fodo", (40, 24, 16), 2),
    (20_000, "cold", "fodo", (64, 64, 1), 2),
    (20_000, "wide", "ring", (32, 32, 8), 1),
    (20_000, "plain", "strong", (32, 32, 8), 1),
    (50_000, "plain", "fodo", (256, 256, 16), 1),   # the potential stays in global memory
])
def test_fused_program_against_oracle(n, beam, lattice, grid, turns):
    from orbit_gb300 import workloads as W  # noqa: F401 (package path)
    from spacecharge import SpaceChargeCalc2p5D
    soa = _beam(n, beam)
    b = gpu_bunch(soa, 2e13 / max(n, 1000))
    lat = _lattice(lattice, SpaceChargeCalc2p5D(*grid))
    prog = lat.fusedProgram(b)
    assert prog is not None and turns * sum(1 for o in prog.ops if o[0] == 32) <= 20
    lat.trackBunchTurns(b, turns)
    ref = soa.copy()
    assert O.run_program(prog.ops, turns, ref, oracle_sync_of(gpu_bunch(soa, 2e13 / max(n, 1000))), [O.OracleSC(*grid)],
                         nthreads=8) == 0
    assert coord_err(b.getCoordinates(), ref) <= TOL
