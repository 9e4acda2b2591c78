"""Which lattice passes run in fixed point and how many particles their FP64
routines take (SpaceChargeCalc2p5D's pass_counters), with the coordinates
against the oracle: declined particles wait for the end of the block's loop and
are taken 32 rounds of a thread at a time.

Tolerance: as tests/test_gpu_fixed_pass.py, 2e-11 over at most 20 kicks."""
import numpy as np
import pytest

import oracle as O
from helpers import coord_err
from test_gpu_fixed_pass import TOL, _beam, _lattice
from test_gpu_parity import gpu_bunch, oracle_sync_of

pytestmark = pytest.mark.gpu

HALO = 0.05  # share of the particles far out


def _coords(n, kind):
    if kind != "halo":
        return _beam(n, kind)
    c = _beam(n, "plain") * np.array([1e-2, 1e-2, 1e-2, 1e-2, 1.0, 1.0])[:, None]
    k = np.random.Generator(np.random.PCG64(3)).permutation(n)[: int(HALO * n)]
    c[:4, k] *= 300.0
    return np.ascontiguousarray(c)


@pytest.mark.parametrize("n,beam,lattice,grid,fixed,low,high", [
    (1023, "plain", "fodo", (32, 32, 8), 1.0, 0.0, 0.0),
    (100_003, "plain", "ring", (64, 48, 16), 1.0, 0.0, 0.0),
    (100_003, "outliers", "drifts", (64, 64, 16), 1.0, 1.0 / 100_003, 6.0 / 100_003),
    (20_000, "plain", "strong", (32, 32, 8), 0.0, 1.0, 1.0),
    (100_003, "halo", "drifts", (64, 64, 16), 1.0, 0.9 * HALO, 1.1 * HALO),
    (33_333, "halo", "fodo", (256, 256, 4), 1.0, 0.9 * HALO, 1.1 * HALO),
    (3_300_000, "halo", "drifts", (128, 128, 4), 1.0, 0.9 * HALO, 1.1 * HALO),  # more than 32 rounds a thread
])
def test_fixed_passes_and_their_exceptions(n, beam, lattice, grid, fixed, low, high):
    from spacecharge import SpaceChargeCalc2p5D
    soa = _coords(n, beam)
    q = 2e9 if beam == "halo" else 2e13  # a weak beam keeps its halo where it is
    b = gpu_bunch(soa, q / n)
    calc = SpaceChargeCalc2p5D(*grid)
    lat = _lattice(lattice, calc)
    prog = lat.fusedProgram(b)
    lat.trackBunch(b)
    kicks = sum(1 for o in prog.ops if o[0] == 32)
    assert 1 <= kicks <= 20
    passes, particles = calc._calc.pass_counters()
    # (a ring's thin kicks alone move no coordinate: such a pass stays in FP64)
    assert passes == fixed * kicks
    assert low * n * kicks <= particles <= high * n * kicks
    ref = soa.copy()
    assert O.run_program(prog.ops, 1, ref, oracle_sync_of(gpu_bunch(soa, q / n)), [O.OracleSC(*grid)], nthreads=8) == 0
    assert coord_err(b.getCoordinates(), ref) <= TOL
