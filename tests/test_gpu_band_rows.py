"""Row bands whose border rows are also the stencil's clamp (centre rows run
from 1 to nx - 2): a last band of one row, whose particles belong to the band
before it, and bands of one row throughout.  Densities against the 9-point
weights in extended precision; a particle that no band deposits is missing
from them and from the sum of the line density, which is the bunch's
macrosize (a particle's two weights add up to one).

Tolerance (relative): TOL_FIELD, as every deposit's; a contribution is rounded
to at most 2^-42 of a particle's charge, and the two of a particle to 2^-41 of
it, so the line density's sum to 4.5e-13 of the whole."""
import numpy as np
import pytest

from helpers import TOL_FIELD, rel_err
from test_gpu_deposit_edges import _coords, _density, _sizes
from test_gpu_parity import gpu_bunch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,grid,coords,sizes", [
    (30_000, (507, 990, 8), "edges", None),       # 22 bands of 23 rows and one of 1
    (30_000, (507, 990, 8), "plain", "plain"),
    (5000, (40, 400, 24_300), "edges", None),     # bands of one row
    (5000, (40, 400, 24_300), "plain", "plain"),
])
def test_every_particle_has_a_band(n, grid, coords, sizes):
    from spacecharge import SpaceChargeCalc2p5D
    soa, w = _coords(n, coords), _sizes(n, sizes)
    b = gpu_bunch(soa, 1e9)
    if w is not None:
        b.addPartAttr("macrosize")
        b._part_attr["macrosize"][:n, 0] = w
        b._host_modified()
    calc = SpaceChargeCalc2p5D(*grid)
    calc.trackBunch(b, 0.5)
    assert rel_err(calc.getRhoGrid().getArray(), _density(calc, grid, soa, w)) <= TOL_FIELD
    total = 1e9 * n if w is None else float(np.sum(w))
    assert abs(float(np.sum(calc.getLongGrid().getArray())) - total) <= TOL_FIELD * total
