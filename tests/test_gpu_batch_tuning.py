"""Launch shapes of a batch set by hand (orbit_batch_set_tuning): those that a
batch of other bunches reported are taken, whatever its sizes made them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("dep_threads", "dep_chunk", "pass_threads", "pass_chunk", "fft_radix2")


def _batch(sizes, grid):
    from orbit_gb300 import workloads as W
    from orbit_gb300.batch import BunchBatch
    from spacecharge import SpaceChargeCalc2p5D
    members = [(W.make_bunch(W.c2_coords(n, seed=n), 1e9), W.fodo_lattice(SpaceChargeCalc2p5D(*grid), cells=1))
               for n in sizes]
    batch = BunchBatch(members)
    assert len(batch.classes()) == 1
    return batch, [b for b, _ in members]


@pytest.mark.parametrize("grid", [(64, 64, 16), (256, 256, 8)])  # one block and row bands
@pytest.mark.parametrize("shape", [(768, 2632, 512, 2632, 1), (768, 256, 512, 1 << 30, 0), (768, 8192, 512, 257, 1)])
def test_shapes_of_other_bunches(shape, grid):
    sizes = (1000, 50_021)
    plain, want = _batch(sizes, grid)
    plain._batch.set_tuning(0, 768, 8192, 512, 4096, shape[4])
    batch, got = _batch(sizes, grid)
    batch._batch.set_tuning(0, *shape)
    for turn in range(2):
        plain.trackTurns(1)
        batch.trackTurns(1)
        assert [batch.classes()[0][k] for k in KEYS] == list(shape)
        for a, b in zip(got, want):  # integer deposits: the shape changes no bit
            assert np.array_equal(a.getCoordinates(), b.getCoordinates())
    # set again once tables and graphs exist
    batch._batch.set_tuning(0, 768, 1111, 512, 3333, shape[4])
    plain.trackTurns(1)
    batch.trackTurns(1)
    for a, b in zip(got, want):
        assert np.array_equal(a.getCoordinates(), b.getCoordinates())


def test_shapes_change_no_bit_of_beams_at_the_limits_of_fixed_point():
    """Flat beams and beams with a halo: whether a pass runs in fixed point, and
    in which units, hangs on the bunch alone."""
    from orbit_gb300 import workloads as W
    from orbit_gb300.batch import BunchBatch
    from spacecharge import SpaceChargeCalc2p5D

    def run(shape):
        members = []
        for k in range(24):
            c = W.c2_coords(3001 + 997 * k, seed=k)
            c[2:4] *= 0.03 * 1.1 ** k
            if k % 3 == 0:
                c[:4, :: 17 + k] *= 60.0
            members.append((W.make_bunch(np.ascontiguousarray(c), 1e6),
                            W.fodo_lattice(SpaceChargeCalc2p5D(32, 32, 8), cells=1)))
        batch = BunchBatch(members)
        batch.classes()
        batch._batch.set_tuning(0, *shape)
        batch.trackTurns(2)
        return [b.getCoordinates() for b, _ in members]

    want = run((768, 8192, 512, 4096, 1))
    for shape in ((768, 2632, 512, 256, 1), (512, 8192, 512, 16384, 1)):
        for k, (a, b) in enumerate(zip(run(shape), want)):
            assert np.array_equal(a, b), k


@pytest.mark.parametrize("shape", [(768, 255, 512, 4096, 1), (640, 8192, 512, 4096, 1), (768, 8192, 640, 4096, 1),
                                   (768, 8192, 512, -1, 1), (768, 8192, 512, 4096, 2)])
def test_other_shapes_are_refused(shape):
    batch, _ = _batch((1000,), (32, 32, 8))
    with pytest.raises(Exception, match="candidate"):
        batch._batch.set_tuning(0, *shape)
