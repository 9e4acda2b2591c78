"""State shared between bunches and calls: batches whose members differ in what
the fixed-point pass depends on, block shapes carried from one batch to another,
and one bunch's moments asked for by two threads.

Tolerance: the members of a mixed batch take the FP64 pass where single-bunch
tracking takes the fixed-point one; 2e-11 for at most 20 kicks (half of
1e-10 per 100 kicks, the bound coordinates are held to elsewhere, for so short a
line)."""
import threading

import numpy as np
import pytest

from helpers import coord_err

pytestmark = pytest.mark.gpu
TOL = 2e-11


def _ring(pole, kl, n, seed):
    from orbit.teapot import MultipoleTEAPOT
    from orbit_gb300 import workloads as W
    from spacecharge import SpaceChargeCalc2p5D
    lat = W.ring_lattice(SpaceChargeCalc2p5D(32, 32, 8), cells=1)
    for node in lat.getNodes():
        if isinstance(node, MultipoleTEAPOT):
            node.setParam("poles", [pole])
            node.setParam("kls", [kl])
    return W.make_bunch(W.c2_coords(n, seed=seed), 1e10), lat


def test_members_of_one_batch_may_differ_in_poles():
    from orbit_gb300.batch import BunchBatch
    first, second = (2, 0.4, 5000, 1), (5, 1e6, 7001, 2)
    members = [_ring(*first), _ring(*second)]
    bb = BunchBatch(members)
    assert len(bb.classes()) == 1
    bb._batch.set_tuning(0, 768, 8192, 512, 4096, 1)
    bb.trackTurns(1)
    for (b, _), spec in zip(members, (first, second)):
        ref, lat = _ring(*spec)
        lat.trackBunch(ref)
        assert coord_err(b.getCoordinates(), ref.getCoordinates()) <= TOL


def test_shapes_reported_by_one_batch_are_taken_by_a_new_one():
    from orbit_gb300 import workloads as W
    from orbit_gb300.batch import BunchBatch
    from spacecharge import SpaceChargeCalc2p5D

    def batch():
        return BunchBatch([(W.make_bunch(W.c2_coords(n, seed=n), 1e9),
                            W.fodo_lattice(SpaceChargeCalc2p5D(64, 64, 16), cells=4)) for n in (100_003, 400_000)])
    tuned = batch()
    tuned.trackTurns(1)
    keys = ("dep_threads", "dep_chunk", "pass_threads", "pass_chunk", "fft_radix2")
    for k, c in enumerate(tuned.classes()):
        fresh = batch()
        assert fresh.classes()[k]["grid"] == c["grid"]
        fresh._batch.set_tuning(k, *(c[q] for q in keys))
        fresh.trackTurns(1)
        assert [fresh.classes()[k][q] for q in keys] == [c[q] for q in keys]


def test_moments_of_one_bunch_from_two_threads():
    from orbit_gb300 import workloads as W
    dev = W.make_bunch(W.c2_coords(50_000, seed=5), 1.0)._device_bunch()
    par = [0.0, 1.9, 0.77, 1e-4, -2e-4, 2.1e-3, 1.7e-3]
    want = {o: dev.xy_moments(o, par) for o in (2, 8)}
    bad = []

    def work(order):
        for _ in range(40):
            if not np.array_equal(dev.xy_moments(order, par), want[order]):
                bad.append(order)
    ts = [threading.Thread(target=work, args=(o,)) for o in want]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
