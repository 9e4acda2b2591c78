"""Removal of particles flagged dead (Bunch.compress), whichever way the flag
came into the bunch."""
from helpers import *  # noqa: F401,F403 (package path)
import numpy as np
import pytest


@pytest.mark.parametrize("way", ["delete", "copy", "twice"])
def test_compress_removes_flagged_particles(way):
    from bunch import Bunch
    b = Bunch()
    for k in range(40):
        b.addParticle(float(k), 0, 0, 0, 0, 0)
    b.compress()
    assert b.getSize() == 40
    for k in (0, 7, 39):
        b.deleteParticleFast(k)
    if way == "copy":
        c = Bunch()
        b.copyBunchTo(c)
        b = c
    b.compress()
    want = [k for k in range(40) if k not in (0, 7, 39)]
    if way == "twice":
        b.addParticle(99.0, 0, 0, 0, 0, 0)
        b.deleteParticleFast(1)
        b.compress()
        want = [want[0]] + want[2:] + [99]
    assert b.getSize() == len(want)
    assert np.array_equal([b.x(i) for i in range(len(want))], want)
