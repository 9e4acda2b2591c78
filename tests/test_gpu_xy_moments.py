"""The x-y moment sums at the edges of their launch: one particle, a warp's
and a block's edges, more particles than threads; orders with their sums in
registers (2-6) and above."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,n", [(2, 1), (3, 31), (4, 257), (5, 77_825), (6, 200_003), (7, 1000), (16, 33)])
@pytest.mark.parametrize("msize", [False, True])
@pytest.mark.parametrize("D", [0.0, 0.7])
def test_xy_moments_against_numpy(order, n, msize, D):
    rng = np.random.default_rng(order * 1000 + n)
    soa = rng.normal(size=(6, n)) * np.array([4e-3, 1e-3, 3e-3, 1e-3, 5.0, 1e-3])[:, None]
    from orbit_gb300 import workloads as W
    b = W.make_bunch(soa, 1e9)
    m = rng.uniform(0.5, 2.0, n) if msize else np.ones(n)
    dev = b._device_bunch()
    if msize:
        dev.set_macrosizes(m)
    ekm, b2, xa, ya, xb, yb = 1.9, 0.77, 1e-4, -2e-4, 2.1e-3, 1.7e-3
    got = dev.xy_moments(order, [D, ekm, b2, xa, ya, xb, yb])
    X, Y = m * ((soa[0] - D * soa[5] / ekm / b2) - xa), m * (soa[2] - ya)
    for j in range(order):
        for i in range(order + 1 - j):
            if i + j < 2:
                continue
            t = X ** i * Y ** j
            s = 1.0 / (xb ** i * yb ** j) + (1.0 if msize else 0.0)
            stray = np.sum(X ** 2 * Y ** order) if not msize and (i, j) == (2, order) else 0.0
            ref, scale = np.sum(t) * s / m.sum() + stray, np.sum(np.abs(t)) * s / m.sum()
            # powers up to 2 * order roundings, sums over at most ~800 terms
            # a thread and a tree: well below 1e-13 of the absolute terms
            assert abs(got[i, j] - ref) <= 1e-13 * scale, (i, j)
    if not msize:
        t = X ** 2 * Y ** order
        assert abs(got[2, order] - np.sum(t)) <= 1e-13 * np.sum(np.abs(t))
    assert (got[0, 0], got[1, 0], got[0, 1]) == (1.0, xa, ya)
