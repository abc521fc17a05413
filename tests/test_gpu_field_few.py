"""Field plots of few points, whose spheres are split over CTAs, against the same points in a plot of many.

The two add a point's N spheres in different orders, so they differ by at most N eps times the sum of the spheres'
magnitudes: with fields of the size of the largest component from every sphere, 300 x 300 x 1.1e-16 = 1e-11 of it at worst,
and the square root of that many roundings in practice; 1e-12 is allowed, the bound of the oracle tests.
"""
import time

import numpy as np
import pytest

from itofoggysim_b200 import scene as S
from test_gpu_mma import scale

pytestmark = pytest.mark.gpu


def setup(n, p):
    sc = S.make_scene(np.full(n, 0.45), 2.0 * n ** (1.0 / 3.0) + 0.5, 2, n_max=p)
    rng = np.random.default_rng(n)
    g = scale(sc)
    x = (rng.standard_normal(g.size) + 1j * rng.standard_normal(g.size)) * g
    lo, hi = sc.centres.min(axis=0) - 1.0, sc.centres.max(axis=0) + 1.0
    pts = lo + (hi - lo) * rng.random((6000, 3))
    pts[0] = sc.centres[-1]                       # inside the last sphere
    return sc, x, pts


@pytest.mark.parametrize("n,p", [(1, 3), (2, 1), (4, 45), (9, 30), (17, 2), (71, 5), (300, 4)])
def test_few_points_equal_many(native, n, p):
    from itofoggysim_b200 import solver
    sc, x, pts = setup(n, p)
    with solver.MultiSphereSolver(sc, pair_tables=-1) as s:
        E, H = s.get_field(x, pts)
        assert np.all(E[0] == 0) and np.all(H[0] == 0) and np.abs(E).max() > 0
        for m in (1, 31, 32, 33, 700, 2400):
            e, h = s.get_field(x, pts[:m])
            assert np.abs(e - E[:m]).max() <= 1e-12 * np.abs(E).max()
            assert np.abs(h - H[:m]).max() <= 1e-12 * np.abs(H).max()
            assert np.array_equal(e == 0, E[:m] == 0)


def test_ten_points_do_not_cost_what_thousands_do(native):
    """Ten points among 2000 spheres: 1/120 of the time of ten thousand; with all spheres in one CTA it was a quarter."""
    from itofoggysim_b200 import solver
    sc, x, pts = setup(2000, 8)
    many = np.concatenate([pts, pts])[:10000]

    def best(s, p):
        t = []
        for _ in range(4):
            t0 = time.perf_counter()
            s.get_field(x, p)
            t.append(time.perf_counter() - t0)
        return min(t)

    with solver.MultiSphereSolver(sc, pair_tables=-1) as s:
        assert best(s, pts[:10]) < 0.2 * best(s, many)
