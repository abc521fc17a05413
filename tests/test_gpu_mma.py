"""The tensor-core FP64 operator (k_direct_mma: over pair tables, and summing the coaxial coefficients itself) at the
orders where its tiles, k-steps and batches end, against the seven-stage translations.  Those still run the ML-FMM's
passes over few entries: with a one-level tree every sphere is every other's near neighbour, so that operator is
the direct one.

All are FP64 chains of at most 4 x 31 products of numbers of the result's size per entry, so they differ by some
hundred roundings at most: 1e-12 of a sphere's largest entry, the bound of the oracle tests.
"""
import math

import numpy as np
import pytest

from itofoggysim_b200 import scene as S

pytestmark = pytest.mark.gpu


def scene(orders, z, seed, row_rule=False):
    p = np.asarray(orders)
    radii = 0.1 + 0.02 * p * (1.0 + 1e-3 * np.arange(len(p)))
    sc = S.make_scene(radii, 4.4 * radii.max() * len(p) ** (1.0 / 3.0), seed, z_coupling=z, reference_row_rule=row_rule)
    order = {float(r): int(q) for r, q in zip(radii, p)}
    sc.n_range_param = np.array([[1, order[float(r)]] for r in sc.radius], np.int32)
    sc.n_range = (1, int(p.max()))
    return sc


def scale(sc):
    g = np.array([math.sqrt(math.factorial(n + m) / math.factorial(n - m))
                  for n in range(1, sc.n_range[1] + 1) for m in range(-n, n + 1)])
    return np.tile(g, 2 * sc.n_spheres)


def seven_stages(sc, x):
    from itofoggysim_b200 import solver
    one = S.Scene(**{**sc.__dict__, "tree_l_max": 1})
    with solver.MultiSphereSolver(one, use_ml_fmm=True, fmm_convention=1, pair_tables=-1) as s:
        return s.calculate_vector_b(x)


def compare(sc, seed=0):
    from itofoggysim_b200 import solver
    rng = np.random.default_rng(seed)
    g = scale(sc)
    x = (rng.standard_normal(g.size) + 1j * rng.standard_normal(g.size)) * g
    n = sc.n_spheres
    ref = (seven_stages(sc, x) / g).reshape(n, -1)
    for tables in (1, -1):
        with solver.MultiSphereSolver(sc, pair_tables=tables) as s:
            y = s.calculate_vector_b(x)
            assert np.array_equal(y, s.calculate_vector_b(x))   # fixed order of sums
        err = np.abs((y / g).reshape(n, -1) - ref).max(axis=1)
        assert np.all(err <= 1e-12 * np.abs(ref).max(axis=1)), (tables, err.max())


@pytest.mark.parametrize("z", [1, 3])
@pytest.mark.parametrize("orders", [
    [1, 1],                              # smallest of all, batches with empty units
    [1, 2, 3, 4, 5],
    [7] * 6, [8, 7, 9, 8, 6, 8],         # one k-step of orders, and the second
    [15] * 5, [16, 15, 17, 16],          # one tile of orders, and the second; one launch template and the next
    [23] * 5, [24, 23, 25, 24, 22],
    [31, 30, 31, 29, 31, 28],            # the largest order
    [31, 1, 16, 7, 24, 11, 2, 30, 8],    # unequal orders in one batch and between target and source
    [12] * 33, [3] * 170,                # more than one block of eight batches in a chunk
])
def test_matches_seven_stages(native, orders, z):
    compare(scene(orders, z, seed=len(orders) + orders[0]))


def test_row_rule_and_single_order_above(native):
    compare(scene([9, 12, 12, 5, 12], 3, 3, row_rule=True))
    compare(scene([32, 20, 9], 3, 4))    # one order above the tensor-core operator's: the other path


def test_coincident_centres_add_the_source(native):
    sc = scene([6, 9, 9, 4], 1, 5)
    sc.centres[2] = sc.centres[1]
    sc.centres[3] = sc.centres[0]
    compare(sc)


def test_axial_pairs(native):
    sc = scene([10, 10, 10, 10, 10], 3, 6)
    sc.centres[:] = 0.0
    sc.centres[:, 2] = np.array([-6.0, -2.0, 0.0, 2.5, 7.0])
    sc.centres[4, 0] = 1e-9              # near the axis, where cos(theta) rounds to +-1
    compare(sc)


def test_nan_stays_with_the_targets_it_reaches(native):
    from itofoggysim_b200 import solver
    sc = scene([5] * 6, 3, 7)
    x = np.ones(sc.vector_length(), np.complex128)
    c = sc.vector_length() // sc.n_spheres
    x[2 * c] = np.nan
    ref = seven_stages(sc, x)
    for tables in (1, -1):
        with solver.MultiSphereSolver(sc, pair_tables=tables) as s:
            y = s.calculate_vector_b(x)
        assert np.array_equal(np.isnan(y.real) | np.isnan(y.imag), np.isnan(ref.real) | np.isnan(ref.imag))


@pytest.mark.parametrize("nv", [1, 3, 35])
def test_block_of_vectors(native, nv):
    """Several vectors per application (35: more than one vector per slab of the final sum) against one at a time."""
    from itofoggysim_b200 import solver
    sc = scene([12, 5, 17, 9, 12, 12, 8], 3, 8)
    g = scale(sc)
    rng = np.random.default_rng(nv)
    X = (rng.standard_normal((nv, g.size)) + 1j * rng.standard_normal((nv, g.size))) * g
    with solver.MultiSphereSolver(sc, pair_tables=1) as s:
        Y = s.calculate_vector_b_block(X) / g
        for v in range(nv):
            y = s.calculate_vector_b(X[v]) / g
            assert np.abs(Y[v] - y).max() <= 1e-13 * np.abs(y).max()


def test_mixed_handle_keeps_both_precisions(native):
    """On a mixed-precision handle FP32 asked for by name and the FP64 steps do not disturb each other's tables."""
    from itofoggysim_b200 import solver
    sc = scene([12, 5, 17, 9, 12], 3, 9)
    g = scale(sc)
    x = np.random.default_rng(1).standard_normal(g.size) * g
    with solver.MultiSphereSolver(sc, pair_tables=1, precision=1) as s:
        y0 = s.calculate_vector_b(x)
        f = s.calculate_vector_b_block(x[None], precision=1)[0]
        y1 = s.calculate_vector_b(x)
        assert np.array_equal(f, s.calculate_vector_b_block(x[None], precision=1)[0])
    with solver.MultiSphereSolver(sc, pair_tables=1, precision=1) as s:
        assert np.array_equal(f, s.calculate_vector_b_block(x[None], precision=1)[0])   # FP32 tables first
        y2 = s.calculate_vector_b(x)
    assert np.array_equal(y0, y1) and np.array_equal(y0, y2)
    assert 0.0 < np.abs((f - y0) / g).max() <= 1e-5 * np.abs(y0 / g).max()
