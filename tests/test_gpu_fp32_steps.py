"""Mixed-precision solves whose Arnoldi steps do run in single precision: scenes with an order above 31, and budgets that
hold the single-precision pair tables alone, with several truncation-order buckets, single and as a block.

FP32 steps reach 1e-6 or so a cycle, so a solve to 1e-12 takes more restarts than the FP64 one: that shows which path ran.
The solution is that of the FP64 solve (the operator's condition is some tens: 1e-9 is allowed).
"""
import dataclasses

import numpy as np
import pytest

from itofoggysim_b200 import scene as S, solver
from test_gpu_mma import scale, scene

pytestmark = pytest.mark.gpu


def waves(n):
    rng = np.random.default_rng(3)
    return dict(wave_theta=rng.uniform(0.1, 3.0, n), wave_phi=rng.uniform(0, 6, n),
                jones=np.tile([1.0, 0.0, 0.0, 0.0], (n, 1)), wave_g=np.ones(n), wave_phase=np.zeros(n),
                wave_d0=np.zeros((n, 3)))


def errors(s, g, want):
    """Both solves of a handle against the FP64 block solution; their restarts."""
    x, st = s.solve()
    xb, _, _, _, stb = s.solve_block()
    assert st["status"] == 0 and stb["status"] == 0
    # the single solve takes the sum of the waves
    for v, w in [(x, want.sum(axis=0))] + list(zip(xb, want)):
        assert np.linalg.norm((v - w) / g) < 1e-9 * np.linalg.norm(w / g)
    return st["restarts"], stb["restarts"]


@pytest.mark.parametrize("tables", [1, -1])
def test_order_above_31(native, tables):
    sc = dataclasses.replace(scene([33, 12, 20, 7, 15, 25, 9, 4, 31], 3, 5), gmres_tolerance=1e-12, gmres_restart=60,
                             **waves(3))
    g = scale(sc)
    with solver.MultiSphereSolver(sc, pair_tables=1) as s:
        want, _, _, _, st = s.solve_block()
        assert errors(s, g, want) == (1, st["restarts"])
    with solver.MultiSphereSolver(sc, pair_tables=tables, precision=1) as s:
        r, rb = errors(s, g, want)
    # without tables a single vector's steps stay FP64: single precision reads its tables, or sums S for a block
    assert (r > 1) == (tables == 1) and rb > st["restarts"]


def test_single_precision_tables_alone(native):
    rng = np.random.default_rng(8)
    n, m = 200, 60
    orders = rng.integers(9, 21, n)
    radii = 0.02 * orders * (1.0 + 1e-4 * np.arange(n))
    sc = S.make_scene(radii, 16.0, 4, z_coupling=3, gmres_tolerance=1e-12, gmres_restart=m, reference_row_rule=False,
                      waves=waves(3))
    order = {float(r): int(q) for r, q in zip(radii, orders)}
    sc.n_range_param = np.array([[1, order[float(r)]] for r in sc.radius], np.int32)
    sc.n_range = (1, 20)
    g = scale(sc)
    with solver.MultiSphereSolver(sc, pair_tables=1) as s:
        want, _, _, _, st64 = s.solve_block()
    # beside the tables the library keeps the Krylov basis once more and 4 GiB; what the handle holds before them is
    # not known here, so the budgets go from too little for either kind to enough for both
    _, table = solver.estimate_solve_bytes(sc)
    base = (4 << 30) + (m + 4) * sc.ragged_unknowns() * 16 + (50 << 20)
    restarts = []
    for f in (0.5, 0.75, 1.0, 1.25, 3.0):
        with solver.MultiSphereSolver(sc, precision=1, memory_budget=int(base + f * table)) as s:
            restarts.append(errors(s, g, want))
    assert restarts[-1] == (1, st64["restarts"])
    assert any(r > 1 and rb > st64["restarts"] for r, rb in restarts)


def test_static_entry_beside_single_precision_tables(native):
    """The FP64 entry without allocation on a mixed-precision handle with both kinds of tables, and the single-precision
    ones made again after a change of the radial function."""
    sc = dataclasses.replace(scene([33, 12, 20, 7, 15], 3, 6), gmres_tolerance=1e-10, gmres_restart=60)
    one = dataclasses.replace(sc, z_coupling=1)
    with solver.MultiSphereSolver(one, pair_tables=1, precision=1) as s:
        fresh = s.solve()[0]
    with solver.MultiSphereSolver(sc, pair_tables=1, precision=1) as s:
        s.solve()
        s.params.precision = 0
        s.params.z_coupling = 1
        s._set()
        x = scale(sc) * np.ones(sc.vector_length())
        y = s.calculate_vector_b(x)
        s.params.precision = 1
        s._set()
        again = s.solve()[0]
        assert np.array_equal(y, s.calculate_vector_b(x))
    assert np.array_equal(again, fresh)
