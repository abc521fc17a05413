"""A vector's result in a block is the same bits whatever else the block holds: the number of vectors, the ones that have
left a block solve, larger calls before on the same handle, and the memory that the handle may use.

Bits, so no tolerance.
"""
import dataclasses

import numpy as np
import pytest

from itofoggysim_b200 import scene as S
from test_gpu_mma import scale, scene

pytestmark = pytest.mark.gpu


def vectors(sc, nv):
    g = scale(sc)
    rng = np.random.default_rng(7)
    return (rng.standard_normal((nv, g.size)) + 1j * rng.standard_normal((nv, g.size))) * g


@pytest.mark.parametrize("orders", [[6] * 90, [5, 9, 12, 14, 17, 21] * 12])
@pytest.mark.parametrize("tables", [1, -1])
def test_operator(native, orders, tables):
    from itofoggysim_b200 import solver
    sc = scene(orders, 3, 21)
    X = vectors(sc, 40)
    with solver.MultiSphereSolver(sc, pair_tables=tables) as s:
        Y1 = s.calculate_vector_b_block(X[:1])
        Y3 = s.calculate_vector_b_block(X[:3])
        Y = s.calculate_vector_b_block(X)
        again = s.calculate_vector_b_block(X[:3])     # after a larger call
    assert np.array_equal(Y1[0], Y[0]) and np.array_equal(Y3, Y[:3]) and np.array_equal(again, Y3)


@pytest.mark.parametrize("budget", [1 << 30, 256 << 20, 128 << 20])
def test_operator_in_little_memory(native, budget):
    """The same where the budget leaves room for the slabs of fewer vectors at a time."""
    from itofoggysim_b200 import solver
    sc = scene([6] * 90, 3, 21)
    X = vectors(sc, 40)
    with solver.MultiSphereSolver(sc, pair_tables=1) as s:
        Y = s.calculate_vector_b_block(X)
    with solver.MultiSphereSolver(sc, pair_tables=1, memory_budget=budget) as s:
        assert np.array_equal(Y, s.calculate_vector_b_block(X))


@pytest.mark.parametrize("tables", [1, -1])
def test_solve(native, tables):
    """With and without the four that have left, and in a block of two."""
    from itofoggysim_b200 import solver
    n = 6
    rng = np.random.default_rng(3)
    base = scene([6] * 90, 3, 21)
    sc = dataclasses.replace(base, wave_theta=rng.uniform(0.1, 3.0, n), wave_phi=rng.uniform(0, 6, n),
                             jones=np.tile([1.0, 0.0, 0.0, 0.0], (n, 1)), wave_g=np.ones(n), wave_phase=np.zeros(n),
                             wave_d0=np.zeros((n, 3)), gmres_restart=4, gmres_tolerance=1e-9)
    two = dataclasses.replace(sc, **{k: getattr(sc, k)[:2] for k in
                                     ("wave_theta", "wave_phi", "jones", "wave_g", "wave_phase", "wave_d0")})
    with solver.MultiSphereSolver(sc, pair_tables=tables) as s:
        x = s.solve_block()[0]
        # four start from their solutions, so they leave at once
        x0 = np.zeros_like(x)
        x0[1:5] = x[1:5]
        alone = s.solve_block(x0=x0)[0]
        fresh = s.solve_block(x0=np.zeros_like(x))[0]
    with solver.MultiSphereSolver(two, pair_tables=tables) as s:
        y = s.solve_block(x0=np.zeros_like(x[:2]))[0]
    assert np.array_equal(fresh[[0, 5]], alone[[0, 5]])
    assert np.array_equal(fresh[:2], y)


def test_slabs_give_way(native):
    """A block application keeps slabs for its vectors in what the budget leaves; a solve that needs that memory afterwards
    gets it: the budgets at which a block solve succeeds are the same with and without an application before."""
    from itofoggysim_b200 import _native, solver
    n = 16
    rng = np.random.default_rng(3)
    sc = dataclasses.replace(scene([6] * 90, 3, 21), wave_theta=rng.uniform(0.1, 3.0, n), wave_phi=rng.uniform(0, 6, n),
                             jones=np.tile([1.0, 0.0, 0.0, 0.0], (n, 1)), wave_g=np.ones(n), wave_phase=np.zeros(n),
                             wave_d0=np.zeros((n, 3)), gmres_restart=60, gmres_tolerance=1e-3)
    X = vectors(sc, 60)

    def solved(budget, before):
        try:
            with solver.MultiSphereSolver(sc, pair_tables=1, memory_budget=budget) as s:
                if before:
                    s.calculate_vector_b_block(X)
                s.solve_block()
            return True
        except _native.FoggyError as e:
            assert e.code == _native.FOGGY_ERR_NOMEM
            return False

    budgets = [mb << 20 for mb in range(40, 400, 12)]
    alone = [solved(b, False) for b in budgets]
    assert True in alone and False in alone
    assert alone == [solved(b, True) for b in budgets]
