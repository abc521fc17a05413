"""GMRES cycles of exactly k columns, k around the 32 rows that a warp's lanes hold of the back substitution: the residual
after them against that of the least-squares problem over the same Krylov space, solved on the host.

Both solve it stably for a basis orthogonal to rounding, so the relative residuals differ by at most about
k eps cond(A) = 60 x 1.1e-16 x 1e3: 1e-11 is allowed.
"""
import dataclasses

import numpy as np
import pytest

from itofoggysim_b200 import scene as S
from test_gpu_mma import scale

pytestmark = pytest.mark.gpu


def optimal_residuals(s, b, g, ks):
    """||b - A x|| / ||b|| of the best x in the Krylov space of k vectors, k in ks"""
    V = [b / np.linalg.norm(b)]
    H = np.zeros((max(ks) + 1, max(ks)), np.complex128)
    out = {}
    for k in range(max(ks)):
        w = s.calculate_vector_b(g * V[k]) / g
        for _ in range(2):
            Q = np.stack(V)
            c = Q.conj() @ w
            H[:k + 1, k] += c
            w = w - c @ Q
        H[k + 1, k] = np.linalg.norm(w)
        V.append(w / H[k + 1, k])
        if k + 1 in ks:
            e = np.zeros(k + 2, np.complex128)
            e[0] = 1.0
            y = np.linalg.lstsq(H[:k + 2, :k + 1], e, rcond=None)[0]
            out[k + 1] = np.linalg.norm(e - H[:k + 2, :k + 1] @ y)
    return out


def test_columns_of_a_cycle(native):
    from itofoggysim_b200 import solver
    ks = (1, 2, 31, 32, 33, 34, 60)
    base = S.make_scene(np.full(48, 0.5), 4.8, 9, m=1.6 + 0.01j, n_max=6, gmres_restart=60, gmres_tolerance=1e-15)
    with solver.MultiSphereSolver(base) as s:
        b = s.get_vector_b()
        g = scale(base)
        want = optimal_residuals(s, b / g, g, ks)
    for k in ks:
        sc = dataclasses.replace(base, gmres_max_iterations=k)
        with solver.MultiSphereSolver(sc) as s:
            x, _ = s.solve(raise_on_error=False)
            r1 = np.linalg.norm((b - s.calculate_vector_b(x)) / g) / np.linalg.norm(b / g)
            x, _, it, _, _ = s.solve_block(raise_on_error=False)
            rb = np.linalg.norm((b - s.calculate_vector_b(x.reshape(-1))) / g) / np.linalg.norm(b / g)
        assert int(np.asarray(it).reshape(-1)[0]) == k
        assert abs(r1 - want[k]) < 1e-11 and abs(rb - want[k]) < 1e-11
