"""GMRES cycles on vectors long enough that a thread of the orthogonalisation has several entries (more than 75776), with
basis sizes around the eight vectors it takes at a time: residuals against the least-squares problem on the host.

The bound is that of test_gpu_back_substitution.py: k eps cond(A) = 17 x 1.1e-16 x 1e3, 1e-11 is allowed."""
import numpy as np
import pytest

from itofoggysim_b200 import scene as S
from test_gpu_back_substitution import optimal_residuals
from test_gpu_mma import scale

pytestmark = pytest.mark.gpu


def test_long_vectors(native):
    from itofoggysim_b200 import solver
    ks = (1, 7, 8, 9, 17)
    base = S.make_scene(np.full(170, 0.5), 8.5, 9, m=1.6 + 0.01j, n_max=15, gmres_restart=20, gmres_tolerance=1e-15)
    assert base.ragged_unknowns() > 75776
    with solver.MultiSphereSolver(base) as s:
        b = s.get_vector_b()
        g = scale(base)
        want = optimal_residuals(s, b / g, g, ks)
        for k in ks:
            s.set_max_iterations(k)
            x, _ = s.solve(raise_on_error=False)
            r1 = np.linalg.norm((b - s.calculate_vector_b(x)) / g) / np.linalg.norm(b / g)
            x = s.solve_block(raise_on_error=False)[0]
            rb = np.linalg.norm((b - s.calculate_vector_b(x.reshape(-1))) / g) / np.linalg.norm(b / g)
            assert abs(r1 - want[k]) < 1e-11 and abs(rb - want[k]) < 1e-11, (k, r1, rb, want[k])
