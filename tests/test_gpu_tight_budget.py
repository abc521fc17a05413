"""Mixed precision where only the single-precision pair tables fit the budget: they serve the Arnoldi steps, single and as a
block, so a solve to 1e-12 takes more restarts than the FP64 one (FP32 steps reach 1e-6 or so a cycle), and the solution is
that of the FP64 solve (the operator's condition is some tens: 1e-9 is allowed)."""
import numpy as np
import pytest

from itofoggysim_b200 import scene as S
from test_gpu_mma import scale

pytestmark = pytest.mark.gpu


def test_single_precision_tables_alone(native):
    from itofoggysim_b200 import solver
    n, p, m = 200, 15, 60
    sc = S.make_scene(np.full(n, 0.5), 16.0, 4, n_max=p, gmres_tolerance=1e-12, gmres_restart=m)
    g = scale(sc)
    with solver.MultiSphereSolver(sc) as s:
        want, st64 = s.solve()
    # double-precision tables of 445 MiB, single-precision ones of half that; beside them the library keeps the Krylov
    # basis once more and 4 GiB.  About 150 MiB are in use before: the budget lies in the middle of those that hold
    # one kind only.
    table = n * (n - 1) // 2 * sum((p - max(1, k) + 1) ** 2 for k in range(p + 1)) * 16
    basis = (m + 4) * n * 2 * p * (p + 2) * 16
    budget = (4 << 30) + basis + (150 << 20) + table * 3 // 4
    with solver.MultiSphereSolver(sc, precision=1, memory_budget=budget) as s:
        x, st = s.solve()
        xb, _, _, _, stb = s.solve_block()
    assert st["restarts"] > st64["restarts"] and stb["restarts"] > st64["restarts"]
    for v in (x, xb.reshape(-1)):
        assert np.linalg.norm((v - want) / g) < 1e-9 * np.linalg.norm(want / g)
