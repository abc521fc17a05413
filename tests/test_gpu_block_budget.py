"""Device memory of a block application on vectors from the host, against the handle's budget: the vectors' copies in the
reference layout, which for one large sphere among small ones are far larger than the solver's own vectors, are kept
on the device within the budget only.  In a process of its own, since the memory pool serves all of them."""
import subprocess
import sys
import os

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import numpy as np, torch
from itofoggysim_b200 import scene as S, solver
radii = np.concatenate([[1.0], 0.1 + 1e-4 * np.arange(200)])
sc = S.make_scene(radii, 12.0, 3, z_coupling=3)
sc.n_range_param = np.array([[1, 30 if r == 1.0 else 1] for r in sc.radius], np.int32)
sc.n_range = (1, 30)
budget = 160 << 20
with solver.MultiSphereSolver(sc, pair_tables=1, memory_budget=budget) as s:
    X = np.ones((40, s.n), np.complex128)
    assert X.nbytes < 256 << 20 and X.nbytes > budget
    Y = s.calculate_vector_b_block(X[:1])
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    Yb = s.calculate_vector_b_block(X)
    used = free - torch.cuda.mem_get_info()[0]
with solver.MultiSphereSolver(sc, pair_tables=1) as s:
    assert np.array_equal(Yb, s.calculate_vector_b_block(X))
assert np.array_equal(Y[0], Yb[0]) and used <= budget, used
"""


def test_host_vectors_stay_within_the_budget(native):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
