"""The ML-FMM's large passes on the tensor cores (k_translate_mma: M2L level by level and the near field, from 4096 list
entries on, over cached blocks), against the same passes by the seven-stage kernel, which runs them where no blocks are
cached.

Both are FP64 chains of at most 4 x 31 products per translation, at most three translations deep, so they differ by some
hundred roundings: 1e-12 of the largest entry, the bound of the oracle tests.  A mixed-precision solve meets its FP64
tolerance of 1e-8, so its solution is within 1e-6 of the FP64 one as in the mixed-precision tests.
"""
import ctypes as C

import numpy as np
import pytest

from itofoggysim_b200 import _native, scene as S
from test_gpu_mma import scale

pytestmark = pytest.mark.gpu


def long_wave(n, wavelength, orders, z=3):
    rng = np.random.default_rng(7)
    radii = rng.uniform(0.1, 0.3, n)
    sc = S.make_scene(radii, (n / 0.04) ** (1.0 / 3.0), 5, lambda_0=wavelength, n_max=max(orders), z_coupling=z,
                      reference_row_rule=False, gmres_tolerance=1e-8)
    sc.n_range_param = np.array([[1, orders[i % len(orders)]] for i in range(sc.n_param)], np.int32)
    return sc


def entries(s, part):
    """List entries of a pass: 5 M2L, 11 near field."""
    cnt = C.c_int32(0)
    _native.check(s.L.foggy_fmm_lists(s.h, part, None, C.byref(cnt)), s.h)
    return cnt.value


@pytest.mark.parametrize("convention", [0, 1])
@pytest.mark.parametrize("n,wavelength,orders,digits", [
    (400, 6.0, [8], 0.0),                        # M2L at the global order
    (400, 6.0, [1, 9, 4, 7, 2, 5, 8], 0.0),      # unequal orders in a batch and between target and source
    (400, 6.0, [6, 3, 8], 3.0),                  # a larger order on each coarser level
    (400, 2.0, [15, 9, 12], 4.0),
    (1000, 4.0, [3, 5], 2.0),                    # more targets than CTAs wanted: one chunk, written in place
])
def test_matches_seven_stages(native, n, wavelength, orders, digits, convention):
    from itofoggysim_b200 import solver
    sc = long_wave(n, wavelength, orders)
    g = scale(sc)
    rng = np.random.default_rng(3)
    x = (rng.standard_normal(g.size) + 1j * rng.standard_normal(g.size)) * g
    kw = dict(use_ml_fmm=True, fmm_convention=convention, fmm_digits=digits)
    with solver.MultiSphereSolver(sc, pair_tables=1, **kw) as s:
        y = s.calculate_vector_b(x) / g
        assert entries(s, 5) >= 4096 and entries(s, 11) >= 4096
        assert np.array_equal(y, s.calculate_vector_b(x) / g)
    with solver.MultiSphereSolver(sc, pair_tables=-1, **kw) as s:
        ref = s.calculate_vector_b(x) / g
    assert 0.0 < np.abs(y - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("digits", [0.0, 3.0])
def test_mixed_solve(native, digits):
    """A mixed-precision handle's Arnoldi steps take these passes too (in FP64; the others in FP32)."""
    from itofoggysim_b200 import solver
    sc = long_wave(400, 6.0, [6, 3, 8])
    g = scale(sc)
    kw = dict(use_ml_fmm=True, fmm_convention=1, fmm_digits=digits)
    with solver.MultiSphereSolver(sc, pair_tables=-1, **kw) as s:
        want, _ = s.solve()
    with solver.MultiSphereSolver(sc, pair_tables=1, precision=1, **kw) as s:
        x, st = s.solve()
        assert entries(s, 5) >= 4096 and entries(s, 11) >= 4096
        xb = s.solve_block()[0].reshape(-1)
    assert st["status"] == 0 and st["backward_error"] <= sc.gmres_tolerance
    for v in (x, xb):
        assert np.linalg.norm((v - want) / g) <= 1e-6 * np.linalg.norm(want / g)
