"""Pair tables of mixed-precision requests in the solve server, seen in the footprint that a request is admitted by (host
logic, on the CPU): up to order 31 the solve builds the double-precision tables alone, so a budget that holds these and not
half as much again gives the request its tables.  Without them every operator application sums the coaxial coefficients
again."""
import numpy as np
import pytest

from itofoggysim_b200 import scene as S, solver
from itofoggysim_b200.server import SolveServer


def footprint(sc, budget, precision):
    with SolveServer(max_concurrent=1, memory_budget=budget) as srv:
        rid = srv.submit(sc, precision=precision)
        return srv.wait(rid)[0]["footprint"]


@pytest.mark.parametrize("order,tables", [(15, 1.0), (31, 1.0), (32, 1.5)])
def test_footprint(native, order, tables):
    sc = S.make_scene(np.full(12, 0.5), 6.0, 1, n_max=order)
    base, tb = solver.estimate_solve_bytes(sc)
    mixed = int(tables * tb)
    assert footprint(sc, base + 2 * tb, 0) == base + tb
    assert footprint(sc, base + 2 * tb, 1) == base + mixed
    assert footprint(sc, base + mixed, 1) == base + mixed
    assert footprint(sc, base + mixed - 1, 1) == base
