"""The oracle's Wigner 3j symbols against Racah's sum in exact rational arithmetic, and the time of the translation
blocks that are made of them: every operator is tested against the oracle, up to order 45.

The recurrence carries 64 bits of mantissa over at most 2 min(j1, j2) + 1 <= 200 steps from either end, a few roundings
each, so its error is some 1e-17 of the family's largest value; with the rounding to 53 bits that is 2e-16 of a symbol
(the symbols are below 1), or 1e-16 of the largest where it is smaller.
"""
import math
import time
from fractions import Fraction

import numpy as np
import pytest


def exact_3j(j1, j2, j3, m1, m2):
    f, m3 = math.factorial, -m1 - m2
    if abs(m1) > j1 or abs(m2) > j2 or abs(m3) > j3 or not abs(j1 - j2) <= j3 <= j1 + j2:
        return 0.0
    s = Fraction(0)
    for t in range(max(0, j2 - j3 - m1, j1 - j3 + m2), min(j1 + j2 - j3, j1 - m1, j2 + m2) + 1):
        s += Fraction((-1) ** t, f(t) * f(j3 - j2 + t + m1) * f(j3 - j1 + t - m2) * f(j1 + j2 - j3 - t)
                      * f(j1 - t - m1) * f(j2 - t + m2))
    sq = s * s * Fraction(f(j1 + j2 - j3) * f(j1 - j2 + j3) * f(-j1 + j2 + j3), f(j1 + j2 + j3 + 1))
    sq *= f(j1 - m1) * f(j1 + m1) * f(j2 - m2) * f(j2 + m2) * f(j3 - m3) * f(j3 + m3)
    # the square root by integers: 200 bits
    v = math.isqrt((sq.numerator << 400) // sq.denominator) / 2 ** 200 if sq else 0.0
    return (-1) ** ((j1 - j2 - m3) & 1) * (v if s >= 0 else -v)


def check(oracle, j1, j2, m1, m2):
    js = range(abs(j1 - j2), j1 + j2 + 1)
    want = np.array([exact_3j(j1, j2, j, m1, m2) for j in js])
    got = np.array([oracle.wigner_3j(j1, j2, j, m1, m2, -m1 - m2) for j in js])
    top = np.abs(want).max()
    assert np.all(np.abs(got - want) <= 1e-16 * top + 1.2e-16 * np.abs(want)), (j1, j2, m1, m2)


def test_small_symbols(oracle):
    for j1 in range(5):
        for j2 in range(5):
            for m1 in range(-j1, j1 + 1):
                for m2 in range(-j2, j2 + 1):
                    check(oracle, j1, j2, m1, m2)


@pytest.mark.parametrize("j1,j2,m1,m2", [
    (45, 45, 0, 0), (45, 44, 0, 0), (45, 45, 45, -45), (45, 45, 45, 45), (45, 45, 44, -45), (45, 1, 30, -1),
    (1, 45, 1, 44), (45, 34, -20, 31), (34, 45, 7, -7), (45, 40, 1, 0), (45, 45, 22, -23), (30, 15, -29, 0),
    (98, 115, -69, -100), (100, 100, 0, 0), (100, 99, 50, -50), (0, 45, 0, -45), (45, 0, -45, 0),
])
def test_large_symbols(oracle, j1, j2, m1, m2):
    check(oracle, j1, j2, m1, m2)


def test_outside_the_triangle(oracle):
    assert oracle.wigner_3j(3, 4, 8, 0, 0, 0) == 0.0 and oracle.wigner_3j(3, 4, 0, 0, 0, 0) == 0.0
    assert oracle.wigner_3j(3, 4, 5, 4, -4, 0) == 0.0 and oracle.wigner_3j(3, 4, 5, 1, 1, 1) == 0.0
    assert oracle.wigner_3j(3, 4, 6, 0, 0, 0) == 0.0   # odd sum


def test_translation_block_of_high_order_in_seconds(oracle):
    """One coefficient block of order 34 (1.5 million entries, up to 35 terms each): 0.8 s on eight cores; 28 s with
    integer sums symbol by symbol, and minutes at order 45, which kept the tests of high orders from ending."""
    t = time.perf_counter()
    oracle.translation_xu(40.0, 1.1, 0.4, (1, 34), (1, 34), 3)
    assert time.perf_counter() - t < 10.0
