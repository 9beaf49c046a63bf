"""The move by a precomputed reciprocal (move1_by: q = fl(a r), fl(q + r (a - q d)),
r = fl(1/d)) against the correctly rounded quotient, in exact rational arithmetic:
the same double for every displacement and cell size tried."""
from fractions import Fraction

import numpy as np
import pytest


@pytest.mark.parametrize("d", [0.3, 0.0216, 0.1, 1.0 / 3.0, 13.5 / 625, 0.7, 3.0, 1e-3, 7.25])
def test_reciprocal_quotient_is_the_rounded_quotient(d):
    rng = np.random.default_rng(int(d * 1e6))
    r, dt = 1.0 / d, 0.05
    u = np.concatenate([rng.normal(0, 0.2, 600), rng.normal(0, 1e-8, 100), [0.0, -0.0, 1.0, 1e-30, -3.5]]).astype(np.float32)
    for v in u:
        a = float(v) * dt
        q = a * r
        e = float(Fraction(a) - Fraction(q) * Fraction(d))           # fma(-q, d, a)
        got = float(Fraction(q) + Fraction(e) * Fraction(r))         # fma(e, r, q)
        assert got == a / d, (v, d)
