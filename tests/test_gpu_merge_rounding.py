"""The mean and the standard error that a merge ends with are rounded as IEEE division and square
root round them.

A cash-or-nothing digital without rates pays 0 or 1 per path, so every sum before the last
operations is exact in FP64 whatever its order, and those operations can be repeated here: with
the first unit's mean m (32 paths), s1 and s2 the sums of (sample - m) and its square and n paths,
price = m + s1/n, m2 = s2 - s1 (s1/n) in one rounding and the standard error
sqrt(m2 / ((n - 1) n)).  Equality of doubles.
"""
from __future__ import annotations

import math
from fractions import Fraction

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

SEED = 21


def _expected(pays):
    n = len(pays)
    m = Fraction(int(pays[:32].sum()), 32)
    ones = int(pays.sum())
    s1 = ones - n * m
    s2 = ones * (1 - m) ** 2 + (n - ones) * m**2
    mean = float(s1) / n
    m2 = float(s2 - s1 * Fraction(mean))
    return float(m) + mean, math.sqrt(m2 / ((n - 1.0) * n))


def test_digital_against_ieee_operations(engine, orc):
    vol, time, top = .2, 1.0, 9984
    threshold = .5 * vol * math.sqrt(time)  # S_T > S_0 without rates
    z = np.array([orc.orc_normal_variate(SEED, p, 0) for p in range(top)])
    assert np.abs(z - threshold).min() > 1e-12
    pays = z > threshold
    sizes = [64, 96, 160, 224, 352, 480, 1000, 1120, 3040, 4000, 5152, 7008, 9000, top]
    c = np.zeros(len(sizes), dtype=G.CONTRACT_DTYPE)
    c["product"], c["spot"], c["strike"], c["vol"], c["time"] = G.DIGITAL, 100.0, 100.0, vol, time
    c["cash_amount"], c["monitoring_points"], c["seed"] = 1.0, 1, SEED
    c["path_count"] = sizes
    batch = engine.price_batch(c, "fp64")
    for i, n in enumerate(sizes):  # n is a multiple of 8: a part unit has 8, 16 or 32 paths
        want = _expected(pays[:n])
        for r in (batch[i], engine.price_batch(c[i:i + 1], "fp64")[0]):
            assert (float(r["price"]), float(r["standard_error"])) == want, n
