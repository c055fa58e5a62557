"""Contracts whose samples overflow FP64 or FP32 (infinity times a discount of zero, infinity less
infinity): price and standard error are both NaN, as sums of such samples are.  A standard error
of zero would call the price exact.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

CASES = {
    # S_T = exp(1000) overflows, the discount exp(-1000) is zero
    "discount": (dict(product=G.EUROPEAN, spot=100.0, strike=100.0, rate=500.0, time=2.0, vol=.2), ("fp64", "fp32")),
    # spot and average overflow on some paths: their difference is not a number
    "difference_call": (dict(product=G.ASIAN, strike_style=1, spot=1e308, strike=1e308, time=1.0, vol=2.0), ("fp64",)),
    "difference_put": (dict(product=G.ASIAN, strike_style=1, type=1, spot=1e308, strike=1e308, time=1.0, vol=2.0),
                       ("fp64",)),
}


def _contract(fields, paths):
    c = np.zeros(1, dtype=G.CONTRACT_DTYPE)
    for name, x in dict(monitoring_points=12, path_count=paths, seed=5, **fields).items():
        c[name] = x
    return c


@pytest.mark.parametrize("paths", [300, 9000])  # FP64 units of 32 paths, FP32 items of 4096
@pytest.mark.parametrize("case", CASES)
def test_batches(engine, case, paths):
    fields, precisions = CASES[case]
    for precision in precisions:
        for c in (_contract(fields, paths), np.repeat(_contract(fields, paths), 2)):
            r = engine.price_batch(c, precision)
            assert np.isnan(r["price"]).all() and np.isnan(r["standard_error"]).all(), (precision, r)


def test_sensitivities(engine):
    r = engine.greeks_batch(_contract(CASES["discount"][0], 5000), 1e-4, 1e-4, "fp64")
    assert np.isnan(r["price"]).all(), r
