"""FP64 sensitivities where a bumped state is outside the fixed-point range and the contract itself
is not: the price output is the pricer's, byte for byte, as everywhere, and the finite differences
are central differences of the stepped states.

vol sqrt(T) = 5: a bump of 90 % takes it past 8 (stepped in FP64), one of 50 % does not.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

VARIANTS = [dict(product=G.EUROPEAN), dict(product=G.EUROPEAN, type=1), dict(product=G.DIGITAL),
            dict(product=G.DIGITAL, type=1, digital_style=1), dict(product=G.ASIAN),
            dict(product=G.ASIAN, average_style=1, type=1), dict(product=G.ASIAN, strike_style=1),
            dict(product=G.BARRIER, barrier=400.0, knock=1), dict(product=G.BARRIER, barrier=20.0, direction=1, type=1),
            dict(product=G.LOOKBACK), dict(product=G.LOOKBACK, strike_style=1, type=1)]


def _book(paths):
    c = np.zeros(len(VARIANTS), dtype=G.CONTRACT_DTYPE)
    for i, fields in enumerate(VARIANTS):
        for name, x in dict(spot=100.0, strike=90.0, rate=.03, carry_yield=.01, vol=2.5, time=4.0, cash_amount=1.0,
                            monitoring_points=40, path_count=paths, seed=3 + i, **fields).items():
            c[name][i] = x
    return c


@pytest.mark.parametrize("bump", [.5, .9])
@pytest.mark.parametrize("paths", [33, 3000])
def test_price_is_the_pricers(engine, paths, bump):
    c = _book(paths)
    p, g = engine.price_batch(c, "fp64"), engine.greeks_batch(c, .01, bump, "fp64")
    assert g["price"][:, 0].tobytes() == p["price"].tobytes()
    assert g["price"][:, 1].tobytes() == p["standard_error"].tobytes()


def test_vega_is_a_central_difference(engine):
    c = _book(3000)
    up, down = c.copy(), c.copy()
    up["vol"] = c["vol"] + .9 * c["vol"]
    down["vol"] = c["vol"] - .9 * c["vol"]
    g = engine.greeks_batch(c, .01, .9, "fp64")["fd_vega"][:, 0]
    a, b = engine.price_batch(up, "fp64")["price"], engine.price_batch(down, "fp64")["price"]
    want = (a - b) / (2 * .9 * c["vol"])
    assert (np.abs(g - want) <= 1e-12 * (np.abs(a) + np.abs(b))).all(), (g, want)
