"""FP32 paths of contracts quoted below 1.2e-38, FP32's smallest normal number: spots, strikes and
payoffs are subnormal, and count.

Against the FP64 engine on the same draws.  Bar: 1e-4 of the price (a spot of 5e-39 has units of
1.4e-45, 3e-7 of it, and a payoff a tenth of that spot four roundings of such units; the FP32
paths themselves are good to 1e-5); American puts, whose regression sums hold products of such
payoffs, 1e-3.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

S = 5e-39
VARIANTS = [dict(product=G.EUROPEAN), dict(product=G.EUROPEAN, type=1, antithetic=1),
            dict(product=G.DIGITAL, digital_style=1), dict(product=G.DIGITAL, cash_amount=S),
            dict(product=G.ASIAN), dict(product=G.ASIAN, average_style=1, type=1), dict(product=G.ASIAN, strike_style=1),
            dict(product=G.BARRIER, barrier=1.3 * S, knock=1, rebate=.1 * S),
            dict(product=G.BARRIER, barrier=.8 * S, direction=1, type=1, brownian_bridge=1),
            dict(product=G.LOOKBACK), dict(product=G.LOOKBACK, strike_style=1, type=1)]


def _book(variants):
    c = np.zeros(len(variants), dtype=G.CONTRACT_DTYPE)
    for i, fields in enumerate(variants):
        for name, x in dict(spot=S, strike=S, rate=.03, carry_yield=.01, vol=.4, time=1.0, monitoring_points=12,
                            path_count=20_000, seed=3 + i, **fields).items():
            c[name][i] = x
    return c


def _close(got, want, rel):
    assert (want > 0.0).all() and (np.abs(got - want) <= rel * want).all(), (got, want)


def test_prices(engine):
    c = _book(VARIANTS)
    _close(engine.price_batch(c, "fp32")["price"], engine.price_batch(c, "fp64")["price"], 1e-4)


def test_sobol_prices(engine):
    c = _book([v for v in VARIANTS if not (v.get("antithetic") or v.get("brownian_bridge"))])
    _close(engine.qmc_batch(c, "fp32")["price"], engine.qmc_batch(c, "fp64")["price"], 1e-4)


def test_sensitivities_price(engine):
    c = _book([v for v in VARIANTS if not (v.get("antithetic") or v.get("brownian_bridge"))])
    got, want = (engine.greeks_batch(c, 1e-3, 1e-3, p)["price"][:, 0] for p in ("fp32", "fp64"))
    _close(got, want, 1e-4)


def test_heston(engine):
    s = np.zeros(2, dtype=G.HESTON_DTYPE)
    for k, v in dict(spot=S, rate=.03, kappa=1.5, theta=.06, xi=.4, rho=-.5, v0=.05, time=1.0).items():
        s[k] = v
    got, want = (engine.heston_qe_batch(s, np.array([.9, 1.0, 1.1]) * S, 0, 12, 20_000, 5, p)["price"]
                 for p in ("fp32", "fp64"))
    _close(got, want, 1e-4)


def test_american_put(engine):
    c = np.zeros(2, dtype=G.LSM_CONTRACT_DTYPE)
    for k, v in dict(strike=S, rate=.06, vol=.3, time=1.0, type=1, monitoring_points=12, path_count=20_000,
                     seed=9).items():
        c[k] = v
    c["spot"] = [.95 * S, 1.05 * S]
    got, want = (engine.lsm_batch(c, p)["price"] for p in ("fp32", "fp64"))
    _close(got, want, 1e-3)
