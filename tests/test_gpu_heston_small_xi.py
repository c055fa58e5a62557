"""FP64 Heston where the variance hardly diffuses (psi far below 2^-13 at every step): prices against
the same scheme in extended precision on the same draws.

The log-spot takes rho / xi times what the variance moves, so a relative rounding of the variance
that repeats at every step is multiplied by hundreds.  The extended values (numpy's longdouble, 64
bits of significand or more) are given the step's exp(-kappa dt) in FP64, as both forms use it.
Bar: 3e-13 of the price, ten times what the present operations err by on these sets in quadruple
precision (at most 2.7e-14); the reference's own order of operations errs by 6e-13 to 2e-12.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

X = np.longdouble
PATHS, SEED, SPOT, RATE = 300, 77, 100.0, .02
SETS = [  # v0, kappa, theta, xi, rho, time, dates
    (.112, 4.03, .0137, .001337, .2987, .0926, 252),
    (.112, 4.03, .0137, .001337, .2987, .0926, 50),
    (.04, 1.5, .04, .01, -.7, 1.0, 252),
    (.04, 1.5, .04, .001, -.7, 1.0, 252),
    (.3, .002, .2, .002, .5, 2.0, 100),
]


def _draws(orc, dates):
    z = np.array([[orc.orc_normal_variate(SEED, p, d) for d in range(dates)] for p in range(PATHS)])
    u = np.array([[orc.orc_uniform_variate(SEED, p, d) for d in range(dates)] for p in range(PATHS)])
    return z.astype(X), np.array([orc.orc_inv_normal_cdf(x) for x in u.ravel()]).reshape(u.shape).astype(X)


@pytest.mark.parametrize("row", SETS)
def test_against_extended_precision(engine, orc, row):
    dates = row[6]
    zs, zv = _draws(orc, dates)
    e = X(np.exp(-row[1] * (row[5] / dates)))
    v0, kappa, theta, xi, rho, time = (X(x) for x in row[:6])
    dt = time / dates
    k1 = dt / 2 * (kappa * rho / xi - X(.5)) - rho / xi
    k2, k3 = k1 + 2 * rho / xi, dt / 2 * (1 - rho * rho)
    v, x = np.full(PATHS, v0), np.full(PATHS, np.log(X(SPOT)))
    for d in range(dates):
        m = theta + (v - theta) * e
        psi = (v * xi * xi * e / kappa * (1 - e) + theta * xi * xi / (2 * kappa) * (1 - e) ** 2) / m**2
        assert psi.max() < 2.0**-13
        h = 2 / psi
        b2 = h - 1 + np.sqrt(h) * np.sqrt(h - 1)
        n = m / (1 + b2) * (np.sqrt(b2) + zv[:, d]) ** 2
        x = x + X(RATE) * dt - rho * kappa * theta * dt / xi + k1 * v + k2 * n + np.sqrt(k3 * (v + n)) * zs[:, d]
        v = n
    strikes = np.array([90.0, 100.0, 105.0])
    want = np.array([float((np.maximum(np.exp(x) - X(k), 0)).mean() * np.exp(-X(RATE) * time)) for k in strikes])
    s = np.zeros(1, dtype=G.HESTON_DTYPE)
    for name, value in dict(spot=SPOT, rate=RATE, v0=row[0], kappa=row[1], theta=row[2], xi=row[3], rho=row[4],
                            time=row[5]).items():
        s[name] = value
    got = engine.heston_qe_batch(s, strikes, 0, dates, PATHS, SEED, "fp64")["price"][0]
    assert (np.abs(got - want) <= 3e-13 * want).all(), (got / want - 1)
