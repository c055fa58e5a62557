"""FP64 likelihood-ratio and pathwise sensitivities at volatilities down to 1e-10 against the
oracle on identical draws.

The estimators hold the draws' own running sum (divided by the volatility, or times the square
root of a date's length), so their accuracy must not depend on how much of the log-spot the draws
make up.  Bar: 1e-11 of the estimate or of its standard error, the larger one (the draws agree to
3e-16, a path's product of 52 to 252 growth factors and sums of as many draws to 3e-14).
"""
from __future__ import annotations

import pytest

import mcd_gpu as G  # noqa: F401  (the engine fixture's library)

pytestmark = pytest.mark.gpu

PATHS, SEED = 4000, 17
VOLS = (1e-2, 1e-5, 1e-8, 1e-10)


def _check(got, want, names):
    for name in names:
        g, w = getattr(got, name), getattr(want, name)
        bar = 1e-11 * max(abs(w.value), w.standard_error)
        assert abs(g.value - w.value) <= bar, (name, g.value, w.value, w.standard_error)
        assert abs(g.standard_error - w.standard_error) <= bar, (name, g.standard_error, w.standard_error)


@pytest.mark.parametrize("dates", [52, 252])
@pytest.mark.parametrize("vol", VOLS)
def test_likelihood_ratio_barrier(engine, orc, vol, dates):
    args = (100.0, 110.0, 60.0, .03, .01, vol, 1.0, 1, 1, 1, 0.0, dates, PATHS, SEED)
    got = engine.likelihood_ratio_barrier(*args, precision="fp64")
    _check(got, orc.orc_lr_barrier(*args), ("delta", "gamma", "vega", "rho"))


@pytest.mark.parametrize("style", [(0, 0), (0, 1), (1, 0), (1, 1)])  # strike, average
@pytest.mark.parametrize("vol", VOLS)
def test_pathwise_asian(engine, orc, vol, style):
    args = (100.0, 90.0, .03, .01, vol, 1.0, 0, *style, 52, PATHS, SEED)
    got = engine.pathwise_asian(*args, precision="fp64")
    _check(got, orc.orc_pathwise_asian(*args), ("delta", "vega", "rho"))
