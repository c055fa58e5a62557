"""FP32 finite differences where a path's growth is below FP32's normal numbers (1.2e-38) and a bump
multiplies it by more than FP32 holds (volatility 4 over 12 years, bumped by 90 %): a subnormal
growth makes that a large number, a flushed one NaN.  (Paths below 1e-45, the least subnormal, have
always been NaN; the four paths here are above.)

Puts, against FP64 on the same draws: the bumped payoffs are the strike's or nothing, so the vegas
agree to FP32's rounding of a strike, 1e-5 of the price over the bump.  The price output is the
path engine's.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("product, dates", [(G.EUROPEAN, 100), (G.ASIAN, 1)])
def test_vega(engine, product, dates):
    c = np.zeros(1, dtype=G.CONTRACT_DTYPE)
    for name, x in dict(product=product, type=1, spot=327.6198173587761, strike=1295.6854740107456,
                        rate=0.6598509075704839, carry_yield=.01, vol=3.9754504351325264, time=12.228484916822675,
                        monitoring_points=dates, path_count=4, seed=2465507424629501706).items():
        c[name] = x
    got, want = (engine.greeks_batch(c, .5, .9, p)[0] for p in ("fp32", "fp64"))
    bar = 1e-5 * want["price"][0] / (.9 * float(c["vol"][0]))
    assert abs(got["fd_vega"][0] - want["fd_vega"][0]) <= bar, (got["fd_vega"], want["fd_vega"])
    assert got["price"][0] == engine.price_batch(c, "fp32")["price"][0]
