"""Heston FP64 at the edges of its units and parameter ranges against the oracle,
and the FP32 kernel around its 256-step table.

Bars: FP64 prices 1e-12 relative on identical draws (the QE step's regrouping
rounds as often as the reference's form), and 1e-12 of one hundredth of the spot
where a few paths' payoffs nearly cancel; standard errors 1e-10; FP32 within a
quarter of a standard error of FP64.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# spot, rate, yield, v0, kappa, theta, xi, rho, time
SETS = {
    "feller_violated": [100.0, .03, 0.0, .01, .5, .02, 1.0, -.9, 1.0],  # the exponential branch often
    "quiet": [100.0, .03, .01, .06, 3.0, .06, .2, -.3, 1.0],            # psi of a few 1e-3
    "perfect_correlation": [100.0, .01, 0.0, .04, 1.0, .04, .3, -1.0, 2.0],
    "from_zero": [100.0, .02, 0.0, 0.0, 2.0, .05, .6, -.5, .5],
}


@pytest.mark.parametrize("name", SETS)
@pytest.mark.parametrize("paths", [1, 33, 131072 + 40])
def test_fp64_units_and_parameter_corners(engine, orc, name, paths):
    hp, steps, seed = O.HestonParams(*SETS[name]), 6, 91
    strikes = np.array([90.0, 100.0, 115.0])
    one = engine.heston_qe_european(SETS[name], 100.0, 0, steps, paths, seed, precision="fp64")
    many = engine.heston_qe_batch([SETS[name]], strikes, 0, steps, paths, seed, "fp64")
    for got, k in [(one, 100.0)] + [(many[0, j], k) for j, k in enumerate(strikes)]:
        price = got.price if hasattr(got, "price") and not isinstance(got, np.void) else got["price"]
        se = got.standard_error if not isinstance(got, np.void) else got["standard_error"]
        ref = orc.orc_heston_qe_european(C.byref(hp), k, 0, steps, paths, seed)
        assert abs(price - ref.price) <= 1e-12 * max(abs(ref.price), 1.0), (k, price, ref.price)
        assert abs(se - ref.standard_error) <= 1e-10 * max(ref.standard_error, 1e-2)


@pytest.mark.parametrize("steps", [255, 256, 257, 520])
def test_fp32_around_the_step_table(engine, steps):
    sets, strikes = [SETS["feller_violated"], SETS["quiet"]], np.array([85.0, 100.0, 120.0])
    for paths in (129, 4097):
        a = engine.heston_qe_batch(sets, strikes, 1, steps, paths, 7, "fp32")
        b = engine.heston_qe_batch(sets, strikes, 1, steps, paths, 7, "fp64")
        assert (a["path_count"] == paths).all()
        assert (np.abs(a["price"] - b["price"]) <= 0.25 * b["standard_error"]).all()
