"""FP32 pricing around the Philox step tables' sizes (256 steps per CTA in the
pricer, 32 per warp in the sensitivities) and at ragged path counts.

The two kernels lay their tables out differently and reduce the same samples in
the same tree, so their prices agree bit for bit; FP64 pricing on the same draws
(other tables, other arithmetic) agrees within a quarter of a standard error,
the FP32 paths' bar.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRODUCTS = {"asian": dict(product=2), "asian_geo_floating": dict(product=2, average_style=1, strike_style=1),
            "barrier": dict(product=3, barrier=80.0, direction=1, knock=1, type=1), "lookback": dict(product=4)}


def _contracts(G, extra, steps, paths):
    c = G.contracts(len(steps) * len(paths))
    c["spot"], c["strike"], c["rate"], c["vol"], c["time"] = 100.0, 98.0, 0.02, 0.3, 1.0
    for k, v in extra.items():
        c[k] = v
    for i, (n, p) in enumerate((n, p) for n in steps for p in paths):
        c["monitoring_points"][i], c["path_count"][i], c["seed"][i] = n, p, 500 + i
    return c


@pytest.mark.parametrize("name", PRODUCTS)
def test_step_tables_and_ragged_counts(engine, gpu_lib, name):
    c = _contracts(gpu_lib, PRODUCTS[name], (1, 31, 32, 33, 255, 256, 257, 600), (1, 127, 129, 4097))
    price = engine.price_batch(c, "fp32")
    greeks = engine.greeks_batch(c, 1e-3, 1e-3, "fp32")
    assert (price["path_count"] == c["path_count"]).all()
    assert (greeks["price"][:, 0] == price["price"]).all()
    assert (greeks["price"][:, 1] == price["standard_error"]).all()
    ref = engine.price_batch(c, "fp64")
    many = c["path_count"] > 100
    # a payoff is a difference of FP32 values near 100 (2^-23 relative): a floating strike over
    # one date is that rounding alone, on both sides
    bar = 0.25 * ref["standard_error"] + 100.0 * 2.0**-23
    assert (np.abs(price["price"] - ref["price"]) <= bar)[many].all()


@pytest.mark.parametrize("options", [dict(antithetic=1), dict(antithetic=1, brownian_bridge=1), dict(brownian_bridge=1)])
def test_options_past_the_table(engine, gpu_lib, options):
    extra = {**PRODUCTS["barrier"], **options}
    c = _contracts(gpu_lib, extra, (256, 257, 520), (129, 4097))
    price, ref = engine.price_batch(c, "fp32"), engine.price_batch(c, "fp64")
    assert (price["path_count"] == c["path_count"]).all()
    assert (np.abs(price["price"] - ref["price"]) <= 0.25 * ref["standard_error"]).all()
