"""FP32 items of 256 to 4096 paths (csrc/context.cpp, convert_contract) at their edges: a
contract alone against the same contract in a batch (equal bytes), the Greeks' price against
the pricer's (equal bits), and FP32 against FP64 on the same draws.

Bar for the last: a quarter of a standard error, and 2e-5 of the spot where few paths or a
mathematically small standard error leave only FP32 rounding of the path.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

PATHS = (1, 127, 128, 129, 255, 256, 257, 511, 513, 4095, 4097, 65536, 65537, 131073, 262145, 1048575, 1048577)
STEPS = (1, 31, 32, 64, 128, 252, 300)
KINDS = {
    "asian": dict(product=G.ASIAN),
    "asian_antithetic_cv": dict(product=G.ASIAN, antithetic=1, control_variate=1),
    "barrier_bridge": dict(product=G.BARRIER, barrier=130.0, direction=0, knock=1, brownian_bridge=1),
    "lookback": dict(product=G.LOOKBACK, type=1, strike_style=1),
    "digital": dict(product=G.DIGITAL, cash_amount=1.0),
}


@pytest.mark.parametrize("kind", KINDS)
def test_items(engine, kind):
    sizes = [(p, n) for p in PATHS for n in STEPS if p * n < 4e7]
    c = np.zeros(len(sizes), dtype=G.CONTRACT_DTYPE)
    for name, v in {**dict(spot=100.0, strike=101.0, rate=.02, vol=.2, time=1.0, seed=3), **KINDS[kind]}.items():
        c[name] = v
    c["path_count"], c["monitoring_points"] = np.array(sizes).T
    got, ref = engine.price_batch(c, "fp32"), engine.price_batch(c, "fp64")
    assert (got["path_count"] == c["path_count"]).all()
    bar = np.maximum(0.25 * ref["standard_error"], 2e-3)
    assert (np.abs(got["price"] - ref["price"]) <= bar).all()
    for i in range(0, len(sizes), 5):
        assert engine.price_batch(c[i:i + 1], "fp32").tobytes() == got[i:i + 1].tobytes(), sizes[i]
    if kind in ("asian", "lookback", "digital"):
        g = engine.greeks_batch(c, 1e-2, 1e-2, "fp32")
        assert (g["price"][:, 0] == got["price"]).all()
