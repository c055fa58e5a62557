"""GPU checks of the FP32 Sobol kernel's four paths per thread and incremental Gray-code
rows (derivative-pricing_gb300/csrc/qmc.cu) at the edges of warps, CTAs and slabs.

Oracle: the FP64 kernel of the same paths (tied to the reference in test_gpu_qmc.py).
Bar per path, relative to the spot: quantile and bridge rounding through the volatility
(1e-6 each), the exponential (1e-6), and for averages the FP32 sum over n points (n 2^-25).
A path left out or taken twice moves the mean by about 10 / paths, above the bar at every
size here.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

PATHS = (1, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 255, 256, 257, 511, 512, 513, 4095, 4096, 4097, 4097 + 128, 12289)
STEPS = (1, 2, 3, 31, 32, 33, 255, 256)
PRODUCTS = (
    dict(product=G.EUROPEAN, type=0, strike=90.0),
    dict(product=G.ASIAN, type=0, strike=90.0, strike_style=0, average_style=0),
    dict(product=G.ASIAN, type=1, strike=110.0, strike_style=0, average_style=1),
    dict(product=G.BARRIER, type=0, strike=90.0, barrier=1e6, direction=0, knock=0),  # out, never hit
    dict(product=G.LOOKBACK, type=1, strike=110.0, strike_style=0),
    dict(product=G.LOOKBACK, type=0, strike=100.0, strike_style=1),
)


@pytest.mark.parametrize("kw", PRODUCTS, ids=lambda k: f"{k['product']}-{k['type']}")
def test_rows_match_fp64(engine, kw):
    sizes = [(p, n) for p in PATHS for n in STEPS]
    arr = np.zeros(len(sizes), dtype=G.CONTRACT_DTYPE)
    for i, (p, n) in enumerate(sizes):
        row = dict(spot=100.0, rate=0.03, carry_yield=0.01, vol=0.2, time=1.0, seed=5, path_count=p,
                   monitoring_points=n)
        row.update(kw)
        for k, v in row.items():
            arr[i][k] = v
    ref = engine.qmc_batch(arr, precision="fp64")
    got = engine.qmc_batch(arr, precision="fp32")
    for i, (p, n) in enumerate(sizes):
        bar = 100.0 * (3e-6 + n * 2.0**-25)
        assert abs(got["price"][i] - ref["price"][i]) <= bar, (p, n, got["price"][i], ref["price"][i])
        one = engine.qmc_batch(arr[i:i + 1], precision="fp32")
        assert one.tobytes() == got[i:i + 1].tobytes(), (p, n)
