"""The autotuners time each launch shape that there is once: FP64 has three path kernels (512, 768
and 1024 threads) and one of the sensitivities, one CTA per SM each.  A shape is run three times
and every run is one timed launch.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu


def test_launches_of_the_autotuners(gpu_lib):
    c = G.contracts(4)
    c["product"] = [G.EUROPEAN, G.ASIAN, G.BARRIER, G.LOOKBACK]
    c["spot"] = c["strike"] = 100.0
    c["barrier"] = 130.0
    c["rate"], c["vol"], c["time"], c["monitoring_points"], c["path_count"] = .03, .25, 1.0, 12, 20_000
    c["seed"] = np.arange(4)
    with G.Engine(0) as e:
        want = e.price_batch(c, "fp64").tobytes()
        e.kernel_timing(reset=True)
        variant, ctas, ms = e.autotune(c, "fp64")
        assert e.kernel_timing(reset=True)[1] == 9
        assert variant in (0, 1, 4) and ctas == 1 and ms > 0.0
        assert e.price_batch(c, "fp64").tobytes() == want
        e.kernel_timing(reset=True)
        assert e.greeks_autotune(c, precision="fp64")[1] == 1
        assert e.kernel_timing(reset=True)[1] == 3
        for tune, least in ((e.autotune, 5), (e.greeks_autotune, 4)):  # FP32: a kernel per variant
            tune(c, precision="fp32")
            assert e.kernel_timing(reset=True)[1] >= 3 * least
