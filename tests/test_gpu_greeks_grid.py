"""FP32 sensitivities at the edges of the grid's rule (CTAs per SM by the batch's items: one item
more than 1, 2, 4 and 8 CTAs on every SM hold): the bytes of a grid of eight CTAs per SM.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("times", [1, 2, 4, 8])
@pytest.mark.parametrize("more", [0, 1])
def test_same_bytes_on_another_grid(engine, times, more):
    items = times * torch.cuda.get_device_properties(0).multi_processor_count + more
    c = G.contracts(items)  # contracts of one date and at most 4096 paths are one item each
    c["product"] = np.arange(items) % 2 * G.LOOKBACK
    c["spot"] = c["strike"] = 100.0
    c["rate"], c["vol"], c["time"], c["monitoring_points"] = .03, .25, 1.0, 1
    c["path_count"] = 100 + np.arange(items) % 300
    c["seed"] = np.arange(items)
    want = engine.greeks_batch(c, precision="fp32").tobytes()
    with G.Engine(0) as e:
        e.set_greeks_launch_shape("fp32", 3, 8)
        assert e.greeks_batch(c, precision="fp32").tobytes() == want
