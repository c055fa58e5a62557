"""One European or digital contract in FP64 (a single launch, csrc/gbm_paths64.cu) against the
same contract in a batch of two (path and merge kernels): equal bytes, at the edges of units and
of the range of path counts that takes the launch, and on repeated calls.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

PATHS = (0, 1, 31, 32, 33, 4095, 131071, 131072, 131072 + 65, 1024 * 4096, 1024 * 4096 + 1)
KINDS = {
    "call": dict(product=G.EUROPEAN),
    "put_antithetic": dict(product=G.EUROPEAN, type=1, antithetic=1),
    "cash": dict(product=G.DIGITAL, cash_amount=2.0),
    "asset_put": dict(product=G.DIGITAL, type=1, digital_style=1, antithetic=1),
    "wide": dict(product=G.EUROPEAN, vol=60.0, time=4.0),  # |log2 S| may pass 2^9: stepped in FP64
}


def _pair(paths, **kw):
    c = np.zeros(2, dtype=G.CONTRACT_DTYPE)
    base = dict(spot=100.0, strike=104.0, rate=.03, carry_yield=.01, vol=.25, time=1.5, cash_amount=1.0,
                monitoring_points=1, seed=9, path_count=paths)
    for name, v in {**base, **kw}.items():
        c[name] = v
    return c


@pytest.mark.parametrize("kind", KINDS)
def test_single_launch_has_the_batch_bits(engine, kind):
    for paths in PATHS if kind != "wide" else PATHS[:6]:
        c = _pair(paths, **KINDS[kind])
        both = engine.price_batch(c, "fp64")
        for _ in range(2):
            one = engine.price_batch(c[:1], "fp64")
            assert one.tobytes() == both[:1].tobytes(), (paths, one, both)


def test_engines_in_threads(engine):
    want = engine.price_batch(_pair(50_000), "fp64")[:1].tobytes()
    bad = []

    def work():
        e = G.Engine(0)
        for _ in range(50):
            if e.price_batch(_pair(50_000)[:1], "fp64").tobytes() != want:
                bad.append(1)

    threads = [threading.Thread(target=work) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
