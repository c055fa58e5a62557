"""FP64 Longstaff-Schwartz batches that walk their dates in one launch (all chunks resident)
against the form of one launch per date, bit for bit, and against the oracle.

A contract is priced alone (one launch up to 304 chunks of 1024 paths) and in a batch with a
contract of 600 chunks, which takes one launch per date.  Bars: equal bytes; 1e-12 relative of
the oracle's price on identical draws.
"""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

ROWS = [  # spot, strike, vol, type, dates, paths
    (40.0, 40.0, .2, 1, 1, 5000),               # no regression
    (40.0, 40.0, .2, 1, 2, 1),                  # one path
    (40.0, 40.0, .3, 0, 3, 33),
    (36.0, 40.0, .4, 1, 12, 1023),
    (80.0, 40.0, .2, 1, 9, 1025),               # dates without four paths in the money
    (10.0, 40.0, .2, 1, 5, 4096),               # every path in the money
    (40.0, 40.0, .25, 1, 33, 32 * 1024),        # one fold group
    (44.0, 40.0, .3, 0, 7, 32 * 1024 + 1),      # a second one, of one path
    (40.0, 40.0, .2, 1, 4, 304 * 1024),         # as many chunks as are resident on 152 SMs
    (40.0, 40.0, .2, 1, 4, 304 * 1024 + 1),
]


def _record(rows):
    arr = np.zeros(len(rows), dtype=G.LSM_CONTRACT_DTYPE)
    for i, (s, k, v, ty, n, paths) in enumerate(rows):
        for name, x in dict(spot=s, strike=k, rate=.06, carry_yield=.01, vol=v, time=1.0, type=ty,
                            monitoring_points=n, path_count=paths, seed=7 + i).items():
            arr[i][name] = x
    return arr


def test_one_launch_has_the_bits_of_a_launch_per_date(engine):
    arr = _record(ROWS + [(40.0, 40.0, .2, 1, 6, 600 * 1024)])
    batch = engine.lsm_batch(arr, "fp64")
    for i in range(len(ROWS)):
        assert engine.lsm_batch(arr[i:i + 1], "fp64").tobytes() == batch[i:i + 1].tobytes(), ROWS[i]
    some = engine.lsm_batch(arr[:8], "fp64")  # several contracts in one launch
    assert some.tobytes() == batch[:8].tobytes()


def test_threads_take_turns(engine):
    """One cooperative launch at a time: the other threads' calls go date by date, same bytes."""
    arr = _record([(40.0, 40.0, .2, 1, 20, 200 * 1024)])
    want, bad = engine.lsm_batch(arr, "fp64").tobytes(), []

    def work():
        e = G.Engine(0)
        bad.extend(1 for _ in range(6) if e.lsm_batch(arr, "fp64").tobytes() != want)

    threads = [threading.Thread(target=work) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("groups", [16, 17])  # group sums added in order, or by the warp's tree
def test_group_folds_against_the_oracle(engine, orc, groups):
    paths, n = groups * 32 * 1024 - 5, 3
    got = engine.monte_carlo_lsm_american(38.0, 40.0, .06, .01, .3, 1.0, 1, n, paths, 3, precision="fp64")
    co, has, ex = (C.c_double * (4 * (n + 1)))(), (C.c_uint8 * (n + 1))(), C.c_int32()
    ref = orc.orc_lsm_american(38.0, 40.0, .06, .01, .3, 1.0, 1, n, paths, 3, co, has, C.byref(ex))
    assert abs(got.price - ref.price) <= 1e-12 * abs(ref.price), (got.price, ref.price)
