"""FP64 Longstaff-Schwartz batches whose one-launch form does not come through go date by date:
when the CTAs' waits for one another run out (here after a single look each; the kernel reports
it and ends), and when the cooperative launch is refused (here by asking for more shared memory
than there is, which the runtime answers without a launch).  Same bytes as the one launch, and the
next ordinary call on the same context has them again.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu


def _puts(rows):
    c = np.zeros(len(rows), dtype=G.LSM_CONTRACT_DTYPE)
    for i, (dates, paths) in enumerate(rows):
        for name, x in dict(spot=38.0, strike=40.0, rate=.06, carry_yield=.01, vol=.3, time=1.0, type=1,
                            monitoring_points=dates, path_count=paths, seed=5 + i).items():
            c[i][name] = x
    return c


BATCHES = {"one": [(20, 200 * 1024)], "several": [(9, 60 * 1024 + 7), (20, 3000), (4, 33 * 1024), (12, 100 * 1024)]}


@pytest.fixture()
def own():
    e = G.Engine(0)
    yield e
    e.close()


def _limit(e, polls=0, shared=0):
    f = e._lib.mcd_test_lsm_chain
    f.argtypes = [C.c_void_p, C.c_uint32, C.c_size_t]
    assert f(e.handle, polls, shared) == 0


def _timed_launches(e, c):
    e.kernel_timing(reset=True)
    r = e.lsm_batch(c, "fp64").tobytes()
    return r, e.kernel_timing(reset=True)[1]


@pytest.mark.parametrize("batch", BATCHES)
def test_waits_that_run_out(own, batch):
    c = _puts(BATCHES[batch])
    want, launches = _timed_launches(own, c)
    assert launches == 1
    for _ in range(3):
        _limit(own, polls=1)
        got, launches = _timed_launches(own, c)
        assert got == want and launches == 2  # the launch that gave up, and the dates
        _limit(own)
        assert _timed_launches(own, c) == (want, 1)


@pytest.mark.parametrize("batch", BATCHES)
def test_refused_launch(own, batch):
    c = _puts(BATCHES[batch])
    want = own.lsm_batch(c, "fp64").tobytes()
    _limit(own, shared=1 << 30)
    assert own.lsm_batch(c, "fp64").tobytes() == want
    _limit(own)
    assert own.lsm_batch(c, "fp64").tobytes() == want


def test_policy_and_greeks_of_a_batch_that_went_date_by_date(own):
    c = _puts(BATCHES["several"])
    want = own.lsm_greeks_batch(c, .01, .01, "fp64").tobytes()
    for kw in (dict(polls=1), dict(shared=1 << 30)):
        _limit(own, **kw)
        assert own.lsm_greeks_batch(c, .01, .01, "fp64").tobytes() == want
