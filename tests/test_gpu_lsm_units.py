"""Longstaff-Schwartz in FP64 at the edges of its units and range, against the
oracle, and the frozen replay against the fit.

Bars: prices 1e-12 relative of the oracle (identical draws; every exercise
decision coincides unless exercise and continuation agree to 1e-14), standard
errors 1e-10, the replayed base price bit for bit.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _fit(engine, orc, args):
    s, k, r, q, v, t, ty, n, paths, seed = args
    res, co, has = engine.monte_carlo_lsm_american(s, k, r, q, v, t, ty, n, paths, seed, precision="fp64", policy=True)
    rc, rh, ex = (C.c_double * (4 * (n + 1)))(), (C.c_uint8 * (n + 1))(), C.c_int32()
    ref = orc.orc_lsm_american(s, k, r, q, v, t, ty, n, paths, seed, rc, rh, C.byref(ex))
    return res, co, has, ref


CASES = [
    (40.0, 40.0, .06, 0.0, .2, 1.0, 1, 33, 1024, 5),      # past one step table
    (36.0, 40.0, .06, 0.0, .4, 2.0, 1, 10, 1023, 6),      # one path short of a chunk
    (44.0, 40.0, .03, .05, .3, 1.0, 0, 12, 5 * 1024 + 1, 7),  # a call, a chunk of one path
    (40.0, 40.0, .05, 0.0, 3.0, 4.0, 1, 6, 3000, 8),      # vol sqrt(T) > 4: stepped without fixed point
    (40.0, 40.0, .06, 0.0, .25, 1.0, 1, 8, 300 * 1024 + 40, 9),  # more than one fold group
]


@pytest.mark.parametrize("args", CASES)
def test_fit_against_oracle_and_replay(engine, orc, args):
    res, co, has, ref = _fit(engine, orc, args)
    assert abs(res.price - ref.price) <= 1e-12 * abs(ref.price), (res.price, ref.price)
    assert abs(res.standard_error - ref.standard_error) <= 1e-10 * ref.standard_error
    s, k, r, q, v, t, ty, n, paths, seed = args
    replay = engine.reprice_against_frozen_policy(s, k, r, q, v, t, ty, n, paths, seed, co, has,
                                                  bool(res.exercise_at_inception), "fp64")
    assert replay == res.price
    g = engine.lsm_frozen_greeks(s, k, r, q, v, t, ty, n, paths, seed, co, has, bool(res.exercise_at_inception),
                                 precision="fp64")
    assert g["price"][0] == res.price


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("steps", [2, 251, 252, 253, 255, 256, 257, 300])
def test_fp32_forward_and_replay_around_the_tables(engine, steps, kind):
    """Stored FP32 paths past the 256-step table, and the replay's two kernels (up to 252
    dates each lane takes its own paths): the fitted price bit for bit."""
    args = (40.0, 40.0, .06, .02, .3, 1.0, kind, steps, 3000, 11)
    res, co, has = engine.monte_carlo_lsm_american(*args, precision="fp32", policy=True)
    assert engine.reprice_against_frozen_policy(*args, co, has, bool(res.exercise_at_inception), "fp32") == res.price
    g = engine.lsm_frozen_greeks(*args, co, has, bool(res.exercise_at_inception), 0.4, 0.003, precision="fp32")
    assert g["price"][0] == res.price
    up = (40.4, *args[1:])  # a bumped scenario is the single replay at the bumped spot
    assert g["scenario"][0] == engine.reprice_against_frozen_policy(*up, co, has, False, "fp32")
