"""FP64 pricing in fixed point at the edges of its dispatch, against the oracle
(the reference's algorithm) on identical draws: unit sizes (32 paths up to
131,071, doubling above), single-lane remainders, contracts outside the
fixed-point range, long and one-step paths, barriers no path can reach.

Bars: 1e-12 relative on prices and 1e-10 on standard errors, as for every FP64
price (the oracle's own rounding over the steps is about 1e-15 per path).
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _contract(G, kind, **kw):
    c = G.contracts(1)
    c["spot"], c["strike"], c["rate"], c["vol"], c["time"] = 100.0, 101.0, 0.03, 0.25, 1.5
    c["monitoring_points"], c["seed"], c["path_count"] = 7, 77, 1000
    product, extra = {
        "european": (G.EUROPEAN, {}), "digital": (G.DIGITAL, {"digital_style": 1}),
        "asian": (G.ASIAN, {}), "asian_floating": (G.ASIAN, {"strike_style": 1, "type": 1}),
        "asian_geo": (G.ASIAN, {"average_style": 1}), "asian_cv": (G.ASIAN, {"control_variate": 1}),
        "barrier": (G.BARRIER, {"barrier": 85.0, "direction": 1, "knock": 1, "type": 1, "rebate": 0.5}),
        "bridge": (G.BARRIER, {"barrier": 120.0, "direction": 0, "knock": 0, "brownian_bridge": 1}),
        "lookback": (G.LOOKBACK, {"type": 1}), "lookback_floating": (G.LOOKBACK, {"strike_style": 1}),
    }[kind]
    c["product"] = product
    for k, v in {**extra, **kw}.items():
        c[k] = v
    return c


KINDS = ["european", "digital", "asian", "asian_floating", "asian_geo", "asian_cv", "barrier", "bridge", "lookback",
         "lookback_floating"]


def _check(engine, orc, c):
    got = engine.price_batch(c, "fp64")
    arr = (O.Contract * len(c))()
    for i, row in enumerate(c):
        for name in row.dtype.names:
            setattr(arr[i], name, row[name].item())
    want = (O.McResult * len(c))()
    orc.orc_price_batch(arr, len(c), 4, 8, want)
    for i in range(len(c)):
        assert got["path_count"][i] == want[i].path_count
        assert abs(got["price"][i] - want[i].price) <= 1e-12 * abs(want[i].price), (i, c[i], got[i], want[i].price)
        # samples round at 4 units of 1.1e-16 of the price: the standard error of equal samples
        # (the control variate of one date) is that rounding on both sides
        floor = 1e-15 * abs(want[i].price)
        assert abs(got["standard_error"][i] - want[i].standard_error) <= 1e-10 * want[i].standard_error + floor, i


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("antithetic", [0, 1])
def test_unit_edges(engine, gpu_lib, orc, kind, antithetic):
    counts = [31, 32, 33, 131071, 131072, 262144 + 65]
    c = np.concatenate([_contract(gpu_lib, kind, path_count=n, antithetic=antithetic, seed=n) for n in counts])
    _check(engine, orc, c)


@pytest.mark.parametrize("kind", KINDS)
def test_steps_and_range(engine, gpu_lib, orc, kind):
    rows = [_contract(gpu_lib, kind, monitoring_points=n, path_count=700) for n in (1, 31, 32, 33, 365)]
    # log2(S/S0) could pass 2^9 on some path: stepped without fixed point
    rows += [_contract(gpu_lib, kind, vol=4.0, time=9.0, path_count=300),
             _contract(gpu_lib, kind, rate=400.0, path_count=300)]
    if kind in ("barrier", "bridge"):
        rows += [_contract(gpu_lib, kind, barrier=b, path_count=300) for b in (1e12, 1e-12)]
    _check(engine, orc, np.concatenate(rows))


def test_constant_samples_have_no_standard_error(engine, gpu_lib):
    # every path pays the same: the shifted sums are exactly zero
    c = _contract(gpu_lib, "digital", strike=1e-9, digital_style=0, cash_amount=3.7, path_count=5000)
    r = engine.price_batch(c, "fp64")
    assert r["standard_error"][0] == 0.0
    assert abs(r["price"][0] - 3.7 * np.exp(-0.03 * 1.5)) < 1e-15 * 4


def test_static_entry_takes_several_launches_on_the_same_scratch(gpu_lib):
    # 70 contracts of 4096 units each: more than the 262,144 partials of the fixed scratch
    c = np.concatenate([_contract(gpu_lib, "european", path_count=131071, seed=i) for i in range(70)])
    with gpu_lib.Engine(0) as eng:
        want = eng.price_batch(c, "fp64")
    fn = gpu_lib.lib().mcd_price_batch_static
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p, C.c_size_t, C.c_int, C.c_void_p, C.c_void_p, C.c_char_p, C.c_size_t]
    out = np.zeros(len(c), dtype=gpu_lib.RESULT_DTYPE)
    msg = C.create_string_buffer(256)
    assert fn(c.ctypes.data, len(c), 0, out.ctypes.data, None, msg, len(msg)) == 0, msg.value.decode()
    assert out.tobytes() == want.tobytes()


@pytest.mark.parametrize("kind", ["european", "asian", "asian_geo", "barrier", "lookback_floating"])
def test_greeks_units_and_range(engine, gpu_lib, kind):
    """Price bit for bit the pricer's at unit edges; outside the fixed-point range the
    estimators still agree with the same contract's fixed-point ones in form."""
    c = np.concatenate([_contract(gpu_lib, kind, path_count=n) for n in (1, 33, 131072 + 64)])
    res, ref = engine.greeks_batch(c, 1e-3, 1e-3, "fp64"), engine.price_batch(c, "fp64")
    assert (res["price"][:, 0] == ref["price"]).all() and (res["price"][:, 1] == ref["standard_error"]).all()
    wide = _contract(gpu_lib, kind, vol=3.0, time=8.0, path_count=2000)  # vol sqrt(T) > 8: stepped in FP64
    r = engine.greeks_batch(wide, 1e-3, 1e-3, "fp64")[0]
    p = engine.price_batch(wide, "fp64")[0]
    assert abs(r["price"][0] - p["price"]) <= 1e-11 * abs(p["price"])
    up, dn = wide.copy(), wide.copy()
    up["spot"], dn["spot"] = 100.1, 99.9
    fd = (engine.price_batch(up, "fp64")["price"][0] - engine.price_batch(dn, "fp64")["price"][0]) / 0.2
    assert abs(r["fd_delta"][0] - fd) <= 1e-8 * abs(fd) + 1e-9
