"""FP64 batches of many small units on a device with little memory left: their partials are taken
in smaller ranges of contracts, and the results are those of a device with room.

A child process fills the device up to 64 MB by plain allocations after warming the kernels up.
In one piece the partials would take 118 MB (prices), 151 MB (sensitivities) and 403 MB (Heston).
"""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C, sys
sys.path.insert(0, %r)
import numpy as np
import mcd_gpu as G

runtime = C.CDLL("libcudart.so.13")
runtime.cudaMalloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
runtime.cudaFree.argtypes = [C.c_void_p]
LEFT = 64 << 20

def free():
    a, b = C.c_size_t(), C.c_size_t()
    assert runtime.cudaMemGetInfo(C.byref(a), C.byref(b)) == 0
    return a.value

def fill():
    held, size = [], 1 << 38
    while size >= 2 << 20:
        p = C.c_void_p()
        if free() - size > LEFT and runtime.cudaMalloc(C.byref(p), size) == 0:
            held.append(p)
        else:
            runtime.cudaGetLastError()
            size >>= 1
    return held

def contracts(n, paths):
    c = G.contracts(n)
    c["spot"] = c["strike"] = 100.0
    c["rate"], c["vol"], c["time"], c["monitoring_points"] = .03, .25, 1.0, 1
    c["path_count"] = paths
    c["seed"] = np.arange(n)
    return c

def sets(n):
    s = np.zeros(n, dtype=G.HESTON_DTYPE)
    for k, v in dict(spot=100.0, rate=.03, kappa=1.5, theta=.04, xi=.5, rho=-.6, v0=.04, time=1.0).items():
        s[k] = v
    s["theta"] += .0001 * np.arange(n)
    return s

strikes = np.linspace(80.0, 120.0, 64)
CASES = {
    "prices": lambda e, k: e.price_batch(contracts(k and 1200 or 3, 131071), "fp64"),
    "sensitivities": lambda e, k: e.greeks_batch(contracts(k and 128 or 3, 131071), 1e-4, 1e-4, "fp64"),
    "heston": lambda e, k: e.heston_qe_batch(sets(k and 64 or 1), strikes, 0, 2, 131071, 5, "fp64"),
}
for name, call in CASES.items():
    with G.Engine(0) as e:
        want = call(e, True).tobytes()
    with G.Engine(0) as e:
        call(e, False)
        held = fill()
        assert LEFT // 4 < free() < 2 * LEFT, free()
        got = call(e, True).tobytes()
        for p in held:
            assert runtime.cudaFree(p) == 0
    assert got == want, name
print("same")
"""


def test_batches_in_ranges_that_fit():
    package = os.path.dirname(os.path.abspath(G.__file__))
    r = subprocess.run([sys.executable, "-c", CHILD % package], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == "same"
