"""A program that resets the device between two uses of the library gets the same prices after
the reset: nothing that the process remembers of the device's memory (the fixed-point tables,
the scratch of the allocation-free entry point) outlives its CUDA context.

The library runs in a child process of its own, without torch, whose context no other test
shares; every context of the library is closed before the reset.
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

c = G.contracts(3)
c["product"] = [G.EUROPEAN, G.ASIAN, G.BARRIER]
c["spot"] = c["strike"] = 100.0
c["barrier"] = 130.0
c["rate"], c["vol"], c["time"], c["monitoring_points"], c["path_count"], c["seed"] = .03, .25, 1.0, 12, 5000, 3
runtime = C.CDLL("libcudart.so.13")

def prices():
    out = []
    with G.Engine(0) as e:
        for precision in ("fp64", "fp32"):
            out.append(e.price_batch(c, precision).tobytes())
        out.append(e.price_batch(c[:1], "fp64").tobytes())
    for precision in (0, 1):
        r = np.zeros(3, dtype=G.RESULT_DTYPE)
        msg = C.create_string_buffer(256)
        f = G.lib().mcd_price_batch_static
        f.argtypes = [C.c_void_p, C.c_size_t, C.c_int, C.c_void_p, C.c_void_p, C.c_char_p, C.c_size_t]
        assert f(c.ctypes.data, 3, precision, r.ctypes.data, None, msg, 256) == 0, msg.value
        out.append(r.tobytes())
    return out

first = prices()
for _ in range(2):
    assert runtime.cudaDeviceReset() == 0
    assert prices() == first
print("same")
"""


def test_prices_after_a_device_reset():
    package = os.path.dirname(os.path.abspath(G.__file__))
    r = subprocess.run([sys.executable, "-c", CHILD % package], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == "same"
