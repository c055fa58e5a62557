"""The integer square root, reciprocal and logarithm (csrc/fixed_root.hpp) against
40-digit values, compiled for the host, with the seeds moved by 2^-22.1 (root) and
2^-22 (reciprocal), more than the GPU's approximations err (2^-22.4 of the root's
seed, 2^-23 of the reciprocal's).

Bars, from the construction.  Root: the first Newton term leaves 2^-38.5 (bias and
seed 2^-19.4, squared, and their product with the seed's 2^-20.9), the second
multiplies that by the seed's error: 2^-59.4, and three truncations of 2^-64.
Reciprocal: the seed's error cubed, 2^-61.2 with the moves made here, and
truncations of 2^-63.
Logarithm: t^6/6 < 2^-62.5, three truncations of 2^-59 and half a unit per ln 2.
"""
from __future__ import annotations

import ctypes as C
import os
import random
import subprocess

import pytest

mp = pytest.importorskip("mpmath")

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "derivative-pricing_gb300", "csrc")
SOURCE = """
#include "fixed_tables.cpp"
#include "fixed_root.hpp"
using namespace mcdg;
extern "C" uint64_t root(uint64_t a, int32_t move) {
    return sqrt_from_seed(a, rsqrt_seed((uint32_t)(a >> 32)) + (uint32_t)move);
}
extern "C" uint64_t rcp(uint64_t m, int32_t move) {
    return rcp_from_seed(m, rcp_seed((uint32_t)(m >> 32)) + (uint32_t)move);
}
extern "C" uint64_t nlog(uint64_t m, int e) {
    const FixedTables& t = fixed_tables();
    const uint32_t i = log_index(m);
    return neg_log(m, e, t.log_c[i], t.log_l[i]);
}
extern "C" double root_double(double x) { return sqrt_int(x); }
extern "C" double rcp_double(double x) { return rcp_int(x); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("root")
    src, so = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++20", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, src, "-o", so],
                   check=True)
    L = C.CDLL(so)
    for name in ("root", "rcp"):
        getattr(L, name).restype, getattr(L, name).argtypes = C.c_uint64, [C.c_uint64, C.c_int32]
    L.nlog.restype, L.nlog.argtypes = C.c_uint64, [C.c_uint64, C.c_int]
    for name in ("root_double", "rcp_double"):
        getattr(L, name).restype, getattr(L, name).argtypes = C.c_double, [C.c_double]
    return L


def _fractions(rng, lo, hi):
    edge = [lo, lo + 1, hi - 1, hi - 2, (lo + hi) // 2] + [lo + 2**k for k in range(0, 62, 3)]
    edge += [hi - 2**k for k in range(0, 62, 3)]
    return edge + [rng.randrange(lo, hi) for _ in range(4000)]


# moves in units of 2^-30
@pytest.mark.parametrize("move", [-240, 0, 240])
def test_square_root(lib, move):
    rng = random.Random(1)
    with mp.workdps(40):
        for a in _fractions(rng, 2**62, 2**64 - 2**44):
            want = mp.sqrt(mp.mpf(a) / 2**64)
            assert abs(mp.mpf(lib.root(a, move)) / 2**64 / want - 1) < mp.mpf(2) ** -59.3, a


@pytest.mark.parametrize("move", [-256, 0, 256])
def test_reciprocal(lib, move):
    rng = random.Random(2)
    with mp.workdps(40):
        for m in _fractions(rng, 2**63, 2**64):
            want = mp.mpf(2) ** 63 / m
            assert abs(mp.mpf(lib.rcp(m, move)) / 2**63 / want - 1) < mp.mpf(2) ** -60, m


def test_logarithm(lib):
    rng = random.Random(3)
    ms = _fractions(rng, 2**63, 2**64) + [2**63 + (i << 53) - d for i in range(1, 1024) for d in (0, 1)]
    with mp.workdps(40):
        for m in ms:
            e = rng.choice([1, 1, 2, 3, 10, 33])
            want = e * mp.log(2) - mp.log(mp.mpf(m) / 2**63)
            assert abs(mp.mpf(lib.nlog(m, e)) / 2**59 - want) < mp.mpf(2) ** -57 + e * mp.mpf(2) ** -60, (m, e)


def test_doubles_round_like_the_library(lib):
    import math
    rng = random.Random(4)
    xs = [1.0, 2.0, 4.0, 0.25, 0.5, 3.0, 1.0 + 2**-52, 2.0 - 2**-52, 4.0 - 2**-51, 2.0**-1000, 2.0**1000]
    xs += [math.ldexp(rng.uniform(1.0, 2.0), rng.randint(-300, 300)) for _ in range(4000)]
    for x in xs:  # the true root or reciprocal rounds to the library's result, or ties within 2^-59
        assert abs(lib.root_double(x) / math.sqrt(x) - 1.0) <= 2.0**-52
        assert abs(lib.rcp_double(x) * x - 1.0) <= 2.0**-52
    same = sum(lib.root_double(x) == math.sqrt(x) for x in xs)
    assert same >= 0.97 * len(xs)
