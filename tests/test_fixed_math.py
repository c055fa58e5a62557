"""The fixed-point quantile and exponential (csrc/fixed_math.hpp) against
40-digit values, compiled for the host.

Bars, from the construction: the quantile's polynomials are truncated below
c5 / 512 < 1.2e-17 and evaluated with three 2^-61 truncations (1.3e-18): 1.4e-17.
The exponential's dropped cubic term is below 2^-64, its products lose a few
units of 2^-63: 2e-18.
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
using namespace mcdg;
extern "C" uint64_t quantile(uint32_t w) {
    const FixedTables& t = fixed_tables();
    const QuantArg a = quant_arg(w);
    return quant_eval(t.lo[a.entry], t.hi[a.entry], a.s);
}
extern "C" uint64_t exponential(uint64_t f) {
    const FixedTables& t = fixed_tables();
    return exp2_frac(f, t.exp_a[exp2_index_a(f)], t.exp_b[exp2_index_b(f)]);
}
extern "C" uint64_t as_double(uint64_t m, int e) { return double_bits(m, e); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    src, so = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++20", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, src, "-o", so],
                   check=True)
    L = C.CDLL(so)
    for name, args in (("quantile", [C.c_uint32]), ("exponential", [C.c_uint64]), ("as_double", [C.c_uint64, C.c_int])):
        getattr(L, name).restype = C.c_uint64
        getattr(L, name).argtypes = args
    return L


def _quantile(w):  # -Phi^-1(w / 2^33)
    q = mp.mpf(w) / 2**33
    if w >= 2**20:
        return -mp.sqrt(2) * mp.erfinv(2 * q - 1)
    z = -mp.sqrt(-2 * mp.log(q)) + mp.mpf("0.4")
    for _ in range(60):  # Newton on log Phi
        step = (mp.log(mp.ncdf(z)) - mp.log(q)) * mp.ncdf(z) / mp.npdf(z)
        z -= step
        if abs(step) < mp.mpf(10) ** -35:
            break
    return -z


def test_quantile_every_octave_and_interval_edges(lib):
    rng = random.Random(5)
    ws = [1, 2, 3, 2**32 - 1, 2**32 - 2]
    for octave in range(32):
        lo = 2**octave
        ws += [lo, 2 * lo - 1] + [rng.randrange(lo, 2 * lo) for _ in range(6)]
        width = lo >> 9
        if width:
            i = rng.randrange(512)
            ws += [lo + i * width, lo + i * width + width - 1]
    with mp.workdps(40):
        worst = max(abs(mp.mpf(lib.quantile(w)) / 2**61 - _quantile(w)) for w in ws)
    assert worst < 1.4e-17, float(worst)


def test_exponential_edges(lib):
    rng = random.Random(6)
    top = 2**64 - 1
    fs = [0, 1, top, top - 1, 2**63, 2**63 - 1]
    for bits in (54, 44):  # table boundaries
        for _ in range(20):
            i = rng.randrange(1, 2 ** (64 - bits))
            fs += [i << bits, (i << bits) - 1]
    fs += [rng.getrandbits(64) for _ in range(300)]
    with mp.workdps(40):
        worst = max(abs(mp.mpf(lib.exponential(f)) / 2**63 - mp.power(2, mp.mpf(f) / 2**64)) for f in fs)
    assert worst < 2e-18, float(worst)


@pytest.mark.parametrize("e", [-511, -1, 0, 7, 511])
def test_double_conversion_rounds_and_carries(lib, e):
    import struct
    for m in (2**63, 2**63 + 1023, 2**63 + 1024, 2**64 - 1, 2**64 - 1025, 0xC000000000000401):
        got = struct.unpack("<d", struct.pack("<Q", lib.as_double(m, e)))[0]
        with mp.workdps(40):
            want = mp.ldexp(mp.mpf(m), e - 63)
            assert abs(mp.mpf(got) - want) <= mp.ldexp(1, e - 53)  # half a unit in the last place
