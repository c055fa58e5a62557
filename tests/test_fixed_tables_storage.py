"""The fixed-point tables (csrc/fixed_tables.cpp) are computed without the heap: the
allocation-free entry point asks for them behind a C interface, where a failed allocation has no
status.  Compiled for the host with an operator new that always fails, and asked for by several
threads at once.
"""
from __future__ import annotations

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "derivative-pricing_gb300", "csrc")
SOURCE = """
#include "fixed_tables.cpp"
#include <cstdio>
#include <cstdlib>
#include <new>
#include <pthread.h>
void* operator new(std::size_t) { throw std::bad_alloc(); }
void operator delete(void*) noexcept {}
void operator delete(void*, std::size_t) noexcept {}
static void* ask(void*) { return (void*)&mcdg::fixed_tables(); }
int main() {
    pthread_t t[4];
    void* seen[4];
    for (auto& x : t) pthread_create(&x, nullptr, ask, nullptr);
    for (int i = 0; i < 4; ++i) pthread_join(t[i], &seen[i]);
    for (void* p : seen) if (p != seen[0]) return 1;
    const mcdg::FixedTables& f = mcdg::fixed_tables();
    // 2^0 and 2^(1/1024) in units of 2^-63, the quantile falling towards q = 1/2
    if (f.exp_a[0] != 1ull << 63 || f.exp_a[1] <= f.exp_a[0] || f.lo[0].c0 <= f.lo[1].c0) return 2;
    std::puts("ok");
}
"""


def test_tables_need_no_heap(tmp_path):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++20", "-O2", "-ffp-contract=off", "-I", CSRC, src, "-o", exe, "-pthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stderr)
