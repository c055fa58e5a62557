"""What a context puts on the GPU when it is created is there before its first call, whatever
the legacy stream (a program's default one) has queued: the context's own stream is not ordered
after that one.

Each round queues some 10 ms of work on the legacy stream, creates an engine behind it and
compares its first call with an idle engine's, byte for byte.
"""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

import mcd_gpu as G

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _busy(x):
    for _ in range(40):
        x = torch.sin(x)
    return x


@pytest.fixture(scope="module")
def work():
    x = torch.rand(1 << 28, device="cuda")
    torch.cuda.synchronize()
    return x


def _contracts():
    c = G.contracts(2)
    c["spot"] = c["strike"] = 100.0
    c["rate"], c["vol"], c["time"], c["monitoring_points"] = .03, .25, 1.0, 1
    c["path_count"], c["seed"] = 20_000, 11
    return c


def test_first_quote_of_an_engine_created_behind_queued_work(engine, work):
    one = _contracts()[:1]  # one European contract: the last CTA is known by a counter set at creation
    want = engine.price_batch(one, "fp64").tobytes()
    for _ in range(10):
        _busy(work)
        with G.Engine(0) as e:
            got = [e.price_batch(one, "fp64").tobytes() for _ in range(3)]
        assert got == [want] * 3
    torch.cuda.synchronize()


def test_first_sobol_batch_of_an_engine_behind_queued_work(engine, work):
    c = _contracts()
    want = engine.qmc_batch(c, "fp32").tobytes()
    for _ in range(5):
        with G.Engine(0) as e:
            _busy(work)
            assert e.qmc_batch(c, "fp32").tobytes() == want
    torch.cuda.synchronize()


_CHILD = """
import sys
sys.path[:0] = [%r, %r]
import torch
import test_gpu_creation_order as T
import mcd_gpu as G
x = torch.rand(1 << 28, device="cuda")
torch.cuda.synchronize()
T._busy(x)
with G.Engine(0) as e:
    print(e.price_batch(T._contracts(), "fp64").tobytes().hex())
"""


def test_first_call_of_a_process_behind_queued_work(engine):
    """The process's one copy of the fixed-point tables has ended before the first kernel."""
    here = os.path.dirname(os.path.abspath(__file__))
    package = os.path.dirname(os.path.abspath(G.__file__))
    want = engine.price_batch(_contracts(), "fp64").tobytes().hex()
    r = subprocess.run([sys.executable, "-c", _CHILD % (here, package)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == want
