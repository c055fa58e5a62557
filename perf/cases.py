"""Workloads by which the engine's speed is followed.

Each case is one call (or one short series of calls) that a user's program makes,
through the public Python entry points: the drop-in module ``mcd`` for single
contracts in its default FP64 arithmetic, and ``mcd_gpu.Engine`` for batches.
``listed()`` names the cases, ``draw()`` gives more of the same ranges,
``prepare()`` makes a program's inputs from a seed, ``run()`` is one pass,
``work()`` what a pass cannot do without, ``exact()`` the same outputs in 64 bits
from plain torch.

Inputs are host records and host numbers, as the pricing API takes them; every
pass uploads them and brings its results back.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "derivative-pricing_gb300"))

import mcd  # noqa: E402  (the drop-in module, on the path set above)
import mcd_gpu as G  # noqa: E402

_engine = None


def engine():
    """The program's one engine (device memory, stream, graphs), kept for its life."""
    global _engine
    if _engine is None:
        _engine = G.Engine(0)
    return _engine


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # An interactive quote: one European option, few paths, the module's defaults
        # (FP64).  Latency and launches are what it costs.
        {"name": "european_small", "kind": "european", "paths": 10_000},
        # One daily-monitored arithmetic Asian with both variance reductions on, FP64:
        # the module's ordinary path-dependent call.
        {"name": "asian_cv", "kind": "asian_cv", "paths": 100_000, "steps": 252},
        # Sensitivities of one position through the module: finite-difference European,
        # likelihood-ratio barrier, pathwise Asian (FP64, weekly dates).
        {"name": "single_greeks", "kind": "single_greeks", "paths": 100_000, "steps": 52},
        # One Heston quasi-exponential call, FP64, daily steps.
        {"name": "heston_single", "kind": "heston_single", "paths": 100_000, "steps": 252},
        # One American put by Longstaff-Schwartz, FP64, 50 dates: a long serial chain of
        # dates over one contract.
        {"name": "american_single", "kind": "american_single", "paths": 131_072, "steps": 50},
        # A book re-priced in the reference's arithmetic (FP64): mixed products, steps
        # and options, ragged path counts.
        {"name": "book_fp64", "kind": "book", "precision": "fp64", "contracts": 64, "options": True,
         "min_paths": 10_000, "max_paths": 300_000},
        # The batch the engine is built for: 4096 path-dependent contracts, FP32 paths,
        # 12 to 252 dates, 1e4 to 1e6 paths each.
        {"name": "book_fp32", "kind": "book", "precision": "fp32", "contracts": 4096, "options": False,
         "min_paths": 10_000, "max_paths": 1_000_000},
        # Batched risk: price and all estimators of 1024 daily-monitored contracts, FP32.
        {"name": "book_greeks", "kind": "book_greeks", "precision": "fp32", "contracts": 1024, "steps": 252,
         "paths": 262_144},
        # A Heston surface: 64 parameter sets against 64 strikes, FP32.
        {"name": "heston_surface", "kind": "heston_surface", "sets": 64, "strikes": 64, "steps": 252,
         "paths": 1_048_576},
        # The American grid fitted and bumped: 20 puts, QR regression, then delta, gamma
        # and vega against the frozen policies, FP32.
        {"name": "american_greeks", "kind": "american_greeks", "contracts": 20, "min_steps": 50, "max_steps": 50,
         "paths": 1_048_576},
        # The same grid by the learned regression (tensor-core network), FP32 paths.
        {"name": "american_learned", "kind": "american_learned", "contracts": 20, "min_steps": 50,
         "max_steps": 50, "paths": 1_048_576},
        # The batch under Sobol points and Brownian bridges, FP32.
        {"name": "book_qmc", "kind": "book_qmc", "precision": "fp32", "contracts": 4096, "min_paths": 10_000,
         "max_paths": 1_000_000},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["european", "asian_cv", "single_greeks", "heston_single", "american_single", "book", "book",
                       "book_greeks", "heston_surface", "american_greeks", "american_learned", "book_qmc"])
    if kind == "european":
        return {"kind": kind, "paths": _log_int(rng, 1_000, 2_000_000)}
    if kind in ("asian_cv", "single_greeks", "heston_single"):
        return {"kind": kind, "paths": _log_int(rng, 1_000, 200_000), "steps": _log_int(rng, 3, 252)}
    if kind == "american_single":
        return {"kind": kind, "paths": _log_int(rng, 5_000, 300_000), "steps": rng.randint(10, 100)}
    if kind == "book":
        precision = rng.choice(["fp64", "fp32"])
        n = _log_int(rng, 3, 100 if precision == "fp64" else 4096)
        return {"kind": kind, "precision": precision, "contracts": n, "options": rng.random() < 0.5,
                "min_paths": 1_000, "max_paths": 300_000}
    if kind == "book_greeks":
        precision = "fp32" if rng.random() < 0.75 else "fp64"
        return {"kind": kind, "precision": precision, "contracts": _log_int(rng, 3, 500 if precision == "fp32" else 24),
                "steps": rng.randint(10, 252), "paths": _log_int(rng, 3_000, 262_144 if precision == "fp32" else 60_000)}
    if kind == "heston_surface":
        return {"kind": kind, "sets": _log_int(rng, 1, 60), "strikes": rng.randint(1, 200),
                "steps": rng.randint(12, 252), "paths": _log_int(rng, 5_000, 1_000_000)}
    if kind in ("american_greeks", "american_learned"):
        lo = rng.randint(5, 50)
        return {"kind": kind, "contracts": _log_int(rng, 2, 60), "min_steps": lo, "max_steps": rng.randint(lo, 80),
                "paths": _log_int(rng, 10_000, 300_000)}
    return {"kind": kind, "precision": "fp32", "contracts": _log_int(rng, 3, 3000), "min_paths": 1_000,
            "max_paths": 500_000}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_VARIANTS = (
    [dict(product=G.ASIAN, average_style=a, strike_style=s, type=t) for a in (0, 1) for s in (0, 1) for t in (0, 1)]
    + [dict(product=G.BARRIER, direction=d, knock=k, type=t) for d in (0, 1) for k in (0, 1) for t in (0, 1)]
    + [dict(product=G.LOOKBACK, strike_style=s, type=t) for s in (0, 1) for t in (0, 1)]
    + [dict(product=G.DIGITAL, digital_style=0, type=t) for t in (0, 1)]
)


def _book(rng, n, min_paths, max_paths, options=False, products=None):
    """Contracts with the batch configuration's distributions (S0 100, K U[80,120], vol U[.1,.5],
    r U[0,.06], T U[.25,2], dates U{12..252}, paths log-uniform); with `options`, some carry
    antithetic pairing, control variates or the bridge correction, and Europeans join."""
    c = G.contracts(n)
    variants = [v for v in _VARIANTS if products is None or v["product"] in products]
    if options:
        variants = variants + [dict(product=G.EUROPEAN, type=t) for t in (0, 1)]
    for i, v in enumerate(rng.integers(0, len(variants), n)):
        for k, value in variants[v].items():
            c[k][i] = value
    c["spot"] = 100.0
    c["strike"] = rng.uniform(80, 120, n)
    c["vol"] = rng.uniform(0.1, 0.5, n)
    c["rate"] = rng.uniform(0.0, 0.06, n)
    c["time"] = rng.uniform(0.25, 2.0, n)
    c["monitoring_points"] = rng.integers(12, 253, n)
    c["path_count"] = np.round(np.exp(rng.uniform(math.log(min_paths), math.log(max_paths), n))).astype(np.uint64)
    h = rng.uniform(0.05, 0.3, n)
    c["barrier"] = np.where(c["direction"] == 0, 100.0 * (1 + h), 100.0 * (1 - h))
    c["seed"] = rng.integers(0, 2**40) + np.arange(n, dtype=np.uint64)
    if options:
        for name in ("antithetic", "control_variate", "brownian_bridge"):
            c[name] = rng.integers(0, 4, n) == 0
    return c


def _puts(rng, n, min_steps, max_steps, paths):
    """American puts around the grid (S0 36..44, K 40, r .06, vol .2-.4, T 1-2)."""
    c = np.zeros(n, dtype=G.LSM_CONTRACT_DTYPE)
    c["spot"] = rng.uniform(36, 44, n)
    c["strike"] = 40.0
    c["rate"] = 0.06
    c["vol"] = rng.uniform(0.2, 0.4, n)
    c["time"] = rng.uniform(1.0, 2.0, n)
    c["type"] = 1
    c["monitoring_points"] = rng.integers(min_steps, max_steps + 1, n)
    c["path_count"] = paths
    c["seed"] = rng.integers(0, 2**40) + np.arange(n, dtype=np.uint64)
    return c


def _heston_sets(rng, n):
    s = np.zeros(n, dtype=G.HESTON_DTYPE)
    s["spot"] = 100.0
    s["rate"] = 0.03
    s["kappa"] = rng.uniform(0.5, 3.0, n)
    s["theta"] = rng.uniform(0.02, 0.09, n)
    s["xi"] = rng.uniform(0.2, 1.0, n)
    s["rho"] = rng.uniform(-0.9, -0.3, n)
    s["v0"] = rng.uniform(0.01, 0.09, n)
    s["time"] = 1.0
    return s


def _inputs(case, seed):
    rng = np.random.default_rng([7, int(seed)])
    kind = case["kind"]
    if kind == "book":
        return _book(rng, case["contracts"], case["min_paths"], case["max_paths"], case["options"])
    if kind == "book_qmc":
        return _book(rng, case["contracts"], case["min_paths"], case["max_paths"])
    if kind == "book_greeks":
        c = _book(rng, case["contracts"], 10, 10, products=(G.ASIAN, G.BARRIER))
        c["monitoring_points"] = case["steps"]
        c["path_count"] = case["paths"]
        return c
    if kind in ("american_greeks", "american_learned"):
        return _puts(rng, case["contracts"], case["min_steps"], case["max_steps"], case["paths"])
    if kind == "american_single":
        return _puts(rng, 1, case["steps"], case["steps"], case["paths"])[0]
    if kind == "heston_surface":
        return {"sets": _heston_sets(rng, case["sets"]), "strikes": np.linspace(70.0, 130.0, case["strikes"]),
                "seed": int(rng.integers(0, 2**40))}
    if kind == "heston_single":
        return {"sets": _heston_sets(rng, 1), "strike": float(rng.uniform(80, 120)),
                "seed": int(rng.integers(0, 2**40))}
    market = {"spot": 100.0, "strike": float(rng.uniform(80, 120)), "rate": float(rng.uniform(0.0, 0.06)),
              "carry_yield": float(rng.uniform(0.0, 0.03)), "vol": float(rng.uniform(0.1, 0.5)),
              "time": float(rng.uniform(0.25, 2.0))}
    return {"market": market, "barrier": float(100.0 * (1 - rng.uniform(0.05, 0.3))),
            "seed": int(rng.integers(0, 2**40))}


def prepare(case, seed):
    state = {"case": case, "in": _inputs(case, seed)}
    if case["kind"] in ("book", "book_greeks", "book_qmc", "heston_surface", "american_greeks", "american_learned"):
        state["engine"] = engine()
    if case["kind"] == "heston_single":
        s = state["in"]["sets"][0]
        state["params"] = mcd.HestonParams(*[float(s[f]) for f in G.HESTON_DTYPE.names])
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _result(r):
    return {"price": np.float64(r.price), "standard_error": np.float64(r.standard_error)}


def _records(r):
    return {name: np.ascontiguousarray(r[name]) for name in ("price", "standard_error", "path_count")}


def run(state):
    case, x = state["case"], state["in"]
    kind = case["kind"]
    call, put = mcd.OptionType.Call, mcd.OptionType.Put
    if kind == "european":
        return _result(mcd.monte_carlo_european(*x["market"].values(), call, case["paths"], x["seed"]))
    if kind == "asian_cv":
        return _result(mcd.monte_carlo_asian(*x["market"].values(), call, mcd.StrikeStyle.Fixed,
                                             mcd.AverageStyle.Arithmetic, case["steps"], case["paths"], x["seed"],
                                             mcd.McOptions(antithetic=True, control_variate=True)))
    if kind == "single_greeks":
        m = x["market"]
        bumps = mcd.default_bump_sizes(m["spot"], m["vol"], m["time"])
        fd = mcd.finite_difference_european(*m.values(), call, case["paths"], x["seed"], bumps)
        lr = mcd.likelihood_ratio_barrier(m["spot"], m["strike"], x["barrier"], m["rate"], m["carry_yield"], m["vol"],
                                          m["time"], put, mcd.BarrierDirection.Down, mcd.BarrierKnock.Out, 0.0,
                                          case["steps"], case["paths"], x["seed"])
        pw = mcd.pathwise_asian(*m.values(), call, mcd.StrikeStyle.Fixed, mcd.AverageStyle.Arithmetic, case["steps"],
                                case["paths"], x["seed"])
        return {"fd": [np.float64(getattr(fd, k)) for k in ("delta", "gamma", "vega", "theta", "rho")],
                "lr": [np.array([getattr(lr, k).value, getattr(lr, k).standard_error])
                       for k in ("delta", "gamma", "vega", "rho")],
                "pathwise": [np.array([getattr(pw, k).value, getattr(pw, k).standard_error])
                             for k in ("delta", "vega", "rho")]}
    if kind == "heston_single":
        return _result(mcd.heston_qe_european(state["params"], x["strike"], call, case["steps"], case["paths"],
                                              x["seed"]))
    if kind == "american_single":
        return _result(mcd.monte_carlo_lsm_american(
            float(x["spot"]), float(x["strike"]), float(x["rate"]), float(x["carry_yield"]), float(x["vol"]),
            float(x["time"]), put, case["steps"], case["paths"], int(x["seed"])))
    eng = state["engine"]
    if kind == "book":
        return _records(eng.price_batch(x, case["precision"]))
    if kind == "book_qmc":
        return _records(eng.qmc_batch(x, case["precision"]))
    if kind == "book_greeks":
        r = eng.greeks_batch(x, 1e-4, 1e-4, case["precision"])
        return {name: np.ascontiguousarray(r[name]) for name in G.GREEK_NAMES}
    if kind == "heston_surface":
        return _records(eng.heston_qe_batch(x["sets"], x["strikes"], 0, case["steps"], case["paths"], x["seed"],
                                            "fp32"))
    if kind == "american_greeks":
        r = eng.lsm_greeks_batch(x, 0.01, 0.01, "fp32")
        out = {name: np.ascontiguousarray(r[name]) for name in ("delta", "gamma", "vega", "scenario")}
        return {"price": r["price"][:, 0].copy(), "price_se": r["price"][:, 1].copy(), **out}
    r = eng.lsm_batch(x, "fp32", "mlp")
    return {name: np.ascontiguousarray(r[name]) for name in ("price", "standard_error", "exercise_at_inception")}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# Floating operations of a path's step: a normal from its uniform (a polynomial of degree 8,
# a logarithm and two products: 20), the log-spot or spot step (4), the payoff's running value (2).
# Philox is integer work and not counted.
_STEP = 26.0


def work(case):
    kind = case["kind"]
    if kind == "european":
        return {"bytes": 200.0, "flops": _STEP * case["paths"]}
    if kind == "asian_cv":  # both antithetic halves, two running averages
        return {"bytes": 200.0, "flops": (_STEP + 10.0) * case["paths"] * case["steps"]}
    if kind == "single_greeks":  # European (nine re-prices of one draw) and two path-dependent calls
        return {"bytes": 600.0, "flops": case["paths"] * (100.0 + (2 * _STEP + 12.0) * case["steps"])}
    if kind == "heston_single":  # two draws and the variance step
        return {"bytes": 200.0, "flops": 70.0 * case["paths"] * case["steps"]}
    if kind == "heston_surface":
        return {"bytes": 72.0 * case["sets"] + 24.0 * case["sets"] * case["strikes"],
                "flops": case["sets"] * case["paths"] * (70.0 * case["steps"] + 3.0 * case["strikes"])}
    if kind in ("book", "book_qmc"):
        lo, hi = float(case["min_paths"]), float(case["max_paths"])
        mean_paths = (hi - lo) / math.log(hi / lo)
        # one of the 22 to 24 variants is terminal in twelve; the dates are U{12..252}
        return {"bytes": 152.0 * case["contracts"],
                "flops": _STEP * case["contracts"] * mean_paths * 132.0 * 11.0 / 12.0}
    if kind == "book_greeks":  # the bumped states and the scores beside the price
        return {"bytes": 336.0 * case["contracts"],
                "flops": (_STEP + 14.0) * case["contracts"] * case["steps"] * float(case["paths"])}
    if kind == "american_single":  # paths written once, a column and the cash flows read and written per date
        d, n, b = float(case["steps"]), float(case["paths"]), 8.0
        return {"bytes": n * (b * (d + 1) + (8 + 2 * b) * d), "flops": n * d * (_STEP + 45.0)}
    d = 0.5 * (case["min_steps"] + case["max_steps"])
    n = float(case["contracts"]) * case["paths"]
    flops = n * d * (_STEP + 45.0)
    if kind == "american_greeks":  # five scenarios on one set of draws
        flops += n * d * (_STEP + 40.0)
    else:  # training: 100 steps of 128 samples, three 64 x 64 products each
        flops += case["contracts"] * 100.0 * 3.0 * 2.0 * 128.0 * 64.0 * 64.0
    return {"bytes": n * (4.0 * (d + 1) + 20.0 * d), "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit values in plain torch
# ---------------------------------------------------------------------------
_DEV = "cuda"
_CHUNK = 1 << 25  # draws held at once


def _philox(seed, paths, draws, stream):
    """Word 0 of Philox4x32-10 at {path_lo, path_hi, draw, stream}, key {seed_lo, seed_hi}: int64 [paths, draws]."""
    mask = 0xFFFFFFFF
    c0 = (paths & mask)[:, None]
    c1 = (paths >> 32)[:, None]
    c2 = draws[None, :]
    c3 = torch.full((1, 1), stream, dtype=torch.int64, device=paths.device)
    k0, k1 = seed & mask, (seed >> 32) & mask
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (((p1 >> 32) & mask) ^ c1 ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c3 ^ k1, p0 & mask)
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c0


def _uniforms(seed, first, count, steps, stream=0):
    p = torch.arange(first, first + count, dtype=torch.int64, device=_DEV)
    d = torch.arange(steps, dtype=torch.int64, device=_DEV)
    return (_philox(int(seed), p, d, stream).double() + 0.5) * 2.0**-32


def _normals(seed, first, count, steps):
    return torch.special.ndtri(_uniforms(seed, first, count, steps))


class _Moments:
    """Mean and standard error over chunks (two-pass per chunk, merged)."""

    def __init__(self):
        self.n, self.mean, self.m2 = 0, 0.0, 0.0

    def add(self, v):
        n, mean = v.numel(), float(v.mean())
        m2 = float((v - mean).square().sum())
        d, total = mean - self.mean, self.n + n
        self.m2 += m2 + d * d * self.n * n / total
        self.mean += d * n / total
        self.n = total

    def se(self):
        return math.sqrt(self.m2 / (self.n - 1) / self.n) if self.n > 1 else 0.0


def _chunks(paths, steps):
    size = max(1, _CHUNK // max(steps, 1))
    for first in range(0, paths, size):
        yield first, min(size, paths - first)


def _kemna_vorst(c):
    vg = c["vol"] / math.sqrt(3.0)
    b = 0.5 * (c["rate"] - c["carry_yield"] - c["vol"] ** 2 / 6.0)
    sd = vg * math.sqrt(c["time"])
    d1 = (math.log(c["spot"] / c["strike"]) + (b + 0.5 * vg * vg) * c["time"]) / sd
    phi = 1.0 if c["type"] == 0 else -1.0

    def cdf(v):
        return 0.5 * math.erfc(-v / math.sqrt(2.0))
    return phi * (c["spot"] * math.exp((b - c["rate"]) * c["time"]) * cdf(phi * d1)
                  - c["strike"] * math.exp(-c["rate"] * c["time"]) * cdf(phi * (d1 - sd)))


def _samples(c, seed, z, first, vol=None):
    """Discounted payoffs of one contract (a dict of its fields) on the draws z [paths, steps]."""
    vol = c["vol"] if vol is None else vol
    n = z.shape[1]
    dt = c["time"] / n
    phi = 1.0 if c["type"] == 0 else -1.0
    x = torch.cumsum((c["rate"] - c["carry_yield"] - 0.5 * vol * vol) * dt + vol * math.sqrt(dt) * z, 1)
    s = c["spot"] * torch.exp(x)
    last = s[:, -1]
    disc = math.exp(-c["rate"] * c["time"])
    product = c["product"]
    if product == G.EUROPEAN:
        return disc * torch.clamp(phi * (last - c["strike"]), min=0.0)
    if product == G.DIGITAL:
        paid = last if c["digital_style"] else torch.full_like(last, c["cash_amount"])
        return disc * torch.where(phi * (last - c["strike"]) > 0.0, paid, 0.0)
    if product == G.ASIAN:
        arith, geo = s.mean(1), c["spot"] * torch.exp(x.mean(1))
        if c["average_style"] == G.ARITHMETIC and c["control_variate"] and c["strike_style"] == G.FIXED:
            a = disc * torch.clamp(phi * (arith - c["strike"]), min=0.0)
            return a - (disc * torch.clamp(phi * (geo - c["strike"]), min=0.0) - _kemna_vorst(c))
        avg = geo if c["average_style"] == G.GEOMETRIC else arith
        ref = last - avg if c["strike_style"] == G.FLOATING else avg - c["strike"]
        return disc * torch.clamp(phi * ref, min=0.0)
    if product == G.BARRIER:
        up = c["direction"] == G.UP
        hit = s >= c["barrier"] if up else s <= c["barrier"]
        if c["brownian_bridge"]:
            u = _uniforms(seed, first, z.shape[0], n, 1)
            lh = math.log(c["barrier"] / c["spot"])
            prev = torch.cat([torch.zeros_like(x[:, :1]), x[:, :-1]], 1)
            p = torch.exp(-2.0 * (lh - prev) * (lh - x) / (vol * vol * dt))
            hit = hit | (u < p)
        touched = hit.any(1)
        pays = ~touched if c["knock"] == G.OUT else touched
        return disc * torch.where(pays, torch.clamp(phi * (last - c["strike"]), min=0.0), c["rebate"])
    hi, lo = torch.clamp(s.amax(1), min=c["spot"]), torch.clamp(s.amin(1), max=c["spot"])
    if c["strike_style"] == G.FIXED:
        v = torch.clamp(hi - c["strike"], min=0.0) if c["type"] == 0 else torch.clamp(c["strike"] - lo, min=0.0)
        return disc * v
    return disc * (last - lo if c["type"] == 0 else hi - last)


def _price(c):
    """(price, standard error) of one contract record."""
    steps = 1 if c["product"] in (G.EUROPEAN, G.DIGITAL) else int(c["monitoring_points"])
    acc = _Moments()
    for first, count in _chunks(int(c["path_count"]), 4 * steps):
        z = _normals(int(c["seed"]), first, count, steps)
        v = _samples(c, int(c["seed"]), z, first)
        if c["antithetic"]:
            v = 0.5 * (v + _samples(c, int(c["seed"]), -z, first))
        acc.add(v)
    return acc.mean, acc.se()


def _field(row):
    return {name: row[name].item() for name in row.dtype.names}


def _european_at(m, seed, paths, spot=None, rate=None, vol=None, time=None):
    c = dict(m, product=G.EUROPEAN, type=0, antithetic=0, path_count=paths, seed=seed, monitoring_points=1)
    for name, v in (("spot", spot), ("rate", rate), ("vol", vol), ("time", time)):
        if v is not None:
            c[name] = v
    return _price(c)[0]


def _exact_single_greeks(case, x):
    m, seed, paths, n = x["market"], x["seed"], case["paths"], case["steps"]
    spot, k, r, q, vol, t = m.values()
    b = mcd.default_bump_sizes(spot, vol, t)
    p0 = _european_at(m, seed, paths)
    up, dn = (_european_at(m, seed, paths, spot=spot + h) for h in (b.spot, -b.spot))
    vu, vd = (_european_at(m, seed, paths, vol=vol + h) for h in (b.vol, -b.vol))
    ru, rd = (_european_at(m, seed, paths, rate=r + h) for h in (b.rate, -b.rate))
    tu, td = (_european_at(m, seed, paths, time=t + h) for h in (b.time, -b.time))
    fd = [(up - dn) / (2 * b.spot), (up - 2 * p0 + dn) / b.spot**2, (vu - vd) / (2 * b.vol),
          -(tu - td) / (2 * b.time), (ru - rd) / (2 * b.rate)]
    lr = [_Moments() for _ in range(4)]
    pw = [_Moments() for _ in range(3)]
    dt = t / n
    sq, disc = math.sqrt(dt), math.exp(-r * t)
    bar = dict(m, product=G.BARRIER, type=1, direction=G.DOWN, knock=G.OUT, rebate=0.0, barrier=x["barrier"],
               brownian_bridge=0)
    i = torch.arange(1, n + 1, dtype=torch.float64, device=_DEV)
    for first, count in _chunks(paths, 6 * n):
        z = _normals(seed, first, count, n)
        h = _samples(bar, seed, z, first)
        z1 = z[:, 0]
        lr[0].add(h * z1 / (spot * vol * sq))
        lr[1].add(h * (z1 * z1 - vol * sq * z1 - 1.0) / (spot * spot * vol * vol * dt))
        lr[2].add(h * ((z * z - 1.0) / vol - sq * z).sum(1))
        lr[3].add(h * ((sq * z / vol).sum(1) - t))
        w = torch.cumsum(z, 1)
        s = spot * torch.exp((r - q - 0.5 * vol * vol) * dt * i + vol * sq * w)
        avg = s.mean(1)
        itm = (avg > k).double()
        pw[0].add(disc * itm * avg / spot)
        pw[1].add(disc * itm * (s * (sq * w - vol * dt * i)).mean(1))
        pw[2].add(disc * itm * (s * (dt * i)).mean(1) - t * disc * torch.clamp(avg - k, min=0.0))
    return {"fd": [np.float64(v) for v in fd], "lr": [np.array([a.mean, a.se()]) for a in lr],
            "pathwise": [np.array([a.mean, a.se()]) for a in pw]}


def _exact_heston(row, strike, steps, paths, seed):
    spot, rate, q, v0, kappa, theta, xi, rho, time = (float(row[f]) for f in G.HESTON_DTYPE.names)
    dt = time / steps
    e = math.exp(-kappa * dt)
    k0 = -rho * kappa * theta * dt / xi
    k1 = 0.5 * dt * (kappa * rho / xi - 0.5) - rho / xi
    k2 = 0.5 * dt * (kappa * rho / xi - 0.5) + rho / xi
    k3 = 0.5 * dt * (1.0 - rho * rho)
    acc = _Moments()
    for first, count in _chunks(paths, 4 * steps):
        zs = _normals(seed, first, count, steps)
        us = _uniforms(seed, first, count, steps, 1)
        zv = torch.special.ndtri(us)
        v = torch.full((count,), v0, dtype=torch.float64, device=_DEV)
        x = torch.full_like(v, math.log(spot))
        for j in range(steps):
            m = theta + (v - theta) * e
            s2 = v * xi * xi * e / kappa * (1 - e) + theta * xi * xi / (2 * kappa) * (1 - e) ** 2
            psi = s2 / (m * m)
            inv = 1.0 / torch.clamp(psi, max=1.5)
            b2 = 2 * inv - 1 + torch.sqrt(2 * inv) * torch.sqrt(2 * inv - 1)
            quad = m / (1 + b2) * (torch.sqrt(b2) + zv[:, j]) ** 2
            p = (psi - 1) / (psi + 1)
            u = us[:, j]
            expo = torch.where(u <= p, 0.0, torch.log((1 - p) / (1 - u)) * m / (1 - p))
            vn = torch.where(psi <= 1.5, quad, expo)
            x = x + (rate - q) * dt + k0 + k1 * v + k2 * vn + torch.sqrt(torch.clamp(k3 * (v + vn), min=0)) * zs[:, j]
            v = vn
        acc.add(math.exp(-rate * time) * torch.clamp(torch.exp(x) - strike, min=0.0))
    return {"price": np.float64(acc.mean), "standard_error": np.float64(acc.se())}


def _laguerre(s, strike):
    x = s / strike
    e = torch.exp(-0.5 * x)
    return torch.stack([e, e * (1 - x), e * (1 - 2 * x + 0.5 * x * x),
                        e * (1 - 3 * x + 1.5 * x * x - x * x * x / 6.0)], 1)


def _exact_american(c):
    """Price and standard error of one put by Longstaff-Schwartz with a Householder QR regression."""
    n, paths = int(c["monitoring_points"]), int(c["path_count"])
    dt = c["time"] / n
    s = torch.empty((n, paths), dtype=torch.float64, device=_DEV)
    for first, count in _chunks(paths, 4 * n):
        z = _normals(int(c["seed"]), first, count, n)
        x = torch.cumsum((c["rate"] - c["carry_yield"] - 0.5 * c["vol"] ** 2) * dt + c["vol"] * math.sqrt(dt) * z, 1)
        s[:, first:first + count] = (c["spot"] * torch.exp(x)).T
    disc = math.exp(-c["rate"] * dt)
    cf = torch.clamp(c["strike"] - s[n - 1], min=0.0)
    for d in range(n - 2, -1, -1):
        cf = cf * disc
        itm = torch.nonzero(s[d] < c["strike"]).flatten()
        if itm.numel() < 4:
            continue
        basis = _laguerre(s[d][itm], c["strike"])
        qm, rm = torch.linalg.qr(basis)
        beta = torch.linalg.solve_triangular(rm, (qm.T @ cf[itm])[:, None], upper=True)
        intrinsic = c["strike"] - s[d][itm]
        cf[itm] = torch.where(intrinsic > (basis @ beta)[:, 0], intrinsic, cf[itm])
    acc = _Moments()
    acc.add(cf * disc)
    now = max(c["strike"] - c["spot"], 0.0)
    return (now, 0.0) if now > acc.mean else (acc.mean, acc.se())


def exact(case, seed):
    x, kind = _inputs(case, seed), case["kind"]
    if kind in ("european", "asian_cv"):
        asian = kind == "asian_cv"
        c = dict(x["market"], product=G.ASIAN if asian else G.EUROPEAN, type=0, strike_style=G.FIXED,
                 average_style=G.ARITHMETIC, antithetic=asian, control_variate=asian, path_count=case["paths"],
                 seed=x["seed"], monitoring_points=case.get("steps", 1))
        p, se = _price(c)
        return {"price": np.float64(p), "standard_error": np.float64(se)}
    if kind == "single_greeks":
        return _exact_single_greeks(case, x)
    if kind == "heston_single":
        return _exact_heston(x["sets"][0], x["strike"], case["steps"], case["paths"], x["seed"])
    if kind == "american_single":
        p, se = _exact_american(_field(x))
        return {"price": np.float64(p), "standard_error": np.float64(se)}
    if kind == "book":
        steps = np.where(x["product"] <= G.DIGITAL, 1, x["monitoring_points"]).astype(np.float64)
        if float((steps * x["path_count"].astype(np.float64)).sum()) > 4e9:  # over about 20 seconds
            return None
        rows = [_price(_field(r)) for r in x]
        return {"path_count": None, "price": np.array([r[0] for r in rows]),
                "standard_error": np.array([r[1] for r in rows])}
    if kind == "american_greeks" and float(case["paths"]) * case["contracts"] * case["max_steps"] < 1.2e9:
        # the price; the sensitivities are taken against the engine's own fitted policy
        rows = [_exact_american(_field(r)) for r in x]
        return {"price": np.array([r[0] for r in rows]), "price_se": np.array([r[1] for r in rows]), "delta": None,
                "gamma": None, "vega": None, "scenario": None}
    # The learned regression's networks and the Sobol directions are the engine's own, and the
    # batched Greeks and the Heston surface take longer than about 20 seconds.
    return None
