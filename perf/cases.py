"""Performance cases of the LSM engine: what its users price, through the public entry points.

Kinds of work:
  call    price_lsm_call: one contract priced by itself (a quote, a risk run's single trade)
  greeks  price_lsm_call_greeks: the same with the pathwise adjoint sensitivities
  paths   simulate_gbm_on_device: seeded path states left on the device for the caller's own work
  rows    price_lsm_call_batch: independent contracts, one population pair each
  groups  price_lsm_call_grouped_batch: market states, each with a strip of strikes
  ragged  price_lsm_call_ragged[_greeks]: contracts with their own path counts and schedules

Markets and Philox seeds are drawn from the preparation's seed, in the ranges of the repository's
batch workloads (tests/_workloads.py) and of its single-contract configurations. What sizes the work
(dates, dividend counts and path counts of every contract) belongs to the case.
"""

from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "finoptions-engine_b200"))

import finoptions as fo  # noqa: E402

POLICIES = {"liquidator": fo.DividendPolicy.LIQUIDATOR, "survivor": fo.DividendPolicy.SURVIVOR}
CONTINUE = fo.InsufficientExerciseSupportPolicy.CONTINUE
FAIL = fo.InsufficientExerciseSupportPolicy.FAIL
EVALUATION_DOMAIN = 1 << 20
CONDITION_LIMIT = 1.0e12  # a batch of random markets keeps rows with very few in-the-money paths


def listed() -> list[dict]:
    return [
        # The smallest call: one exercise date and one cash dividend; latency and launches count.
        {"name": "call_two_dates", "kind": "call", "paths": 65536, "dates": 1, "dividends": 1, "degree": 4,
         "policy": "liquidator"},
        # An indicative quote: few paths, monthly dates, a low degree.
        {"name": "call_monthly_4k", "kind": "call", "paths": 4099, "dates": 12, "dividends": 0, "degree": 2,
         "policy": "liquidator"},
        # An ordinary price: weekly dates, a ragged path count, cash dividends.
        {"name": "call_weekly_100k", "kind": "call", "paths": 100003, "dates": 52, "dividends": 2, "degree": 3,
         "policy": "survivor"},
        # The benchmark contract: weekly dates, 2^20 training and evaluation paths.
        {"name": "call_weekly_1m", "kind": "call", "paths": 1048576, "dates": 52, "dividends": 0, "degree": 4,
         "policy": "liquidator"},
        # A population beyond the on-chip capacity of the backward pass.
        {"name": "call_monthly_3m", "kind": "call", "paths": 3000001, "dates": 12, "dividends": 1, "degree": 4,
         "policy": "liquidator"},
        # Price and every sensitivity of one weekly contract with two cash dividends.
        {"name": "greeks_weekly_256k", "kind": "greeks", "paths": 262143, "dates": 52, "dividends": 2, "degree": 4,
         "policy": "liquidator"},
        # Path export for a caller's own device work.
        {"name": "paths_weekly_256k", "kind": "paths", "paths": 262144, "dates": 52, "dividends": 2,
         "policy": "liquidator"},
        # A small blotter: independent rows on a uniform mesh with continuous yields.
        {"name": "rows_96", "kind": "rows", "rows": 96, "paths": 16384, "dates": 16, "degree": 3},
        # One underlying's book refresh: 128 states x 8 strikes.
        {"name": "groups_128x8", "kind": "groups", "groups": 128, "strikes": 8, "paths": 32768, "degree": 4,
         "model": "cash"},
        # The benchmark batch: 4,096 states x 8 strikes.
        {"name": "groups_4096x8", "kind": "groups", "groups": 4096, "strikes": 8, "paths": 32768, "degree": 4,
         "model": "cash"},
        # A desk's uneven book, prices only and with every sensitivity.
        {"name": "ragged_1024", "kind": "ragged", "rows": 1024, "most_paths": 262144, "most_dates": 104, "degree": 4,
         "greeks": False},
        {"name": "ragged_greeks_1024", "kind": "ragged", "rows": 1024, "most_paths": 262144, "most_dates": 104,
         "degree": 4, "greeks": True},
    ]


def draw(rng) -> dict:
    def spread(lo: int, hi: int) -> int:
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("call", "call", "greeks", "paths", "rows", "groups", "groups", "ragged", "ragged"))
    if kind in ("call", "greeks", "paths"):
        dates = spread(1, 104)
        case = {"kind": kind, "paths": spread(4096, min(3000000, 110_000_000 // dates)), "dates": dates,
                "dividends": rng.randint(0, min(4, dates)), "policy": rng.choice(sorted(POLICIES))}
        return case if kind == "paths" else {**case, "degree": rng.randint(2, 4)}
    if kind == "rows":
        return {"kind": kind, "rows": spread(16, 1024), "paths": spread(4096, 32768), "dates": rng.randint(8, 52),
                "degree": rng.randint(2, 4)}
    if kind == "groups":
        groups, strikes = spread(16, 1024), rng.randint(1, 12)
        return {"kind": kind, "groups": groups, "strikes": strikes, "paths": spread(8192, 32768),
                "degree": rng.randint(2, 4), "model": rng.choice(("cash", "yield", "escrowed"))}
    return {"kind": kind, "rows": spread(32, 1024), "most_paths": spread(16384, 262144),
            "most_dates": rng.randint(12, 104), "degree": rng.randint(2, 4), "greeks": rng.random() < 0.5}


# ---- inputs ---------------------------------------------------------------------------------------


def _contract(case: dict, seed: int) -> dict:
    """One contract near the money on equally spaced dates; a call of one date is the two-date
    contract (times 0, T/2, T), others exercise at the origin (not with one date) and at every date."""
    rng = np.random.default_rng([seed, 1])
    n = 2 if case["dates"] == 1 else case["dates"]
    maturity = float(rng.uniform(0.8, 1.25))
    rate, dividend_yield = float(rng.uniform(0.01, 0.05)), float(rng.uniform(0.0, 0.03))
    spot = float(rng.uniform(80.0, 125.0))
    times = [maturity * (i / n) for i in range(n + 1)]
    picks = sorted(int(v) for v in rng.choice(np.arange(1, n), size=min(case["dividends"], n - 1), replace=False))
    return {
        "spot": spot, "strike": spot * float(rng.uniform(0.95, 1.02)), "times": times,
        "log_discounts": [0.0] + [-rate * t for t in times[1:]],
        "yields": [0.0] + [dividend_yield * t for t in times[1:]],
        "dividends": [(i, float(rng.uniform(0.5, 2.0))) for i in picks],
        "exercise": [1] if case["dates"] == 1 else list(range(n)), "expiry": n,
        "volatility": float(rng.uniform(0.2, 0.35)), "stream": int(rng.integers(1, 1 << 40)),
    }


def _group_markets(rng: np.random.Generator, shape: np.random.Generator, groups: int, least: int, most: int,
                   cash: int):
    """Exercise times T k / n (k = 1..n-1, n uniform in least..most) and up to `cash` dividend dates
    picked among them, for `groups` states; the counts come from `shape`, the times from `rng`."""
    maturity = rng.uniform(0.25, 2.0, groups)
    n = shape.integers(least, most + 1, groups)
    k = np.arange(1, most)[None, :]
    live = k < n[:, None]
    times = np.where(live, maturity[:, None] * (k / n[:, None]), np.inf)
    wanted = np.minimum(shape.integers(0, cash + 1, groups), n - 1)
    order = np.argsort(np.where(live, rng.random(live.shape), 2.0), axis=1)
    rank = np.empty_like(order)
    np.put_along_axis(rank, order, np.broadcast_to(np.arange(order.shape[1]), order.shape), axis=1)
    paid = live & (rank < wanted[:, None])

    def ragged(mask):
        return np.concatenate([[0], np.cumsum(mask.sum(axis=1))]).astype(np.int64), times[mask]

    return maturity, ragged(live), ragged(paid)


def _method(case: dict, paths: int, stream: int, support, **more) -> fo.Lsm:
    return fo.Lsm(training_paths=paths, evaluation_paths=paths, training_stream=fo.RandomStream(seed=stream, domain=0),
                  evaluation_stream=fo.RandomStream(seed=stream, domain=EVALUATION_DOMAIN),
                  insufficient_exercise_support=support, polynomial_degree=case["degree"], **more)


@functools.cache
def _executor() -> fo.CudaExecutor:
    """The program's one executor: it owns the device arenas and the tuned batch shapes."""
    return fo.CudaExecutor(device=0)


def prepare(case: dict, seed: int) -> dict:
    executor = _executor()
    kind = case["kind"]
    if kind in ("call", "greeks", "paths"):
        c = _contract(case, seed)
        times = tuple(c["times"])
        common = {
            "initial_spot": c["spot"],
            "schedule": fo.EventSchedule(times=times,
                                         dividends=tuple(fo.CashDividend(node=i, amount=a) for i, a in c["dividends"]),
                                         exercise_nodes=tuple(c["exercise"]), expiry_node=c["expiry"]),
            "curve": fo.LogDiscountCurve(times=times, log_discounts=tuple(c["log_discounts"])),
            "dividend_yield_curve": fo.CumulativeDividendYieldCurve(times=times, cumulative_yields=tuple(c["yields"])),
            "volatility": fo.ConstantVolatility(c["volatility"]), "dividend_policy": POLICIES[case["policy"]],
            "executor": executor,
        }
        if kind == "paths":
            return {"kind": kind, "args": {**common, "paths": case["paths"],
                                           "random_stream": fo.RandomStream(seed=c["stream"], domain=0)}}
        return {"kind": kind, "args": {**common, "strike": c["strike"],
                                       "method": _method(case, case["paths"], c["stream"], FAIL)}}
    rng = np.random.default_rng([seed, 2])
    shape = np.random.default_rng([case.get("groups", 0), case.get("rows", 0), case["paths"] if "paths" in case else 41])
    stream = int(rng.integers(1, 1 << 40))
    if kind == "rows":
        r = case["rows"]
        spots = rng.uniform(50.0, 150.0, r)
        return {"kind": kind, "args": {
            "initial_spots": spots, "strikes": spots * rng.uniform(0.8, 1.2, r), "maturities": rng.uniform(0.25, 2.0, r),
            "rates": rng.uniform(0.0, 0.06, r), "volatilities": rng.uniform(0.1, 0.6, r),
            "dividends": fo.ContinuousDividendYieldBatch(rng.uniform(0.0, 0.05, r)),
            "mesh": fo.UniformExerciseMesh(base_intervals=case["dates"], origin_exercise=fo.OriginExercise.EXCLUDED),
            "executor": executor,
            "method": _method(case, case["paths"], stream, CONTINUE, condition_limit=CONDITION_LIMIT)}}
    if kind == "groups":
        g = case["groups"]
        spots = rng.uniform(50.0, 150.0, g)
        maturity, exercise, cash = _group_markets(rng, shape, g, 12, 52, 4)
        strip = np.linspace(0.8, 1.2, case["strikes"]) if case["strikes"] > 1 else np.ones(1)
        schedules = fo.RaggedCashDividends(cash[0], cash[1], rng.uniform(0.5, 3.0, cash[1].size))
        if case["model"] == "cash":
            dividends = fo.CashDividendBatch(schedules, fo.DividendPolicy.LIQUIDATOR, fo.MaturityBoundary.STRICTLY_BEFORE)
        elif case["model"] == "escrowed":
            dividends = fo.EscrowedCashDividendBatch(schedules, fo.EscrowedVolatilityConvention.PREPAID_FORWARD,
                                                     fo.MaturityBoundary.STRICTLY_BEFORE)
        else:
            dividends = fo.ContinuousDividendYieldBatch(rng.uniform(0.0, 0.05, g))
        return {"kind": kind, "args": {
            "groups": fo.LsmStrikeGroups(
                group_offsets=(np.arange(g + 1) * case["strikes"]).astype(np.uint32), initial_spots=spots,
                strikes=(spots[:, None] * strip).reshape(-1), maturities=maturity, rates=rng.uniform(0.0, 0.06, g),
                volatilities=rng.uniform(0.1, 0.6, g), dividends=dividends),
            "mesh": fo.ExplicitExerciseMesh(schedules=fo.RaggedExerciseTimes(*exercise),
                                            origin_exercise=fo.OriginExercise.EXCLUDED),
            "executor": executor,
            "method": _method(case, case["paths"], stream, CONTINUE, condition_limit=CONDITION_LIMIT)}}
    r = case["rows"]
    least = min(8192, case["most_paths"])
    paths = np.floor(np.exp(shape.uniform(math.log(least), math.log(case["most_paths"]), r))).astype(np.uint64)
    spots = rng.uniform(20.0, 500.0, r)
    maturity, exercise, cash = _group_markets(rng, shape, r, 4, case["most_dates"], 6)
    return {"kind": "ragged", "greeks": case["greeks"], "args": {
        "contracts": fo.LsmRaggedContracts(
            initial_spots=spots, strikes=spots * rng.uniform(0.8, 1.2, r), maturities=maturity,
            rates=rng.uniform(0.0, 0.08, r), volatilities=rng.uniform(0.1, 0.8, r),
            exercise=fo.RaggedExerciseTimes(*exercise), training_paths=paths, evaluation_paths=paths,
            dividend_yields=np.where(np.arange(r) % 2 == 0, rng.uniform(0.0, 0.05, r), 0.0),
            cash_dividends=fo.RaggedCashDividends(cash[0], cash[1], rng.uniform(0.1, 3.0, cash[1].size))),
        "origin_exercise": fo.OriginExercise.EXCLUDED, "executor": executor,
        "training_stream": fo.RandomStream(seed=stream, domain=0),
        "evaluation_stream": fo.RandomStream(seed=stream, domain=EVALUATION_DOMAIN),
        "insufficient_exercise_support": CONTINUE, "polynomial_degree": case["degree"],
        "condition_limit": CONDITION_LIMIT}}


# ---- one pass -------------------------------------------------------------------------------------

COLUMNS = ("prices", "sample_standard_deviations", "standard_errors", "origin_decisions_fitted", "origin_exercised",
           "regression_nodes", "no_training_support_nodes", "insufficient_exercise_support_nodes",
           "minimum_in_the_money_training_paths", "maximum_regression_condition_numbers", "early_exercise_paths",
           "expiry_paths")


def _call_outputs(result) -> dict:
    fits = [d for d in result.fit_diagnostics if type(d) is fo.RegressionFitDiagnostics]
    return {
        "moments": np.array((result.price, result.sample_standard_deviation, result.standard_error)),
        "counts": np.array(result.exercise_counts), "in_the_money": np.array([d.in_the_money_paths for d in fits]),
        "mean": np.array([d.predictor_mean for d in fits]), "scale": np.array([d.predictor_scale for d in fits]),
        "condition": np.array([d.condition_number for d in fits]),
    }


def run(state: dict):
    kind, args = state["kind"], state["args"]
    if kind == "call":
        return _call_outputs(fo.price_lsm_call(**args))
    if kind == "greeks":
        g = fo.price_lsm_call_greeks(**args)
        return {**_call_outputs(g.result), "first": np.array((g.delta, g.vega)),
                "log_discounts": np.array(g.log_discount_sensitivities),
                "dividends": np.array(g.dividend_sensitivities)}
    if kind == "paths":
        return fo.simulate_gbm_on_device(**args).states
    if kind == "rows":
        batch, greeks = fo.price_lsm_call_batch(**args), None
    elif kind == "groups":
        batch, greeks = fo.price_lsm_call_grouped_batch(**args), None
    elif state["greeks"]:
        batch, greeks = fo.price_lsm_call_ragged_greeks(**args)
    else:
        batch, greeks = fo.price_lsm_call_ragged(**args), None
    out = {name: getattr(batch, name) for name in COLUMNS}
    if greeks is not None:
        out.update(delta=greeks.delta, vega=greeks.vega, log_discounts=greeks.log_discount_sensitivities,
                   dividends=greeks.dividend_sensitivities)
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------

NORMAL_STEP = 40.0  # one normal (its uniforms excepted), one exponential, one multiplication
DECIDE = 12.0       # standardise, predict, compare
REGRESS = 40.0      # power sums and response sums of one in-the-money path


def work(case: dict) -> dict:
    """Floating-point operations of the simulated path-steps, the regressions over the in-the-money
    half of the paths and the exercise decisions; bytes of the inputs and results."""
    kind = case["kind"]
    if kind == "paths":
        n = 2 if case["dates"] == 1 else case["dates"]
        return {"bytes": 8.0 * (n + 1) * case["paths"], "flops": NORMAL_STEP * n * case["paths"]}
    if kind in ("call", "greeks"):
        steps, strikes, rows = float(case["paths"]) * (2 if case["dates"] == 1 else case["dates"]), 1, 1
    elif kind == "rows":
        steps, strikes, rows = float(case["paths"]) * case["rows"] * case["dates"], 1, case["rows"]
    elif kind == "groups":
        steps, strikes = float(case["paths"]) * case["groups"] * 32, case["strikes"]
        rows = case["groups"] * strikes
    else:
        least, most = min(8192, case["most_paths"]), case["most_paths"]
        mean = (most - least) / math.log(most / least) if most > least else most
        steps, strikes, rows = mean * case["rows"] * (4 + case["most_dates"]) / 2, 1, case["rows"]
    return {"bytes": 1000.0 * rows, "flops": steps * (2 * NORMAL_STEP + strikes * 0.5 * (2 * DECIDE + REGRESS))}


# ---- the same results in plain numpy / torch binary64 ---------------------------------------------


def _tables() -> tuple[np.ndarray, np.ndarray]:
    """The 256-layer ZIGNOR tables from the published construction (r, v as the engine states them)."""
    r, v = 3.6541528853610088, 0.00492867323399
    x = np.zeros(257)
    x[0], x[1] = v / math.exp(-0.5 * r * r), r
    for i in range(2, 256):
        x[i] = math.sqrt(-2.0 * math.log(v / x[i - 1] + math.exp(-0.5 * x[i - 1] ** 2)))
    return x, np.exp(-0.5 * x * x)


def _words(seed: int, domain: int, path: np.ndarray, index: np.ndarray) -> np.ndarray:
    """Word `index` of each path's Philox4x32-10 stream (two 64-bit words per block, low half first)."""
    mask = np.uint64(0xFFFFFFFF)
    block = index >> np.uint64(1)
    c0, c1, c2 = block & mask, block >> np.uint64(32), path.astype(np.uint64)
    c3 = np.full_like(c0, domain)
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c2 = (p1 >> np.uint64(32)) ^ c1 ^ np.uint64(k0), (p0 >> np.uint64(32)) ^ c3 ^ np.uint64(k1)
        c1, c3 = p1 & mask, p0 & mask
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    odd = (index & np.uint64(1)).astype(bool)
    return np.where(odd, c2 | (c3 << np.uint64(32)), c0 | (c1 << np.uint64(32)))


def _normals(seed: int, domain: int, paths: int, count: int) -> np.ndarray:
    """[count, paths] standard normals of the streams (seed, domain, path)."""
    tx, tf = _tables()
    r = tx[1]
    path = np.arange(paths, dtype=np.uint64)
    at = np.zeros(paths, dtype=np.uint64)
    out = np.empty((count, paths))

    def take(who):
        w = _words(seed, domain, path[who], at[who])
        at[who] += np.uint64(1)
        return w

    def candidate(w):
        layer = (w & np.uint64(255)).astype(np.int64)
        unit = (w >> np.uint64(12)).astype(np.float64) * 2.0**-51 - 1.0
        return layer, unit, unit * tx[layer]

    def open_unit(w):
        return (w >> np.uint64(12)).astype(np.float64) * 2.0**-52 + 2.0**-53

    for i in range(count):
        who = np.arange(paths)
        layer, unit, value = candidate(take(who))
        while True:
            fine = np.abs(value) < tx[layer + 1]
            out[i, who[fine]] = value[fine]
            who, layer, unit, value = who[~fine], layer[~fine], unit[~fine], value[~fine]
            if not who.size:
                break
            tail = layer == 0
            rest, sign = who[tail], unit[tail] < 0.0
            while rest.size:
                x = np.log(open_unit(take(rest))) / r
                y = np.log(open_unit(take(rest)))
                good = -2.0 * y >= x * x
                out[i, rest[good]] = np.where(sign[good], x[good] - r, r - x[good])
                rest, sign = rest[~good], sign[~good]
            who, layer, value = who[~tail], layer[~tail], value[~tail]
            if not who.size:
                break
            u = (take(who) >> np.uint64(11)).astype(np.float64) * 2.0**-53
            good = tf[layer + 1] + (tf[layer] - tf[layer + 1]) * u < np.exp(-0.5 * value * value)
            out[i, who[good]] = value[good]
            who = who[~good]
            if not who.size:
                break
            layer, unit, value = candidate(take(who))
    return out


def _states(c: dict, policy: str, z: np.ndarray, lib=np, spot=None, sigma=None, logs=None, amounts=None):
    """States at the exercise nodes (before a cash dividend) and at expiry (after one)."""
    times, q = c["times"], c["yields"]
    logs = c["log_discounts"] if logs is None else logs
    sigma = c["volatility"] if sigma is None else sigma
    spot = c["spot"] if spot is None else spot
    amounts = [a for _, a in c["dividends"]] if amounts is None else amounts
    paid = {node: j for j, (node, _) in enumerate(c["dividends"])}
    s, rows = spot + 0.0 * z[0], []

    def jump(s, node):
        if node not in paid:
            return s
        left = s - amounts[paid[node]]
        return lib.where(left > 0.0, left, 0.0 * left if policy == "liquidator" else s)

    if 0 in c["exercise"]:
        rows.append(s)
    for i in range(len(times) - 1):
        dt = times[i + 1] - times[i]
        drift = -(logs[i + 1] - logs[i]) - (q[i + 1] - q[i]) - 0.5 * sigma * sigma * dt
        s = s * lib.exp(sigma * math.sqrt(dt) * z[i] + drift)
        if i + 1 == c["expiry"]:
            rows.append(jump(s, i + 1))
        elif i + 1 in c["exercise"]:
            rows.append(s)
        s = jump(s, i + 1)
    return rows


def _price(c: dict, policy: str, degree: int, paths: int, support_continues: bool, domains: tuple[int, int]):
    """Outputs of one contract: moments of the payoff, stopping counts and the regressions."""
    nodes = [*c["exercise"], c["expiry"]]
    logs, strike = np.array(c["log_discounts"]), c["strike"]
    train = _states(c, policy, _normals(c["stream"], domains[0], paths, len(c["times"]) - 1))
    value = np.maximum(train[-1] - strike, 0.0)
    rules, fits, later = {}, [], nodes[-1]
    for row in range(len(nodes) - 2, -1, -1):
        value = value * math.exp(logs[later] - logs[nodes[row]])
        later = nodes[row]
        if nodes[row] == 0:
            rules[row] = bool(max(c["spot"] - strike, 0.0) > value.mean())
            continue
        s = train[row]
        itm = s > strike
        n = int(itm.sum())
        if n < degree + 1 and (support_continues or n == 0):
            rules[row] = None
            fits.append((0, 0.0, 0.0, 0.0))
            continue
        x = s[itm] / strike
        mean = x.mean()
        scale = math.sqrt(np.mean((x - mean) ** 2))
        design = np.vander((x - mean) / scale, degree + 1, increasing=True)
        orthogonal, upper = np.linalg.qr(design)
        coef = np.linalg.solve(upper, orthogonal.T @ value[itm])
        rules[row] = (mean, scale, coef)
        fits.append((n, mean, scale, np.linalg.cond(upper)))
        now = s[itm] - strike
        value[itm] = np.where(now > design @ coef, now, value[itm])
    z = _normals(c["stream"], domains[1], paths, len(c["times"]) - 1)
    states = _states(c, policy, z)
    payoff, stop = np.zeros(paths), np.full(paths, len(nodes) - 1)
    alive = np.ones(paths, dtype=bool)
    for row in range(len(nodes) - 1):
        rule = rules[row]
        if rule is None or rule is False:
            continue
        if rule is True:
            now = alive
        else:
            mean, scale, coef = rule
            y = np.polynomial.polynomial.polyval((states[row] / strike - mean) / scale, coef)
            now = alive & (states[row] > strike) & (states[row] - strike > y)
        payoff[now] = np.maximum(states[row][now] - strike, 0.0) * math.exp(logs[nodes[row]])
        stop[now] = row
        alive &= ~now
    payoff[alive] = np.maximum(states[-1][alive] - strike, 0.0) * math.exp(logs[nodes[-1]])
    fits = fits[::-1]
    deviation = payoff.std(ddof=1)
    result = {"moments": np.array((payoff.mean(), deviation, deviation / math.sqrt(paths))),
              "counts": np.bincount(stop, minlength=len(nodes)), "fits": fits, "origin": rules.get(0) is True}
    return result, z, stop, nodes


def _greeks(c: dict, policy: str, z: np.ndarray, stop: np.ndarray, nodes: list[int]) -> dict:
    """Sensitivities of the mean payoff with every path's stopping row held fixed, by torch autograd."""
    leaf = lambda v: torch.tensor(v, dtype=torch.float64, requires_grad=True)  # noqa: E731
    spot, sigma, logs = leaf(c["spot"]), leaf(c["volatility"]), leaf(c["log_discounts"])
    amounts = leaf([a for _, a in c["dividends"]])
    rows = torch.stack(_states(c, policy, torch.from_numpy(z), torch, spot, sigma, logs, amounts))
    at = torch.from_numpy(stop)
    held = rows.gather(0, at[None, :])[0]
    discount = torch.exp(logs[torch.tensor(nodes)][at])
    price = (torch.clamp(held - c["strike"], min=0.0) * discount).mean()
    grads = torch.autograd.grad(price, (spot, sigma, logs, amounts), allow_unused=True)
    return {"first": np.array((float(grads[0]), float(grads[1]))), "log_discounts": grads[2].numpy(),
            "dividends": np.zeros(0) if grads[3] is None else grads[3].numpy()}


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("call", "greeks", "paths"):
        c = _contract(case, seed)
        n = len(c["times"]) - 1
        if case["paths"] * n > 14_000_000:
            return None
        if kind == "paths":
            return np.stack(_states(c, case["policy"], _normals(c["stream"], 0, case["paths"], n)))
        got, z, stop, nodes = _price(c, case["policy"], case["degree"], case["paths"], False, (0, EVALUATION_DOMAIN))
        fits = got.pop("fits")
        if got.pop("origin"):
            return None
        columns = {name: np.array([f[i] for f in fits]) for i, name in
                   enumerate(("in_the_money", "mean", "scale", "condition"))}
        greeks = _greeks(c, case["policy"], z, stop, nodes) if kind == "greeks" else {}
        return {**got, **columns, **greeks}
    if kind != "rows" or case["rows"] * case["paths"] * case["dates"] > 26_000_000:
        return None
    a = prepare(case, seed)["args"]
    moments, conditions = [], []
    for r in range(case["rows"]):
        n, maturity = case["dates"], float(a["maturities"][r])
        times = [maturity * (i / n) for i in range(n + 1)]
        c = {"spot": float(a["initial_spots"][r]), "strike": float(a["strikes"][r]), "times": times,
             "log_discounts": [-float(a["rates"][r]) * t for t in times],
             "yields": [float(a["dividends"].annualized_decimals[r]) * t for t in times], "dividends": [],
             "exercise": list(range(1, n)), "expiry": n, "volatility": float(a["volatilities"][r]),
             "stream": a["method"].training_stream.seed}
        got, *_ = _price(c, "liquidator", case["degree"], case["paths"], True, (r, EVALUATION_DOMAIN + r))
        moments.append(got["moments"])
        conditions.append(max(f[3] for f in got["fits"]))
    out = dict.fromkeys(COLUMNS)
    price, deviation, error = np.array(moments).T
    out.update(prices=price, sample_standard_deviations=deviation, standard_errors=error,
               maximum_regression_condition_numbers=np.array(conditions))
    return out
