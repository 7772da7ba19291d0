"""The calls whose speed matters to a user of this package, as cases to measure: quotes and revaluations through
`optlab_b200`'s public entry points, from the smallest call to a risk revaluation of a book.

`listed()` names the cases; `draw(rng)` gives one more of the same ranges; `prepare` builds what a caller has in hand
before the call (requests, plans, surfaces), `run` is one call with its whole result, `work` the operations and bytes
that call cannot do without, and `exact` the same result in 64 bits by plain torch.
"""

from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path(__file__).resolve().parents[1] / "option-pricing-lab_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import optlab_b200 as ob  # noqa: E402
from optlab_b200 import engine, requests, script, surfaces, workloads  # noqa: E402
from optlab_b200._abi import (  # noqa: E402
    BARRIER,
    OB_MODEL_HESTON_QE,
    OB_MODEL_PATHS,
    OB_PRODUCT_AUTOCALL,
    OB_PRODUCT_LADDER,
)
from optlab_b200.adjoint import AdjointPlan, VegaNodes, autocall_greeks  # noqa: E402
from optlab_b200.batch import Batch, sample_book  # noqa: E402
from optlab_b200.models import (  # noqa: E402
    Basket,
    HestonModel,
    HestonParams,
    Leverage,
    LocalVolModel,
    SLVModel,
    correlation_root,
)

STEPS_PER_YEAR = 252
SMOOTHING = 0.005


# ------------------------------------------------------------------------------------------------------- the cases


def listed():
    return [
        # the smallest call: one option ladder quoted on few paths, everything uploaded and read back in the call
        {"name": "qe_quote", "family": "qe", "paths": 2**12, "steps": 252, "precision": "fp64"},
        # the Heston QE ladder at its benchmark size
        {"name": "qe_ladder", "family": "qe", "paths": 2**16, "steps": 252, "precision": "fp64"},
        # an indicative quote of a two-year local-vol Phoenix on a count of paths that fills no block evenly
        {"name": "phoenix_quote", "family": "phoenix", "model": "lv", "names": 1, "paths": 20002, "years": 2,
         "table": "grid", "precision": "fp32", "keep_plan": False},
        # the local-vol Phoenix at its benchmark size, on a plan that the pricing program keeps
        {"name": "phoenix_lv", "family": "phoenix", "model": "lv", "names": 1, "paths": 2**20, "years": 3,
         "table": "grid", "precision": "fp32", "keep_plan": True},
        # the same product on the rows a plan tabulates (801 points for every step), priced in one call
        {"name": "phoenix_rows", "family": "phoenix", "model": "lv", "names": 1, "paths": 400000, "years": 2,
         "table": "rows", "precision": "fp32", "keep_plan": False},
        # the worst of three names
        {"name": "worst_of_3", "family": "phoenix", "model": "lv", "names": 3, "paths": 500000, "years": 3,
         "table": "grid", "precision": "fp32", "keep_plan": True},
        # the path engine as the structured-products packages call it: quarterly columns and a daily window
        {"name": "paths_lv", "family": "paths", "model": "lv", "names": 1, "paths": 200000, "years": 3,
         "window": True, "precision": "fp32"},
        # a basket of two stochastic-local-vol names, columns only
        {"name": "paths_slv", "family": "paths", "model": "slv", "names": 2, "paths": 60002, "years": 1,
         "window": False, "precision": "fp32"},
        # the Phoenix as a payoff script, compiled once
        {"name": "script_phoenix", "family": "script", "paths": 2**19, "years": 3, "table": "grid",
         "precision": "fp32"},
        # price, deltas and node vegas of a worst-of: the forward and the backward pass
        {"name": "greeks_worst_of", "family": "greeks", "names": 3, "paths": 2**17, "years": 4,
         "precision": "fp32"},
        # a stochastic-local-vol calibration
        {"name": "leverage", "family": "leverage", "particles": 200000, "years": 1, "precision": "fp32"},
        # a risk revaluation: a small book under spot and vol scenarios, uploaded and captured once
        {"name": "book", "family": "book", "trades": 32, "log2_lo": 12, "log2_hi": 16, "vol_moves": 8,
         "precision": "fp32"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["qe", "phoenix", "phoenix", "phoenix", "paths", "paths", "script", "greeks", "leverage",
                         "book"])
    if family == "qe":
        return {"family": family, "paths": 2 * _log_uniform(rng, 2**10, 2**16), "steps": rng.randint(12, 504),
                "precision": rng.choice(["fp64", "fp64", "fp32"])}
    if family == "phoenix":
        precision = rng.choice(["fp32", "fp32", "fp32", "fp64"])
        model = rng.choice(["lv", "lv", "lv", "heston", "slv"])
        names = rng.randint(1, 5) if model == "lv" else rng.randint(1, 3)
        most = 2**19 if precision == "fp32" else 2**15
        return {"family": family, "model": model, "names": names, "paths": 2 * _log_uniform(rng, 2**10, most // names),
                "years": rng.randint(1, 3), "table": rng.choice(["grid", "rows"]), "precision": precision,
                "keep_plan": rng.random() < 0.5}
    if family == "paths":
        model = rng.choice(["lv", "lv", "heston", "slv"])
        names = rng.randint(1, 3)
        return {"family": family, "model": model, "names": names, "paths": 2 * _log_uniform(rng, 2**10, 2**17 // names),
                "years": rng.randint(1, 3), "window": rng.random() < 0.5,
                "precision": rng.choice(["fp32", "fp32", "fp64"])}
    if family == "script":
        return {"family": family, "paths": 2 * _log_uniform(rng, 2**10, 2**18), "years": rng.randint(1, 3),
                "table": rng.choice(["grid", "rows"]), "precision": "fp32"}
    if family == "greeks":
        return {"family": family, "names": rng.randint(1, 4), "paths": 2 * _log_uniform(rng, 2**11, 2**16),
                "years": rng.randint(1, 4), "precision": "fp32"}
    if family == "leverage":
        return {"family": family, "particles": 2 * _log_uniform(rng, 2**13, 2**17), "years": rng.randint(1, 3),
                "precision": "fp32"}
    return {"family": family, "trades": rng.randint(6, 24), "log2_lo": 11, "log2_hi": rng.randint(12, 15),
            "vol_moves": rng.randint(1, 8), "precision": "fp32"}


# ----------------------------------------------------------------------------------------------------- the inputs


def _market(rng):
    return workloads.FlatMarket(100.0, float(rng.uniform(0.0, 0.04)), float(rng.uniform(0.0, 0.03)))


def _heston(rng):
    return (float(rng.uniform(0.03, 0.06)), float(rng.uniform(1.0, 2.0)), float(rng.uniform(0.03, 0.06)),
            float(rng.uniform(0.4, 0.6)), float(rng.uniform(-0.8, -0.5)))


def _surface(rng, horizon):
    T = horizon * np.arange(1, 41) / 40
    return surfaces.SSVI.power_law(float(rng.uniform(-0.7, -0.4)), 1.0, 0.5, T, float(rng.uniform(0.03, 0.06)) * T)


def _mc_seed(rng):
    return int(rng.integers(1, 2**62))


def _tables(rng, names, years, table, dt, t0):
    """(step_row, lo, inv_dx, rows, n_x) of the names' surfaces: 40 expiries x 200 points, or 801 points a step."""
    step_row, lo, inv, rows, at = [], [], [], [], 0
    for _ in range(names):
        s = _surface(rng, float(years))
        if table == "grid":
            g = workloads.lv_grid(s, horizon=float(years))
            block, row_of = (g.lo, g.inv_dx, g.rows), g.row_of(t0)
        else:
            block, row_of = surfaces.local_var_rows(s, t0, ob.N_X), np.arange(len(t0))
        step_row.append(row_of + at)
        at += len(block[0])
        lo.append(block[0]), inv.append(block[1]), rows.append(block[2])
    return np.stack(step_row).astype(np.int32), np.concatenate(lo), np.concatenate(inv), np.vstack(rows)


def _corr(rng, names):
    rho = float(rng.uniform(0.3, 0.7))
    return np.full((names, names), rho) + (1.0 - rho) * np.eye(names)


def _phoenix_sim(case, seed):
    """The arguments of a Phoenix's `mc_request`, and the market."""
    rng = np.random.default_rng(seed)
    names, years, model = case["names"], case["years"], case.get("model", "lv")
    m = _market(rng)
    dt, t0 = workloads.uniform_grid(float(years), years * STEPS_PER_YEAR)
    t_end = np.concatenate([[0.0], t0 + dt])
    args = {
        "model": OB_MODEL_PATHS, "dt": dt, "t0": t0, "spot": np.full(names, m.spot), "n_pairs": case["paths"] // 2,
        "seed": _mc_seed(rng), "root": correlation_root(_corr(rng, names)) if names > 1 else np.eye(1),
        "kind": np.full(names, {"lv": 1, "heston": 2, "slv": 3}[model], np.int32), "cvar": np.zeros(names),
        "log_fwd": np.tile(m.log_fwd(t_end), (names, 1)),
    }
    if model != "lv":
        args["heston"] = np.array([_heston(rng) for _ in range(names)])
    if model != "heston":
        step_row, lo, inv, rows = _tables(rng, names, years, case.get("table", "grid"), dt, t0)
        if model == "slv":  # the leverage squared: the local variance over the variance's long-run mean
            rows = rows / 0.045
        args |= {"step_row": step_row, "lo": lo, "inv_dx": inv, "table": rows, "n_x": rows.shape[1]}
    ph = workloads.Phoenix(years=float(years))
    args |= workloads.autocall_fields(ph, m, STEPS_PER_YEAR)
    return args, m


def _ladder(case, seed):
    rng = np.random.default_rng(seed)
    m = _market(rng)
    steps = case["steps"]
    T = steps / STEPS_PER_YEAR
    dt, t0 = workloads.uniform_grid(T, steps)
    strikes = np.append(np.arange(80.0, 120.0 + 1e-9, 4.0), 100.0)
    barrier = np.zeros(len(strikes), np.int32)
    barrier[-1] = BARRIER["up-out"]
    level = np.zeros(len(strikes))
    level[-1] = 130.0
    return {
        "model": OB_MODEL_HESTON_QE, "dt": dt, "t0": t0, "spot": [m.spot], "n_pairs": case["paths"] // 2,
        "seed": _mc_seed(rng), "heston": _heston(rng), "r": m.r, "q": m.q, "product": OB_PRODUCT_LADDER,
        "leg_type": np.ones(len(strikes), np.int32), "leg_strike": strikes, "leg_barrier": barrier,
        "leg_level": level, "discount": float(m.D(T)),
    }


def _script_text(years):
    """A Phoenix in the payoff language: quarterly coupons with memory, a call, a knock-in watched daily."""
    lines = ["underlying X", "param S0 = 100", "param cb = 0.7", "param cpn = 0.02", "param call = 1.0",
             "param ki = 0.6", "param K = 1.0"]
    n_obs = 4 * years
    for j in range(1, n_obs + 1):
        t = j / 4
        lines.append(f"event t={t!r} pay t={t!r}")
        if j == 1:
            lines.append("  missed = 0")
        lines += ["  perf = X / S0", "  if perf >= cb then", "    pay cpn * (1 + missed) as coupon", "    missed = 0",
                  "  else", "    missed = missed + 1", "  end"]
        if j < n_obs:
            lines += ["  if perf >= call then", "    pay 1 as redemption", "    terminate", "  end"]
        else:
            lines += [f"  knocked = lowest(X, t=0, t={t!r}, n={STEPS_PER_YEAR * years}) < ki * S0",
                      "  if knocked then", "    pay 1 - max(K - perf, 0) as redemption", "  else",
                      "    pay 1 as redemption", "  end"]
        lines.append("end")
    return "\n".join(lines) + "\n"


def _paths_plan(case, seed):
    """(plan, kept observations, windows, seed) of a path-engine call."""
    rng = np.random.default_rng(seed)
    names, years, model = case["names"], case["years"], case["model"]
    markets = [_market(rng) for _ in range(names)]
    models = []
    for _ in range(names):
        h = HestonParams(*_heston(rng))
        if model == "lv":
            models.append(LocalVolModel(_surface(rng, float(years))))
        elif model == "heston":
            models.append(HestonModel(h))
        else:
            t = np.arange(12 * years) / 12.0
            x = np.linspace(-1.0, 1.0, 81) * (0.1 + 0.6 * np.sqrt(t))[:, None]
            models.append(SLVModel(h, Leverage(t, x, 1.0 - 0.25 * np.tanh(2.0 * x) + 0.1 * x * x)))
    if names == 1:
        target, market = models[0], markets[0]
    else:
        labels = [f"n{a}" for a in range(names)]
        target = Basket(labels, dict(zip(labels, models)), dict(zip(labels, markets)), _corr(rng, names))
        market = None
    per = STEPS_PER_YEAR // 4
    if case["window"]:  # every daily step is an observation; the quarterly ones are kept
        times = np.arange(1, STEPS_PER_YEAR * years + 1) / STEPS_PER_YEAR
        keep, windows = np.arange(per - 1, len(times), per), ((0, len(times) - 1),)
    else:
        times = np.arange(1, 4 * years + 1) / 4
        keep, windows = None, ()
    return ob.plan(target, market, times), keep, windows, _mc_seed(rng)


class _Greeks:
    """A worst-of's request, its vega nodes and the adjoint plan a risk program keeps."""

    def __init__(self, case, seed):
        self.args, _ = _phoenix_sim(dict(case, model="lv", table="grid"), seed)
        years, names = case["years"], case["names"]
        self.held = requests.mc_request(**self.args)
        T = years * np.arange(1, 41) / 40
        self.row_name, self.row_T = np.repeat(np.arange(names), 40), np.tile(T, names)
        self.node_T, self.node_k = years * np.arange(1, 11) / 10, np.linspace(-1.0, 0.5, 15)
        self.nodes = VegaNodes(self.row_name, self.row_T, self.args["lo"], self.args["inv_dx"], self.args["n_x"],
                               self.node_T, self.node_k)
        self.plan = AdjointPlan(self.held, SMOOTHING, case["precision"])


def _leverage_inputs(case, seed):
    rng = np.random.default_rng(seed)
    return HestonParams(*_heston(rng)), _surface(rng, 3.0), workloads.FlatMarket(100.0, 0.02, 0.01), _mc_seed(rng)


def _book(case, seed):
    half = (case["vol_moves"] + 1) // 2
    shifts = np.array([0.01, -0.01, 0.02, -0.02])[:half]
    skews = np.array([0.01, -0.01, 0.02, -0.02])[:case["vol_moves"] - half]
    return sample_book(n_trades=case["trades"], seed=seed, paths_log2=(case["log2_lo"], case["log2_hi"]),
                       years=(1, 3), n_surfaces=5, vol_shifts=shifts, skew_tilts=skews)


def prepare(case, seed):
    family = case["family"]
    state = {"case": case}
    if family == "qe":
        state["held"] = requests.mc_request(**_ladder(case, seed))
    elif family == "phoenix":
        state["held"] = requests.mc_request(**_phoenix_sim(case, seed)[0])
        if case["keep_plan"]:
            state["plan"] = engine.McPlan(state["held"], case["precision"])
    elif family == "paths":
        state["plan"], state["keep"], state["windows"], state["seed"] = _paths_plan(case, seed)
    elif family == "script":
        args, m = _phoenix_sim(dict(case, model="lv", names=1), seed)
        comp = script.compile_script(_script_text(case["years"]))
        state["held"] = script.script_request(comp, requests.mc_request(**args), lambda t: float(m.D(t)))
    elif family == "greeks":
        state["greeks"] = _Greeks(case, seed)
    elif family == "leverage":
        state["inputs"] = _leverage_inputs(case, seed)
    else:
        state["batch"] = Batch(_book(case, seed), case["precision"])
        state["batch"].capture()
    return state


def run(state):
    case = state["case"]
    family = case["family"]
    if family in ("qe", "phoenix"):
        if "plan" in state:
            state["plan"].run(case["paths"] // 2)
            price, se = requests.result_arrays(state["plan"].result())
        else:
            price, se = requests.result_arrays(engine.mc_price(state["held"], case["precision"]))
        return {"price": price, "se": se}
    if family == "paths":
        spots, extremes, _ = ob.run(state["plan"], case["paths"] // 2, state["seed"], keep=state["keep"],
                                    windows=state["windows"], precision=case["precision"])
        return {"spots": spots, "extremes": extremes}
    if family == "script":
        r = script.run(state["held"], case["precision"])
        return {"price": r.price, "se": r.se}
    if family == "greeks":
        g = state["greeks"]
        out = autocall_greeks(g.held, g.nodes, SMOOTHING, case["precision"], plan=g.plan)
        return {k: out[k] for k in ("price", "price_se", "delta", "delta_se", "vega", "vega_se")}
    if family == "leverage":
        params, surface, market, seed = state["inputs"]
        slv = ob.calibrate_leverage(params, surface, market, float(case["years"]), n_particles=case["particles"],
                                    rng=seed, precision=case["precision"])
        return {"x_grids": slv.leverage.x_grids, "values": slv.leverage.values}
    state["batch"].launch()
    price, se, _ = state["batch"].result()
    return {"price": price, "se": se}


def work(case):
    """Operations (integer ones of the generator included) and bytes (inputs once, results once) of one call. Per
    name, path and step: half a normal draw of a pair's two legs (about 20 operations) and the step (about 20 under
    local vol, 35 with a variance process, 200 in 64 bits for the quadratic-exponential scheme)."""
    family = case["family"]
    if family == "qe":
        return {"bytes": 8 * 64, "flops": 220.0 * case["paths"] * case["steps"]}
    if family == "leverage":
        steps = 100 * case["years"] + 60
        return {"bytes": 8.0 * steps * (801 + 2 * 81), "flops": 100.0 * case["particles"] * steps}
    if family == "book":
        mean = 2.0 ** (0.5 * (case["log2_lo"] + case["log2_hi"]))
        return {"bytes": 8.0 * 5 * 40 * 200 * (1 + case["vol_moves"]),
                "flops": 40.0 * case["trades"] * mean * 504 * 2.5 * (1 + 0.75 * case["vol_moves"])}
    names, steps = case.get("names", 1), case["years"] * STEPS_PER_YEAR
    rows = 0 if case.get("model") == "heston" else steps * 801 if (case.get("table") == "rows" or family == "paths") \
        else 40 * 200
    per = 40.0 if case.get("model", "lv") == "lv" else 75.0
    w = {"bytes": 8.0 * names * rows, "flops": per * case["paths"] * steps * names}
    if family == "paths":
        w["bytes"] += 8.0 * names * case["paths"] * (4 * case["years"] + (2 if case["window"] else 0))
    if family == "greeks":  # the states written and read back, the sweep's step
        w["bytes"] += 8.0 * names * case["paths"] * steps
        w["flops"] *= 1.75
    return w


# ------------------------------------------------------------------------------------------------ exact, in 64 bits


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _philox(pair, block, tag, seed):
    """The four 32-bit outputs (as int64) of Philox4x32-10 for counter (pair, block | tag << 32), key seed."""
    mask = 0xFFFFFFFF
    x, y = pair & mask, pair >> 32
    z, w = torch.full_like(pair, block & mask), torch.full_like(pair, (block >> 32) | tag)
    k0, k1 = seed & mask, seed >> 32
    for _ in range(10):
        p0, p1 = x * 0xD2511F53, z * 0xCD9E8D57  # 64-bit products, wrapping: only their bits are used
        x, y, z, w = ((p1 >> 32) & mask) ^ y ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ w ^ k1, p0 & mask
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return x, y, z, w


def _box_muller(a, b):
    u, v = (a.double() + 0.5) * 2.0**-32, (b.double() + 0.5) * 2.0**-32
    r, t = torch.sqrt(-2.0 * torch.log(u)), 2.0 * math.pi * v
    return r * torch.cos(t), r * torch.sin(t)


class _Stream:
    """A pair's normals in order, for every pair at once."""

    def __init__(self, pair, seed, tag=0):
        self.pair, self.seed, self.tag, self.block, self.left = pair, seed, tag, 0, []

    def next(self):
        if not self.left:
            a, b, c, d = _philox(self.pair, self.block, self.tag, self.seed)
            self.left = [*_box_muller(a, b), *_box_muller(c, d)]
            self.block += 1
        return self.left.pop(0)


def _pairs(n):
    return torch.arange(n, dtype=torch.int64, device=_device())


def _legs(z):
    return torch.stack([z, -z])


def _cell(lo, inv, n_x, x):
    """Interval and weight of x in a row of n_x uniform points, clamped as the engine clamps it."""
    u = ((x - lo) * inv).clamp(0.0, n_x - 1 - 1e-4)
    j = u.long()
    return j, u - j


def _walk(sim, normals=None):
    """Yields (step end, x) with x (names, 2 legs, pairs) the log of S / F, step by step (log-Euler; a Heston variance
    by full truncation)."""
    names, pairs = len(sim["kind"]), sim["n_pairs"]
    kind = int(sim["kind"][0])
    dev = _device()
    root = sim["root"]
    main, aux = _Stream(_pairs(pairs), sim["seed"]), _Stream(_pairs(pairs), sim["seed"], 0x80000000)
    x = torch.zeros((names, 2, pairs), dtype=torch.float64, device=dev)
    h = np.asarray(sim["heston"], float).reshape(names, 5) if kind >= 2 else None
    v = [torch.full((2, pairs), float(h[a][0]), dtype=torch.float64, device=dev) for a in range(names)] if kind >= 2 else None
    table = torch.tensor(sim["table"], dtype=torch.float64, device=dev).reshape(-1) if kind != 2 else None
    yield 0, x
    for i, dt in enumerate(np.asarray(sim["dt"], float)):
        z = [main.next() for _ in range(names)]
        zr = [(aux if kind == 3 else main).next() for _ in range(names)] if kind >= 2 else None
        new = []
        for a in range(names):
            za = _legs(sum(float(root[a][b]) * z[b] for b in range(names)))
            if kind != 2:
                row = int(sim["step_row"][a][i])
                n_x = sim["n_x"]
                j, w = _cell(float(sim["lo"][row]), float(sim["inv_dx"][row]), n_x, x[a])
                y = table[row * n_x + j]
                var = y + w * (table[row * n_x + j + 1] - y)
            if kind >= 2:
                _, kappa, theta, xi, rho = (float(p) for p in h[a])
                vp = v[a].clamp(min=0.0)
                var = vp if kind == 2 else var * vp
                wa = _legs(sum(float(root[a][b]) * zr[b] for b in range(names)))
                v[a] = v[a] + kappa * (theta - vp) * dt + xi * torch.sqrt(vp * dt) * (rho * za + math.sqrt(1 - rho * rho) * wa)
            new.append(x[a] - 0.5 * dt * var + torch.sqrt(var * dt) * za)
        x = torch.stack(new)
        yield i + 1, x


def _estimate(y):
    """(price, standard error) of pair values (outputs, pairs), as the engine estimates them."""
    n = y.shape[1]
    mean = y.mean(1)
    var = ((y * y).mean(1) - mean * mean).clamp(min=0.0)
    return mean.cpu().numpy(), torch.sqrt(var / (n - 1)).cpu().numpy()


def _exact_phoenix(sim):
    """The Phoenix's four outputs: value, called, knocked in, coupons."""
    at = {int(s): j for j, s in enumerate(sim["obs_step"])}
    last = len(at) - 1
    low = pv = missed = alive = called = knocked = coupons = None
    for i, x in _walk(sim):
        if i == 0:
            zero = torch.zeros_like(x[0])
            low, pv, missed, called, knocked, coupons = (zero.clone() for _ in range(6))
            alive = zero == 0
            continue
        lf = torch.tensor(np.asarray(sim["log_fwd"])[:, i], device=x.device)[:, None, None]
        lp = (x + lf).min(0).values
        low = torch.minimum(low, lp)
        if i not in at:
            continue
        j = at[i]
        D = float(sim["obs_discount"][j])
        hit = alive & (lp >= math.log(sim["coupon_barrier"]))
        times = 1.0 + missed
        pv = pv + torch.where(hit, D * sim["coupon"] * times, zero)
        coupons = coupons + torch.where(hit, times, zero)
        missed = torch.where(hit, zero, missed + 1.0)
        if j < last:
            call = alive & (lp >= math.log(sim["trigger"][j]))
            pv, called, alive = pv + torch.where(call, D, 0.0), called + call, alive & ~call
        else:
            ki = alive & (low < math.log(sim["ki_barrier"]))
            put = (sim["put_strike"] - torch.exp(lp)).clamp(min=0.0)
            pv = pv + torch.where(alive, D * (1.0 - torch.where(ki, put, zero)), zero)
            knocked = knocked + ki
    return torch.stack([t.mean(0) for t in (pv, called, knocked, coupons)])


def _exact_ladder(sim):
    """The ladder's payments and the mean spot under Andersen's quadratic-exponential scheme, martingale-corrected."""
    v0, kappa, theta, xi, rho = sim["heston"]
    dt, mu = float(sim["dt"][0]), sim["r"] - sim["q"]
    E = math.exp(-kappa * dt)
    k12 = 0.5 * dt * (kappa * rho / xi - 0.5)
    c1, c2 = xi * xi * E * (1 - E) / kappa, theta * xi * xi * (1 - E) ** 2 / (2 * kappa)
    K1, K2, K3 = k12 - rho / xi, k12 + rho / xi, 0.5 * dt * (1 - rho * rho)
    A, K0_plain = K2 + 0.5 * K3, -rho * kappa * theta * dt / xi
    stream = _Stream(_pairs(sim["n_pairs"]), sim["seed"])
    y = torch.zeros((2, sim["n_pairs"]), dtype=torch.float64, device=_device())
    v = torch.full_like(y, v0)
    top = torch.full_like(y, -math.inf)
    for _ in range(len(sim["dt"])):
        zv, zx = _legs(stream.next()), _legs(stream.next())
        m = theta + (v - theta) * E
        psi = (v * c1 + c2) / (m * m)
        quad = psi <= 1.5
        inv = 2.0 / torch.where(quad, psi, torch.ones_like(psi))
        b2 = inv - 1.0 + torch.sqrt(inv) * torch.sqrt((inv - 1.0).clamp(min=0.0))
        a, b = m / (1.0 + b2), torch.sqrt(b2)
        arg_q = 1.0 - 2.0 * A * a
        p = (psi - 1.0) / (psi + 1.0)
        beta = (1.0 - p) / m
        tail = torch.special.ndtr(-zv)
        jump = torch.where(tail >= 1.0 - p, torch.zeros_like(v), torch.log((1.0 - p) / tail) / beta)
        arg_e = p + beta * (1.0 - p) / (beta - A)
        vn = torch.where(quad, a * (b + zv) ** 2, jump)
        fine = torch.where(quad, arg_q > 0.0, beta > A)
        K0 = torch.where(quad, -A * b2 * a / arg_q + 0.5 * torch.log(arg_q), -torch.log(arg_e)) - (K1 + 0.5 * K3) * v
        K0 = torch.where(fine, K0, torch.full_like(K0, K0_plain))
        y = y + mu * dt + K0 + K1 * v + K2 * vn + torch.sqrt((K3 * (v + vn)).clamp(min=0.0)) * zx
        v = vn
        top = torch.maximum(top, y)
    S = float(sim["spot"][0]) * torch.exp(y)
    out = []
    for K, bar, level in zip(sim["leg_strike"], sim["leg_barrier"], sim["leg_level"]):
        pay = sim["discount"] * (S - K).clamp(min=0.0)
        if bar:
            pay = torch.where(top >= math.log(level / float(sim["spot"][0])), torch.zeros_like(pay), pay)
        out.append(pay.mean(0))
    return torch.stack([*out, S.mean(0)])


def _exact_paths(case, seed):
    p, keep, windows, mc_seed = _paths_plan(case, seed)
    sim = {"kind": p.kind, "n_pairs": case["paths"] // 2, "seed": mc_seed, "root": p.root, "heston": p.heston,
           "dt": p.dt, "step_row": p.step_row, "lo": p.lo, "inv_dx": p.inv_dx, "table": p.table, "n_x": p.n_x}
    names = len(p.kind)
    keep = np.arange(p.n_obs) if keep is None else keep
    column = {int(j): c for c, j in enumerate(keep)}
    spots = [np.empty((case["paths"], len(keep)), order="F") for _ in range(names)]
    lows, highs = [[None] * len(windows) for _ in range(names)], [[None] * len(windows) for _ in range(names)]
    obs = {}
    for j, s in enumerate(p.obs_step):
        obs.setdefault(int(s), []).append(j)
    for i, x in _walk(sim):
        for j in obs.get(i, ()):
            for a in range(names):
                S = (float(p.fwd[a][j]) * torch.exp(x[a])).reshape(-1)
                if j in column:
                    spots[a][:, column[j]] = S.cpu().numpy()
                for k, (first, last) in enumerate(windows):
                    if first <= j <= last:
                        lows[a][k] = S if j == first else torch.minimum(lows[a][k], S)
                        highs[a][k] = S if j == first else torch.maximum(highs[a][k], S)
    extremes = [[(lows[a][k].cpu().numpy(), highs[a][k].cpu().numpy()) for k in range(len(windows))]
                for a in range(names)]
    return {"spots": spots, "extremes": extremes}


def _ramp(d, scale):
    return (d / scale + 0.5).clamp(0.0, 1.0)


def _smooth_phoenix(sim, lp, low):
    """The Phoenix's value on each leg with its digitals smoothed: lp (observations, 2, pairs), low (2, pairs)."""
    eps, last = SMOOTHING, lp.shape[0] - 1
    cb, ki, K = sim["coupon_barrier"], sim["ki_barrier"], sim["put_strike"]
    pv, alive, missed = 0.0, torch.ones_like(low), torch.zeros_like(low)
    for j in range(last + 1):
        p, D = torch.exp(lp[j]), float(sim["obs_discount"][j])
        c = _ramp(p - cb, eps * cb)
        pv = pv + D * sim["coupon"] * (1.0 + missed) * c * alive
        missed = (1.0 - c) * (missed + 1.0)
        if j < last:
            q = _ramp(p - sim["trigger"][j], eps * sim["trigger"][j])
            pv, alive = pv + D * q * alive, alive * (1.0 - q)
        else:
            pv = pv + D * alive * (1.0 - _ramp(ki - torch.exp(low), eps * ki) * (K - p).clamp(min=0.0))
    return pv


def _tents(points, nodes):
    """(points, nodes) weights of linear interpolation on the nodes, flat beyond the ends."""
    x = np.clip(points, nodes[0], nodes[-1])
    j = np.clip(np.searchsorted(nodes, x, side="right") - 1, 0, len(nodes) - 2)
    f = (x - nodes[j]) / (nodes[j + 1] - nodes[j])
    w = np.zeros((len(x), len(nodes)))
    w[np.arange(len(x)), j] = 1.0 - f
    w[np.arange(len(x)), j + 1] += f
    return torch.tensor(w, device=_device())


def _exact_greeks(case, seed):
    g, _ = _phoenix_sim(dict(case, model="lv", table="grid"), seed)
    names, steps, pairs, n_x = case["names"], len(g["dt"]), g["n_pairs"], g["n_x"]
    dev = _device()
    states = torch.empty((steps + 1, names, 2, pairs), dtype=torch.float64, device=dev)
    at = {int(s): j for j, s in enumerate(g["obs_step"])}
    lp_obs = torch.empty((len(at), 2, pairs), dtype=torch.float64, device=dev)
    who_obs = torch.empty((len(at), 2, pairs), dtype=torch.int64, device=dev)
    low = torch.zeros((2, pairs), dtype=torch.float64, device=dev)
    low_step, low_name = torch.zeros_like(low, dtype=torch.int64), torch.zeros_like(low, dtype=torch.int64)
    for i, x in _walk(g):
        states[i] = x
        if i == 0:
            continue
        lf = torch.tensor(np.asarray(g["log_fwd"])[:, i], device=dev)[:, None, None]
        lp, who = (x + lf).min(0)
        less = lp < low
        low, low_step = torch.where(less, lp, low), torch.where(less, i, low_step)
        low_name = torch.where(less, who, low_name)
        if i in at:
            lp_obs[at[i]], who_obs[at[i]] = lp, who
    lp_obs.requires_grad_(True), low.requires_grad_(True)
    value = _smooth_phoenix(g, lp_obs, low)
    d_obs, d_low = torch.autograd.grad(value.sum(), (lp_obs, low))
    d_obs, d_low, value = 0.5 * d_obs, 0.5 * d_low, value.detach()
    delta = []
    for a in range(names):
        per = (d_obs * (who_obs == a)).sum(0) + d_low * (low_name == a)
        delta.append(per.sum(0))
    mean, se = _estimate(value.mean(0)[None, :])
    d_mean, d_se = _estimate(torch.stack(delta))
    table = torch.tensor(g["table"], dtype=torch.float64, device=dev).reshape(-1)
    grad = torch.zeros_like(table)
    back = torch.zeros((names, 2, pairs), dtype=torch.float64, device=dev)
    for i in range(steps, 0, -1):
        for a in range(names):
            if i in at:
                back[a] += d_obs[at[i]] * (who_obs[at[i]] == a)
            back[a] += d_low * ((low_step == i) & (low_name == a))
            row = int(g["step_row"][a][i - 1])
            lo, inv = float(g["lo"][row]), float(g["inv_dx"][row])
            x, x_new, hdt = states[i - 1, a], states[i, a], -0.5 * float(g["dt"][i - 1])
            u = (x - lo) * inv
            inside = (u > 0.0) & (u < n_x - 1 - 1e-4)
            j, w = _cell(lo, inv, n_x, x)
            y, dy = table[row * n_x + j], table[row * n_x + j + 1] - table[row * n_x + j]
            var = y + w * dy
            vb = back[a] * (hdt + (x_new - x - var * hdt) / (2.0 * var))
            at_left = (row * n_x + j).reshape(-1)
            grad.index_add_(0, at_left, (vb * (1.0 - w)).reshape(-1))
            grad.index_add_(0, at_left + 1, (vb * w).reshape(-1))
            back[a] += torch.where(inside, vb * dy * inv, torch.zeros_like(vb))
    years = case["years"]
    T, node_T = years * np.arange(1, 41) / 40, years * np.arange(1, 11) / 10
    phi = _tents(T, node_T)
    h = (2.0 * torch.sqrt(table) * grad / pairs).reshape(names, 40, n_x)
    vega = torch.zeros((names, 10, 15), dtype=torch.float64, device=dev)
    for a in range(names):
        for e in range(40):
            r = a * 40 + e
            k = float(g["lo"][r]) + np.arange(n_x) / float(g["inv_dx"][r])
            vega[a] += phi[e][:, None] * (h[a, e] @ _tents(k, np.linspace(-1.0, 0.5, 15)))[None, :]
    spot = np.asarray(g["spot"], float)
    # the vegas' standard errors come from how the pairs fall into batches, which is the engine's own affair
    return {"price": float(mean[0]), "price_se": float(se[0]), "delta": d_mean / spot, "delta_se": d_se / spot,
            "vega": vega.cpu().numpy(), "vega_se": None}


def _exact_leverage(case, seed):
    """The particle method in 64 bits with the request's grid: histogram quantiles, a Nadaraya-Watson regression over
    bins, an Euler step."""
    params, surface, _, mc_seed = _leverage_inputs(case, seed)
    dev = _device()
    n_x, n_bins, n_fine, pairs = 81, 400, 8192, case["particles"] // 2
    from optlab_b200.models import time_grid

    grid = time_grid([float(case["years"])], 1 / 100, 1 / 2000)
    dt, t0 = np.diff(grid), grid[:-1]
    lv_lo, lv_inv, lv_rows = surfaces.local_var_rows(surface, t0, ob.N_X)
    T1 = min(1.0, float(surface.maturities[-1]))
    atm = float(np.sqrt(surface.theta(T1) / T1))
    pair, n = _pairs(pairs), 2.0 * pairs
    x = torch.zeros((2, pairs), dtype=torch.float64, device=dev)
    v = torch.full_like(x, params.v0)
    steps = torch.arange(n_x, device=dev, dtype=torch.float64) / (n_x - 1)
    out_x, out_v = np.empty((len(dt), n_x)), np.empty((len(dt), n_x))

    def interp(at, a, b, y):
        u = (at - a) / (b - a) * (len(y) - 1)
        j = u.clamp(0, len(y) - 1).long().clamp(max=len(y) - 2)
        w = u - j
        inside = y[j] * (1 - w) + y[j + 1] * w
        return torch.where(u > 0, torch.where(u >= len(y) - 1, y[-1], inside), y[0])

    for i, h in enumerate(dt):
        if i == 0:
            xe = (-6.0 + 12.0 * steps) * atm * math.sqrt(max(h, 1e-4))
            cond = torch.full_like(xe, params.v0)
        else:
            lo, hi = float(x.min()), float(x.max())
            width = (hi - lo) / n_fine
            fine = torch.bincount(((x - lo) / width).long().clamp(0, n_fine - 1).reshape(-1), minlength=n_fine).double()
            cum, ends = torch.cumsum(fine, 0), []
            for q in (0.0005, 0.9995):
                k = int(((cum >= q * n) & (fine > 0)).nonzero()[0])
                ends.append(lo + (k + (q * n - float(cum[k] - fine[k])) / float(fine[k])) * width)
            xe = ends[0] + (ends[1] - ends[0]) * steps
            wc = (hi + 1e-12 - lo) / n_bins
            k = ((x - lo) / wc).long().clamp(0, n_bins - 1).reshape(-1)
            count = torch.bincount(k, minlength=n_bins).double()
            v_sum = torch.zeros(n_bins, dtype=torch.float64, device=dev).index_add_(0, k, v.reshape(-1))
            centres = lo + (torch.arange(n_bins, device=dev) + 0.5) * wc
            bw = atm * math.sqrt(max(t0[i], 0.15)) * n**-0.2
            weight = torch.exp(-0.5 * ((xe[:, None] - centres[None, :]) / bw) ** 2)
            mass = weight @ count
            cond = torch.where(mass > 1e-8, (weight @ v_sum) / mass.clamp(min=1e-300), v.sum() / n)
        row = torch.tensor(lv_rows[i], device=dev)
        loc = interp(xe, lv_lo[i], lv_lo[i] + (ob.N_X - 1) / lv_inv[i], row)
        lev = torch.sqrt(loc / cond.clamp(min=1e-8)).clamp(0.05, 8.0)
        out_x[i], out_v[i] = xe.cpu().numpy(), lev.cpu().numpy()
        a, b, _, _ = _philox(pair, i + 1, 0, mc_seed)
        z1, z2 = (_legs(z) for z in _box_muller(a, b))
        L = interp(x, xe[0], xe[-1], lev)
        vp = v.clamp(min=0.0)
        var = L * L * vp
        zx = params.rho * z2 + math.sqrt(1 - params.rho**2) * z1
        v = v + params.kappa * (params.theta - vp) * h + params.xi * torch.sqrt(vp * h) * z2
        x = x - 0.5 * var * h + torch.sqrt(var * h) * zx
    return {"x_grids": out_x, "values": out_v}


def exact(case, seed):
    family = case["family"]
    if family == "book":
        return None  # some hundreds of simulations: minutes in plain torch
    if family == "paths":
        return _exact_paths(case, seed)
    if family == "greeks":
        return _exact_greeks(case, seed)
    if family == "leverage":
        return _exact_leverage(case, seed)
    if family == "qe":
        y = _exact_ladder(_ladder(case, seed))
    else:
        y = _exact_phoenix(_phoenix_sim(dict(case, names=case.get("names", 1)), seed)[0])
    price, se = _estimate(y)
    if family == "script":
        return {"price": float(price[0]), "se": float(se[0])}
    return {"price": price, "se": se}
