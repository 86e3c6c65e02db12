"""Performance cases of the pricing engine: the work a user's program has it do,
through its public entry points (``price_plain``, ``price_batch``, ``PreparedBatch``,
``Server``, ``MCDispatcher``).

Sizes are those of ``quantkos_b200.workloads``, of the tests and of ``bench.py``, or
generic.  Contracts are built from the seed: the Philox key, the strike and the market
and model parameters.  Results of an FP32 contract are returned as float32 (its paths
are simulated in FP32), those of an FP64 contract as float64.  Finite-difference Greeks
are asked for in FP64, the precision a configuration file gets unless it says
otherwise: the second differences of FP32 prices (gamma, vomma, vanna) are of the order
of the FP32 rounding of the paths.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import quantkos_b200 as qk
from quantkos_b200 import workloads as W

MODELS = {"heston": qk.HESTON, "bates": qk.BATES}
SCHEMES = {"euler": qk.EULER, "milstein": qk.IMPLICIT_MILSTEIN, "qe": qk.ANDERSEN_QE}


def listed():
    return [
        # one small quote: a few launches, a copy each way and the host's planning
        {"name": "quote_small_fp64", "kind": "batch", "model": "heston", "scheme": "euler", "fp64": True,
         "legs": "european", "paths": 10_007, "steps": 12, "greeks": False, "antithetic": False},
        # a desk repricing the same two-leg contract on every market tick (graph replay)
        {"name": "reprice_prepared_fp32", "kind": "prepared", "model": "heston", "scheme": "qe", "fp64": False,
         "legs": "european_asian", "paths": 200_000, "steps": 64, "greeks": False, "antithetic": False},
        # a configuration file run as the reference runs it: FP64, payoff percentiles
        {"name": "dispatcher_fp64", "kind": "dispatcher", "model": "heston", "scheme": "qe", "fp64": True,
         "legs": "asian", "paths": 100_000, "steps": 128, "greeks": False, "antithetic": False},
        # the plain method on one European call (1,048,576 x 252, Heston Euler)
        {"name": "plain_euler_1m", "kind": "plain", "model": "heston", "scheme": "euler", "fp64": True,
         "legs": "european", "paths": 1_048_576, "steps": 252, "greeks": False, "antithetic": False},
        # the plain method with every Greek by bump and reprice: 12 pricings of a ragged path count
        {"name": "plain_qe_asian_greeks", "kind": "plain", "model": "bates", "scheme": "qe", "fp64": True,
         "legs": "asian", "paths": 100_003, "steps": 126, "greeks": True, "antithetic": False},
        # five payoffs of one Bates-QE pass in FP32 (16,777,216 x 252)
        {"name": "bates_qe_five_16m", "kind": "batch", "model": "bates", "scheme": "qe", "fp64": False,
         "legs": "five", "paths": 16_777_216, "steps": 252, "greeks": False, "antithetic": False},
        # the reference's published benchmark: Heston-QE arithmetic Asian call, 5,000,000 x 365
        {"name": "asian_qe_5m_365", "kind": "batch", "model": "heston", "scheme": "qe", "fp64": False,
         "legs": "asian", "paths": 5_000_000, "steps": 365, "greeks": False, "antithetic": False},
        # American put by Longstaff-Schwartz, six-term basis, 50 dates, FP32
        {"name": "american_4m_fp32", "kind": "american", "model": "heston", "scheme": "qe", "fp64": False,
         "basis": "poly", "paths": 4_194_304, "steps": 250, "dates": 50},
        # the reference's own American mode: Laguerre basis, every step a date, FP64
        {"name": "american_laguerre_fp64", "kind": "american", "model": "heston", "scheme": "milstein", "fp64": True,
         "basis": "laguerre", "paths": 300_001, "steps": 100, "dates": 0},
        # an overnight book of mixed contracts in FP32
        {"name": "book_fp32", "kind": "book", "fp64": False, "contracts": 32, "paths_lo": 100_000,
         "paths_hi": 2_000_000, "greeks": False},
        # a small book with all Greeks in FP64 (96 pricing tasks in one call)
        {"name": "book_fp64_greeks", "kind": "book", "fp64": True, "contracts": 8, "paths_lo": 10_000,
         "paths_hi": 200_000, "greeks": True},
        # a burst of requests to a running server, 30% American
        {"name": "serve_burst_fp32", "kind": "serve", "fp64": False, "contracts": 48, "paths_lo": 100_000,
         "paths_hi": 2_000_000, "greeks": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["batch", "batch", "plain", "plain", "prepared", "american", "book", "dispatcher"])
    if kind == "book":
        fp64 = rng.random() < 0.5
        return {"kind": kind, "fp64": fp64, "contracts": rng.randint(2, 8) if fp64 else rng.randint(8, 32),
                "paths_lo": 10_000 if fp64 else 100_000, "paths_hi": 200_000 if fp64 else _log_int(rng, 2e5, 2e6),
                "greeks": fp64 and rng.random() < 0.7}
    model, scheme = rng.choice(sorted(MODELS)), rng.choice(sorted(SCHEMES))
    if kind == "american":
        if rng.random() < 0.5:
            return {"kind": kind, "model": model, "scheme": scheme, "fp64": False, "basis": "poly",
                    "paths": _log_int(rng, 1e6, 4e6), "steps": 50 * rng.randint(1, 5), "dates": 50}
        dates = rng.choice([0, 10, 25])
        return {"kind": kind, "model": model, "scheme": scheme, "fp64": True,
                "basis": rng.choice(["poly", "laguerre"]), "paths": _log_int(rng, 2e4, 5e5),
                "steps": 50 * rng.randint(1, 2), "dates": dates}
    fp64 = kind in ("plain", "dispatcher") or (kind == "batch" and rng.random() < 0.3)
    legs = rng.choice(["european", "asian", "barrier", "binary", "lookback", "european_asian", "five"])
    lo, hi = (1e4, 1e6) if fp64 else (3e5, 8e6)
    if kind == "prepared":
        lo, hi = 2e5, 1e6
    if kind == "dispatcher":
        legs, hi = rng.choice(["european", "asian", "lookback"]), 3e5
    greeks = kind == "plain" and rng.random() < 0.4
    if greeks:
        hi = 2e5
    anti = kind == "batch" and rng.random() < 0.2
    paths = _log_int(rng, lo, hi)
    return {"kind": kind, "model": model, "scheme": scheme, "fp64": fp64, "legs": legs,
            "paths": paths + paths % 2 if anti else paths, "steps": _log_int(rng, 10, 365), "greeks": greeks,
            "antithetic": anti}


# ------------------------------------------------------------------ inputs
def _legs(name, K):
    P = qk.payoff
    five = [P(qk.EUROPEAN, qk.CALL, K), P(qk.ASIAN, qk.CALL, K), P(qk.BARRIER_UP_OUT, qk.CALL, K, 1.3 * K),
            P(qk.LOOKBACK_FLOATING, qk.PUT, K), P(qk.BINARY_CASH, qk.CALL, 1.05 * K)]
    return {"european": five[:1], "asian": five[1:2], "barrier": five[2:3], "lookback": five[3:4],
            "binary": five[4:], "european_asian": five[:2], "five": five}[name]


def _market(case, rng):
    bates = case["model"] == "bates"
    return dict(S0=100.0, v0=float(rng.uniform(0.03, 0.06)), r=0.03, q=0.0, model=MODELS[case["model"]],
                scheme=SCHEMES[case["scheme"]], kappa=2.0, theta=0.04, sigma=float(rng.uniform(0.2, 0.4)),
                rho=float(rng.uniform(-0.8, -0.5)), lambda_j=0.1 if bates else 0.0, mu_j=-0.05, sigma_j=0.1,
                T=case["steps"] / 252.0 if case["steps"] >= 50 else 0.5, n_steps=case["steps"],
                n_paths=case["paths"], seed=int(rng.integers(1, 2 ** 62)),
                precision=qk.FP64 if case["fp64"] else qk.FP32)


def _contracts(case, seed):
    rng = np.random.default_rng([int(seed), 977])
    kind = case["kind"]
    prec = qk.FP64 if case["fp64"] else qk.FP32
    if kind in ("book", "serve"):
        sizes = (case["paths_lo"], case["paths_hi"])
        cs = [W._draw_contract(rng, i, prec, 0.3 if kind == "serve" else 0.0, sizes, (300_000, 2_000_000))
              for i in range(case["contracts"])]
        key = int(rng.integers(1, 2 ** 62))
        for c in cs:
            c.seed = key
        return cs
    m = _market(case, rng)
    K = float(rng.uniform(95.0, 105.0))
    if kind == "american":
        return [qk.make_contract(**m, payoffs=[qk.payoff(qk.AMERICAN, qk.PUT, K)],
                                 lsm_basis=qk.LSM_POLY_SV if case["basis"] == "poly" else qk.LSM_LAGUERRE3,
                                 lsm_dates=case["dates"])]
    return [qk.make_contract(**m, payoffs=_legs(case["legs"], K), antithetic=case["antithetic"])]


class _State:
    """What a user's program keeps between calls."""

    server = prepared = config = None

    def __init__(self, case, seed):
        self.kind, self.fp64 = case["kind"], case["fp64"]
        self.contracts = _contracts(case, seed)
        self.greeks = W.batch_greeks() if case.get("greeks") else None
        if self.kind == "prepared":
            self.handle = qk.Handle(0)  # a prepared set belongs to its handle
            self.prepared = qk.PreparedBatch(self.contracts, self.greeks, self.handle)
        elif self.kind == "serve":
            self.server = qk.Server(hbm_budget_mib=8192)
        elif self.kind == "dispatcher":
            c, cfg = self.contracts[0], qk.UInputs()
            model = "bates" if c.model == qk.BATES else "heston"
            fields = {"S0": c.S0, "v0": c.v0, "r": c.r, "q": c.q, "opt_type": c.payoffs[0].type,
                      "opt_right": c.payoffs[0].right, "K": c.payoffs[0].strike, "model": c.model,
                      "scheme": c.scheme, "t_end": c.T, "inp_dt": c.T / c.n_steps * (1.0 + 1e-9),
                      "n_paths": c.n_paths, "seed": c.seed >> 1 or 1, "analyze_distribution": 1, "paths_file": "",
                      "out_dir": "", "bates_lambda": c.lambda_j, "bates_mu": c.mu_j, "bates_sigma_j": c.sigma_j,
                      model + "_k": c.kappa, model + "_theta": c.theta, model + "_sigma": c.sigma,
                      model + "_rho": c.rho}
            for k, v in fields.items():
                setattr(cfg, k, v)
            self.config = cfg.validate()

    def __del__(self):
        if self.server is not None:
            self.server.stop()


def prepare(case, seed):
    return _State(case, seed)


# ------------------------------------------------------------------ one pass
_FIELDS = ("price", "std_error", "prob_itm")
_GREEKS = ("delta", "gamma", "vega", "vomma", "vanna", "rho", "theta")


def _table(results, fp64, greeks):
    dtype = np.float64 if fp64 else np.float32
    return {f: np.array([leg[f] for r in results for leg in r["legs"]], dtype=dtype)
            for f in _FIELDS + (_GREEKS if greeks else ())}


def run(state):
    if state.kind == "dispatcher":
        res = qk.MCDispatcher(state.config).launch_montecarlo()
        p = res.OptionPrice
        return {"price": np.array([p.option_price]), "std_error": np.array([p.standard_error]),
                "prob_itm": np.array([p.prob_itm]), "percentiles": np.array(list(p.percentiles.values()))}
    if state.kind == "plain" or (state.kind == "american" and state.fp64):
        results = [qk.price_plain(c, state.greeks) for c in state.contracts]
    elif state.kind == "prepared":
        state.prepared.run()
        results = state.prepared.fetch()
    elif state.kind == "serve":
        tickets = [state.server.submit(c) for c in state.contracts]
        results = []
        for t in tickets:
            while (r := state.server.poll(t, 1000)) is None:
                pass
            results.append(r)
    else:
        results = qk.price_batch(state.contracts, state.greeks)
    return _table(results, state.fp64, state.greeks is not None)


# Arithmetic of one path-step (a transcendental function, square root or division counts
# as one operation; the generator's 32-bit integer operations are counted too).
_STEP_FLOPS = {qk.EULER: 55.0, qk.IMPLICIT_MILSTEIN: 58.0, qk.ANDERSEN_QE: 75.0}


def work(case):
    flops = byts = 0.0
    for c in _contracts(case, 0):
        bumps = 12 if case.get("greeks") else 1
        flops += bumps * float(c.n_paths) * c.n_steps * (_STEP_FLOPS[c.scheme] + (4.0 if c.model == qk.BATES else 0.0))
        byts += bumps * 512.0
        if c.payoffs[0].type == qk.AMERICAN:
            # spot (and variance) of every path at every exercise date, written once and read once
            dates = c.lsm_dates or c.n_steps
            per = (2 if c.lsm_basis == qk.LSM_POLY_SV else 1) * (8 if case["fp64"] else 4)
            byts += 2.0 * per * c.n_paths * dates
            flops += 60.0 * c.n_paths * dates
    return {"bytes": byts, "flops": flops}


# ------------------------------------------------------------------ the values in 64 bits
def _mulhilo(m, x):
    p = x * m  # wraps modulo 2^64
    return (p >> 32) & 0xFFFFFFFF, p & 0xFFFFFFFF


def _philox(block, path, stream, domain, key):
    """Philox4x32-10 (Salmon et al., SC'11): counter (block, path, stream, domain)."""
    M0, M1 = 0xD2511F53, 0xCD9E8D57
    M0, M1 = M0 - 2 ** 64 if M0 >= 2 ** 63 else M0, M1
    full = torch.full_like
    x, y, z, w = full(path, block), path, full(path, stream), full(path, domain)
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        h0, l0 = _mulhilo(M0, x)
        h1, l1 = _mulhilo(M1, z)
        x, y, z, w = h1 ^ y ^ k0, l1, h0 ^ w ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return x, y, z, w


def _u01(w, fp64):
    return (w.double() + 0.5) * 2.0 ** -32 if fp64 else ((w >> 9).double() + 0.5) * 2.0 ** -23


def _normals(wa, wb, fp64):
    rad = torch.sqrt(-2.0 * torch.log(_u01(wa, fp64)))
    ang = 2.0 * math.pi * (_u01(wb, fp64) - 0.5)
    return rad * torch.cos(ang), rad * torch.sin(ang)


def _consts(cs, n_steps, eps):
    """Step constants of the contracts `cs` (a base and its bumps), one row each."""
    rows = []
    for c in cs:
        dt = c["T"] / n_steps
        q = c["q"] + (c["lam"] * math.expm1(c["mu"] + 0.5 * c["sj"] ** 2) if c["bates"] else 0.0)
        k, th, sg, rho = c["kappa"], c["theta"], c["sigma"], c["rho"]
        e = math.exp(-k * dt)
        d = {"drift": (c["r"] - q) * dt, "dt": dt, "sdt": math.sqrt(dt), "S0": c["S0"], "v0": c["v0"], "e": e,
             "rho": rho, "rhoc": math.sqrt(1 - rho * rho), "k": k, "th": th, "sg": sg, "iden": 1 / (1 + k * dt)}
        d["tm"] = th * (1 - e)
        d["f1"], d["f2"] = sg * sg * e / k * (1 - e), th * sg * sg / (2 * k) * (1 - e) ** 2
        ros = rho / sg
        g = 0.5 * dt * (k * ros - 0.5)
        d["K1"], d["K2"], d["K3"] = g - ros, g + ros, 0.5 * dt * (1 - rho * rho)
        d["A"] = d["K2"] + 0.5 * d["K3"]
        rows.append(d)
    return {n: torch.tensor([[r[n]] for r in rows], dtype=torch.float64, device="cuda") for n in rows[0]}


def _step(c, scheme, lx, v, Z1, Z2, eps):
    """(log S, v) after one step; rows of the constants against paths."""
    if scheme != qk.ANDERSEN_QE:
        sq = torch.sqrt(v)
        lx = lx + c["drift"] - 0.5 * c["dt"] * v + sq * c["sdt"] * (c["rho"] * Z1 + c["rhoc"] * Z2)
        noise = c["sg"] * c["sdt"] * sq * Z1
        if scheme == qk.EULER:
            vn = v * (1 - c["k"] * c["dt"]) + c["k"] * c["th"] * c["dt"] + noise
        else:
            vn = c["iden"] * (v + c["k"] * c["th"] * c["dt"] + noise + 0.25 * c["sg"] ** 2 * c["dt"] * (Z1 * Z1 - 1))
        return lx, vn.clamp_min(0.0)
    m, s2 = v * c["e"] + c["tm"], v * c["f1"] + c["f2"]
    psi = s2 / (m * m)
    ip = 2.0 / psi
    b2 = ip - 1.0 + torch.sqrt((ip * (ip - 1.0)).clamp_min(0.0))
    a = m / (1.0 + b2)
    vn = a * (torch.sqrt(b2.clamp_min(0.0)) + Z1) ** 2
    sA = torch.minimum(c["A"].expand_as(a), 0.5 / a - eps)
    t = 1.0 - 2.0 * sA * a
    logM = sA * b2 * a / t - 0.5 * torch.log(t)
    rare = (psi > 1.5) | (m <= eps) | (psi <= eps)
    if bool(rare.any()):
        p = (psi - 1.0) / (psi + 1.0)
        beta = (1.0 - p) / m
        U = 0.5 * (1.0 + torch.erf(Z1 / math.sqrt(2.0)))
        ve = torch.where(U <= p, 0.0, torch.log((1.0 - p) / (1.0 - U.clamp_max(1.0 - eps))) / beta)
        sA = torch.minimum(c["A"].expand_as(beta), beta - eps)
        le = torch.log(p + beta * (1.0 - p) / (beta - sA))
        vn, logM = torch.where(psi > 1.5, ve, vn), torch.where(psi > 1.5, le, logM)
        vn, logM = torch.where(psi <= eps, m, vn), torch.where(psi <= eps, 0.0, logM)
        vn, logM = torch.where(m <= eps, 0.0, vn), torch.where(m <= eps, 0.0, logM)
    lx = lx + c["drift"] - logM - (c["K1"] + 0.5 * c["K3"]) * v + c["K1"] * v + c["K2"] * vn \
        + torch.sqrt(c["K3"] * (v + vn)) * Z2
    return lx, vn


def _jumps(c, n, path, stream, key, words, fp64):
    """log jump factor of step n, or None when no path jumps (a contract, no bumps of T inside)."""
    L = math.exp(-c["lam"] * c["T"] / c["n_steps"])
    L = L if fp64 else float(np.float32(L))
    if fp64:
        u = _u01(words[1], True)
    else:
        hi = ((words[0][0] & 0x1FF) << 9) | (words[0][1] & 0x1FF)
        u = (((hi << 5) | (words[1] >> 27)).double() + 0.5) * 2.0 ** -23
    idx = torch.nonzero(u >= L).flatten()
    if not len(idx):
        return None
    p, prod = path[idx], u[idx]
    first = _philox(n, p, stream, 1, key)
    N = torch.zeros_like(prod)
    going = torch.ones_like(prod, dtype=torch.bool)
    k = 1
    while bool(going.any()):
        word = first[k + 1] if k < 3 else _philox(n, p, stream, 3 + (k - 3) // 4, key)[(k - 3) % 4]
        N = N + going
        prod = torch.where(going, prod * _u01(word, fp64), prod)
        going = going & (prod >= L)
        k += 1
    return idx, N, _normals(first[0], first[1], fp64)[0]


def _simulate(cs, c, first, count, fp64, anti, sink):
    """Rows `cs` (contract and bumps on the same draws) for `count` lane units from `first`;
    sink(n, log S, v) after every step, log S and v of shape (rows, paths)."""
    eps = 1e-12 if fp64 else 1e-6
    k = _consts(cs, c.n_steps, eps)
    key, stream = c.seed, c.stream & 0xFFFFFFFF
    path = torch.arange(first, first + count, dtype=torch.int64, device="cuda")
    one = torch.ones(1, count * (2 if anti else 1), dtype=torch.float64, device="cuda")
    lx, v = torch.log(k["S0"]) * one, k["v0"] * one
    w = wp = None
    for n in range(c.n_steps):
        if n % 2 == 0:
            w = _philox(n // 2, path, stream, 0, key)
        if c.model == qk.BATES and n % 4 == 0:
            wp = _philox(n // 4, path, stream, 2, key)
        wa, wb = w[2 * (n % 2)], w[2 * (n % 2) + 1]
        Z1, Z2 = _normals(wa, wb, fp64)
        if anti:
            Z1, Z2 = torch.cat([Z1, -Z1]), torch.cat([Z2, -Z2])
        lx, v = _step(k, c.scheme, lx, v, Z1, Z2, eps)
        if c.model == qk.BATES:
            for r, row in enumerate(cs):
                j = _jumps(dict(row, n_steps=c.n_steps), n, path, stream, key, ((wa, wb), wp[n % 4]), fp64)
                if j is not None:
                    idx, N, Z = j
                    for s in ((1.0, -1.0) if anti else (1.0,)):
                        at = idx if s > 0 else idx + count
                        lx[r, at] += N * row["mu"] + s * torch.sqrt(N) * row["sj"] * Z
        sink(n, lx, v)


def _rows(c, g):
    """The contract and its bumps in normalised units, and each one's role."""
    base = dict(S0=1.0, v0=c.v0, r=c.r, q=c.q, T=c.T, kappa=c.kappa, theta=c.theta, sigma=c.sigma, rho=c.rho,
                lam=c.lambda_j, mu=c.mu_j, sj=c.sigma_j, bates=c.model == qk.BATES)
    if g is None:
        return [base]
    h, up, dn = g.bump_S_rel, c.v0 * (1 + g.bump_vol), c.v0 * (1 - g.bump_vol)
    bumps = [{}, {"S0": 1 + h}, {"S0": 1 - h}, {"v0": up}, {"v0": dn}, {"r": c.r + g.bump_r_abs},
             {"r": c.r - g.bump_r_abs}, {"T": c.T - g.bump_T_abs}, {"S0": 1 + h, "v0": up}, {"S0": 1 - h, "v0": up},
             {"S0": 1 + h, "v0": dn}, {"S0": 1 - h, "v0": dn}]
    return [dict(base, **b) for b in bumps]


def _payoff(p, n, S, ssum, smax, smin, S0):
    K, B = p.strike / S0, p.barrier / S0
    call = p.right == qk.CALL
    intr = lambda x, k: (x - k if call else k - x).clamp_min(0.0)  # noqa: E731
    if p.type == qk.ASIAN:
        return intr(ssum / n, K)
    if p.type == qk.BARRIER_UP_OUT:
        return torch.where(smax < B, intr(S, K), 0.0)
    if p.type == qk.BARRIER_DOWN_OUT:
        return torch.where(smin > B, intr(S, K), 0.0)
    if p.type == qk.LOOKBACK_FLOATING:
        return S - smin if call else smax - S
    if p.type == qk.BINARY_CASH:
        return ((S > K) if call else (S < K)).double()
    return intr(S, K)


def _forward(c, g, fp64, keep=False):
    """Leg results of one forward contract (and leg 0's payoffs, for the percentiles)."""
    rows, anti = _rows(c, g), bool(c.antithetic)
    R, P, n = len(rows), c.n_payoffs, c.n_steps
    units = c.n_paths // 2 if anti else c.n_paths
    chunk = max(1, min(units, (1 << 20) // R // (2 if anti else 1)))
    if units < (1 << 21) // R:
        chunk = units
    acc = torch.zeros(4, R, P, dtype=torch.float64, device="cuda")
    shift, kept = None, []
    eps = 1e-12 if fp64 else 1e-6
    for first in range(0, units, chunk):
        s = {}

        def sink(i, lx, v):
            S = torch.exp(lx)
            if i == 0:
                S0 = torch.tensor([[r["S0"]] for r in rows], dtype=torch.float64, device="cuda")
                s["sum"], s["max"], s["min"] = S, torch.maximum(S, S0), torch.minimum(S, S0)
            else:
                s["sum"], s["max"], s["min"] = s["sum"] + S, torch.maximum(s["max"], S), torch.minimum(s["min"], S)
            s["S"] = S

        _simulate(rows, c, first, min(chunk, units - first), fp64, anti, sink)
        x = torch.stack([_payoff(c.payoffs[k], n, s["S"], s["sum"], s["max"], s["min"], c.S0) for k in range(P)], 1)
        itm = (x > eps).double()
        if anti:
            h = x.shape[2] // 2
            x, itm = 0.5 * (x[..., :h] + x[..., h:]), 0.5 * (itm[..., :h] + itm[..., h:])
        if keep:
            kept.append(x[0, 0])
        shift = x.mean(2, keepdim=True) if shift is None else shift
        d = x - shift
        acc += torch.stack([torch.full_like(acc[0], x.shape[2]), d.sum(2), (d * d).sum(2), itm.sum(2)])
    N, D, Q, I = acc.cpu().numpy()
    mean, var = shift[..., 0].cpu().numpy() + D / N, (Q - D * D / N) / np.maximum(N - 1, 1)
    scale = np.array([1.0 if c.payoffs[k].type == qk.BINARY_CASH else c.S0 for k in range(P)])
    eff = np.array([[math.exp(-r["r"] * r["T"])] for r in rows]) * scale
    p = mean * eff
    legs = []
    for k in range(P):
        leg = {"price": p[0, k], "std_error": math.sqrt(var[0, k] / N[0, k]) * eff[0, k], "prob_itm": (I / N)[0, k]}
        if g is not None:
            h, hv, q = c.S0 * g.bump_S_rel, c.v0 * g.bump_vol, p[:, k]
            leg.update(delta=(q[1] - q[2]) / (2 * h), gamma=(q[1] - 2 * q[0] + q[2]) / (h * h),
                       vega=(q[3] - q[4]) / (2 * hv), vomma=(q[3] - 2 * q[0] + q[4]) / (hv * hv),
                       rho=(q[5] - q[6]) / (2 * g.bump_r_abs), theta=(q[7] - q[0]) / g.bump_T_abs,
                       vanna=(q[8] - q[9] - q[10] + q[11]) / (4 * h * hv))
        legs.append(leg)
    return {"legs": legs, "payoffs": torch.cat(kept).cpu().numpy() * eff[0, 0] if keep else None}


def _american(c, fp64):
    """Longstaff-Schwartz on the same paths: least squares of the discounted cash flow over
    the in-the-money paths at every date, exercise where the payoff beats the fit."""
    D = c.lsm_dates or c.n_steps
    stride, K, row = c.n_steps // D, c.payoffs[0].strike / c.S0, _rows(c, None)
    S = torch.empty(D, c.n_paths, dtype=torch.float64, device="cuda")
    V = torch.empty_like(S)

    for first in range(0, c.n_paths, 1 << 20):
        cnt = min(1 << 20, c.n_paths - first)

        def sink(i, lx, v):
            if (i + 1) % stride == 0:
                S[i // stride, first:first + cnt] = torch.exp(lx[0])
                V[i // stride, first:first + cnt] = v[0]

        _simulate(row, c, first, cnt, fp64, False, sink)
    disc = math.exp(-c.r * stride * c.T / c.n_steps)
    put = c.payoffs[0].right == qk.PUT
    intr = lambda s: (K - s if put else s - K).clamp_min(0.0)  # noqa: E731
    cf = intr(S[-1])
    for d in range(D - 2, -1, -1):
        iv = intr(S[d])
        cf = cf * disc
        itm = iv > 0
        x, v, y = S[d][itm] / K, V[d][itm], cf[itm]
        if c.lsm_basis == qk.LSM_POLY_SV:
            x, v = x - x.mean() if len(x) else x, v - v.mean() if len(v) else v
            X = torch.stack([torch.ones_like(x), x, x * x, x ** 3, v, x * v], 1)
        else:
            X = torch.stack([torch.ones_like(x), 1 - x, (0.5 * x - 2) * x + 1, ((-x / 6 + 1.5) * x - 3) * x + 1], 1)
        if len(x) < X.shape[1]:
            hold = y.mean().expand_as(y) if len(x) else y
        else:
            sc = X.norm(dim=0).clamp_min(1e-300)
            Xs = X / sc
            G = Xs.T @ Xs
            if c.lsm_basis != qk.LSM_POLY_SV:
                G = G + torch.diag(1e-8 / (sc * sc))
            hold = Xs @ torch.linalg.solve(G, Xs.T @ y)
        cf[itm] = torch.where(iv[itm] > hold, iv[itm], y)
    cf = (cf * disc)
    n, mean, sd = c.n_paths, float(cf.mean()), float(cf.std())
    itm = float((cf > (1e-12 if fp64 else 1e-6)).double().mean())
    now = max(K - 1.0, 0.0) if put else max(1.0 - K, 0.0)
    if now > mean:
        mean, sd, itm = now, 0.0, 1.0
    return {"legs": [{"price": mean * c.S0, "std_error": sd / math.sqrt(n) * c.S0, "prob_itm": itm}]}


def exact(case, seed):
    if case["kind"] == "serve":
        return None
    cs, fp64 = _contracts(case, seed), case["fp64"]
    g = W.batch_greeks() if case.get("greeks") else None
    if case["kind"] == "dispatcher":
        c = cs[0]
        c.seed = c.seed >> 1 or 1
        r = _forward(c, None, True, keep=True)
        leg, pay = r["legs"][0], np.sort(r["payoffs"])
        N = float(len(pay))
        at = [0] + [int(N * f) for f in (0.01, 0.05, 0.1, 0.2, 0.3, 0.4, 0.5, 0.6, 0.7, 0.8, 0.9, 0.95, 0.99)] + [-1]
        return {"price": np.array([leg["price"]]), "std_error": np.array([leg["std_error"]]),
                "prob_itm": np.array([leg["prob_itm"]]), "percentiles": pay[at]}
    results = [_american(c, fp64) if c.payoffs[0].type == qk.AMERICAN else _forward(c, g, fp64) for c in cs]
    return _table(results, True, g is not None)
