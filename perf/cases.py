"""The work that users of this package have it do, as measured cases.

A user solves life-cycle models by backward induction and simulates them
forward: one parameter set at a time while a model is developed, batches of
parameter sets or a stream of requests in an estimation.  The cases call the
package's public entry points -- ``Model.solve``, ``Model.simulate``,
``BatchSolver``, ``SimPlan`` and ``Server`` -- on the package's example models,
whose sizes span the benchmark's configurations (100 to 2000 grid points,
horizons of 5 to 60 periods, batches of 1 to 256, 10,000 subjects).

Kinds of case:

- ``solve``: ``Model.solve`` of one parameter set, host arrays back;
- ``batch``: ``BatchSolver`` -- parameters uploaded, every instance solved, the
  value and policy arrays left on the device;
- ``sim``: ``SimPlan`` -- the simulations of solved instances;
- ``sim_call``: ``Model.simulate`` from given value functions;
- ``serve``: ``Server.run`` over a stream of solve + simulate requests.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from pylcm_b200 import examples
from pylcm_b200.batch import BatchSolver
from pylcm_b200.engine import SolveEngine
from pylcm_b200.serving import Server
from pylcm_b200.simulate import SimPlan
from pylcm_b200.solvers import FUESEnvelope, LTMEnvelope, MSSEnvelope, RFCEnvelope

ENVELOPES = {
    "fues": FUESEnvelope,
    "rfc": RFCEnvelope,
    "ltm": LTMEnvelope,
    "mss": MSSEnvelope,
}


def listed() -> list[dict]:
    return [
        # one solve of a small deterministic model, as in developing a model
        # or in a test: launches and host work count
        {"name": "solve_small", "kind": "solve", "model": "retirement", "periods": 5, "wealth": 100, "cons": 100,
         "precision": "fp64"},
        # one solve of the benchmark's stochastic model with the default
        # (double precision) arguments
        {"name": "solve_stochastic", "kind": "solve", "model": "stochastic", "periods": 40, "wealth": 500,
         "cons": 500, "precision": "fp64"},
        # the benchmark's headline: 256 parameter sets in the fast form
        {"name": "batch_fp32", "kind": "batch", "model": "stochastic", "batch": 256, "periods": 40, "wealth": 500,
         "cons": 500, "precision": "fp32"},
        # a batch in double precision throughout, odd grid sizes
        {"name": "batch_fp64", "kind": "batch", "model": "stochastic", "batch": 48, "periods": 12, "wealth": 333,
         "cons": 401, "precision": "fp64"},
        # two continuous states and a 32-state shock at full grid size, fast form
        {"name": "hc_fp32", "kind": "batch", "model": "hc", "batch": 2, "periods": 8, "wealth": 1000, "hc": 50,
         "shock": 32, "cons": 300, "precision": "fp32"},
        # the same model, smaller and ragged, double precision
        {"name": "hc_fp64", "kind": "batch", "model": "hc", "batch": 3, "periods": 6, "wealth": 413, "hc": 23,
         "shock": 11, "cons": 157, "precision": "fp64"},
        # DC-EGM with the FUES envelope at the benchmark's grids
        {"name": "dcegm_fues", "kind": "batch", "model": "dcegm", "batch": 32, "periods": 20, "wealth": 2000,
         "envelope": "fues", "taste": False, "precision": "fp64"},
        # taste shocks on the discrete choice, ragged grids
        {"name": "dcegm_taste", "kind": "batch", "model": "dcegm", "batch": 12, "periods": 10, "wealth": 777,
         "envelope": "fues", "taste": True, "precision": "fp64"},
        # another envelope of the candidate rows
        {"name": "dcegm_mss", "kind": "batch", "model": "dcegm", "batch": 6, "periods": 8, "wealth": 500,
         "envelope": "mss", "taste": False, "precision": "fp64"},
        # the simulation step of a batch of solved instances (counter stream)
        {"name": "sim_batch", "kind": "sim", "model": "stochastic", "batch": 16, "periods": 40, "wealth": 500,
         "cons": 500, "subjects": 10000, "precision": "fp32"},
        # one simulation through the model (the reference's random stream)
        {"name": "sim_call", "kind": "sim_call", "model": "stochastic", "periods": 10, "wealth": 250, "cons": 500,
         "subjects": 10000, "precision": "fp64"},
        # a job stream of the serving loop: both model families mixed
        {"name": "serve", "kind": "serve", "requests": 64, "subjects": 10000, "precision": "fp32"},
    ]


def _spread(rng, lo: int, hi: int) -> int:
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["solve", "batch", "batch", "hc", "dcegm", "dcegm", "sim", "sim_call", "serve"])
    prec = rng.choice(["fp32", "fp64"])
    if kind == "solve":
        return {"kind": "solve", "model": rng.choice(["retirement", "stochastic"]), "periods": _spread(rng, 3, 40),
                "wealth": _spread(rng, 50, 600), "cons": _spread(rng, 50, 600), "precision": prec}
    if kind == "batch":
        # at most a quarter of the headline's (state, action) pairs
        w, c, t = _spread(rng, 60, 800), _spread(rng, 60, 800), _spread(rng, 4, 40)
        most = max(2, int(256 * 500 * 500 * 40 / (4 * w * c * t)))
        return {"kind": "batch", "model": "stochastic", "batch": _spread(rng, 2, min(256, most)), "periods": t,
                "wealth": w, "cons": c, "precision": prec}
    if kind == "hc":
        return {"kind": "batch", "model": "hc", "batch": rng.randint(1, 3), "periods": rng.randint(3, 6),
                "wealth": _spread(rng, 90, 1000), "hc": rng.randint(9, 40), "shock": rng.choice([4, 7, 16, 32]),
                "cons": _spread(rng, 60, 300), "precision": prec}
    if kind == "dcegm":
        env = rng.choice(["fues", "fues", "rfc", "ltm", "mss"])
        return {"kind": "batch", "model": "dcegm", "batch": rng.randint(1, 12), "periods": rng.randint(4, 16),
                "wealth": _spread(rng, 90, 2000 if env in ("fues", "rfc") else 600), "envelope": env,
                "taste": rng.random() < 0.5, "precision": "fp64"}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(8, 48), "subjects": _spread(rng, 500, 10000),
                "precision": "fp32"}
    c = {"kind": kind, "model": "stochastic", "periods": _spread(rng, 4, 30), "wealth": _spread(rng, 90, 600),
         "cons": _spread(rng, 90, 600), "subjects": _spread(rng, 300, 10000), "precision": prec}
    if kind == "sim":
        c["batch"] = rng.randint(1, 12)
    return c


# ---------------------------------------------------------------------------
# a program keeps its models: one object per structure, many parameter sets
_MODELS: dict = {}


def _model(case: dict):
    key = tuple(case.get(k) for k in ("model", "periods", "wealth", "cons", "hc", "shock", "envelope", "taste"))
    if key not in _MODELS:
        m = case["model"]
        if m == "retirement":
            mod = examples.retirement_model(case["periods"], case["wealth"], case["cons"])
        elif m == "stochastic":
            mod = examples.stochastic_model(case["periods"], case["wealth"], case["cons"])
        elif m == "hc":
            mod = examples.hc_model(case["periods"], case["wealth"], case["hc"], case["shock"], case["cons"])
        else:
            mod = examples.dcegm_model(n_periods=case["periods"], n_savings=case["wealth"], n_wealth=case["wealth"],
                                       taste=case["taste"], envelope=ENVELOPES[case["envelope"]]())
        _MODELS[key] = mod
    return _MODELS[key]


def _draws(case: dict, seed: int) -> list[dict]:
    """The structural parameters of every instance, from the benchmark's
    ranges."""
    rng = np.random.default_rng([seed, 17])
    return [{"beta": float(rng.uniform(0.90, 0.99)), "crra": float(rng.uniform(1.0, 5.0)),
             "r": float(rng.uniform(0.01, 0.06)), "seed": int(rng.integers(1 << 31))}
            for _ in range(case.get("batch", 1))]


def _params(case: dict, d: dict) -> dict:
    m = case["model"]
    if m == "retirement":
        return examples.retirement_params(d["beta"])
    if m == "stochastic":
        return examples.stochastic_params(beta=d["beta"], crra=d["crra"], interest_rate=d["r"])
    if m == "hc":
        return examples.hc_params(seed=d["seed"], n_shock=case["shock"], beta=d["beta"], crra=d["crra"],
                                  interest_rate=d["r"])
    return examples.dcegm_params(seed=d["seed"], taste_scale=0.05 if case["taste"] else None, beta=d["beta"],
                                 crra=d["crra"], interest_rate=d["r"])


def _subjects(case: dict, seed: int, k: int) -> dict:
    """Initial conditions: wealth U[1, 50], income around its nodes, all in
    the working regime (its id is 0)."""
    rng = np.random.default_rng([seed, 23, k])
    n = case["subjects"]
    sd = 0.1 / math.sqrt(1 - 0.81)
    return {"wealth": rng.uniform(1.0, 50.0, n), "income": sd * np.clip(rng.standard_normal(n), -2.9, 2.9),
            "regime_id": np.zeros(n, dtype=np.int64)}


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "serve":
        reqs = examples.serving_requests(case["requests"], seed=seed, n_agents=case["subjects"])
        srv = Server(precision=case["precision"], max_batch=64, n_streams=4, hbm_budget_bytes=20 << 30)
        return {"kind": kind, "server": srv, "requests": reqs}
    model = _model(case)
    params = [_params(case, d) for d in _draws(case, seed)]
    st = {"kind": kind, "model": model, "params": params, "precision": case["precision"]}
    if kind == "batch":
        st["solver"] = BatchSolver(model, case["batch"], case["precision"], template_params=params[0])
        st["packed"] = st["solver"].pack(params)
    elif kind == "sim":
        plan = SolveEngine(model, case["precision"]).plan(params)
        plan.run()
        st["sim"] = SimPlan(plan, instances=[(k, _subjects(case, seed, k), seed * 1000 + k)
                                             for k in range(case["batch"])])
    elif kind == "sim_call":
        st["V"] = model.solve(params=params[0], log_level="off", precision=case["precision"])
        st["ic"] = _subjects(case, seed, 0)
        st["seed"] = seed
    return st


def _stack(by_period) -> dict:
    """{period: {regime: array}} -> {regime: periods stacked}."""
    out: dict = {}
    for p in sorted(by_period):
        for r, v in by_period[p].items():
            out.setdefault(r, []).append(v)
    return {r: np.stack(v) for r, v in out.items()}


def run(state: dict):
    kind = state["kind"]
    if kind == "solve":
        V, pol = state["model"].solve(params=state["params"][0], log_level="off", precision=state["precision"],
                                      return_policy=True)
        return {"V": _stack(V), "policy": _stack(pol)}
    if kind == "batch":
        s = state["solver"]
        s.upload(state["packed"])
        s.run()
        return {"V": s.plan.V, "policy": s.plan.pol}
    if kind == "sim":
        state["sim"].run()
        return [{"states": g["S"], "actions": g["A"], "regime": g["R"], "value": g["val"]} for g in state["sim"].groups]
    if kind == "sim_call":
        res = state["model"].simulate(params=state["params"][0], initial_conditions=state["ic"],
                                      period_to_regime_to_V_arr=state["V"], log_level="off", seed=state["seed"],
                                      precision=state["precision"])
        ps = [res.periods[p] for p in sorted(res.periods)]
        return {"regime": np.stack([d["regime_id"] for d in ps]), "value": np.stack([d["value"] for d in ps]),
                "states": {n: np.stack([d["states"][n] for d in ps]) for n in ps[0]["states"]},
                "actions": {n: np.stack([d["actions"][n] for d in ps]) for n in ps[0]["actions"]}}
    results = state["server"].run(state["requests"], realtime=False)
    # every request's moments, padded to the longest horizon of the stream
    out = {}
    for i, r in enumerate(results):
        for name, m in r.moments.items():
            out.setdefault(name, np.full((len(results), 60), np.nan))[i, : len(m)] = m
    return out


# ---------------------------------------------------------------------------
def _serve_mean() -> dict:
    # the stream's mean request: half grid search (7 incomes), half DC-EGM
    # (16 shocks), 770 grid points, 37 periods
    return {"states": 37 * (0.5 * 14 * 770 + 0.5 * 17 * 770), "periods": 37}


def work(case: dict) -> dict:
    """Bytes: every period's value array written once and read once by the
    period before, the policies written once (a simulation: the subjects'
    arrays, the value arrays read once).  Flops: Q at every (state, action)
    pair as the models define it -- 10 operations with one continuous state,
    16 with two -- or, for DC-EGM, 40 per savings node and shock."""
    kind = case["kind"]
    if kind == "serve":
        m = _serve_mean()
        n = case["requests"]
        return {"bytes": n * (20 * m["states"] + case["subjects"] * m["periods"] * 44),
                "flops": n * (10 * m["states"] * 400 + case["subjects"] * m["periods"] * 600 * 10)}
    b, T, w = case.get("batch", 1), case["periods"], case["wealth"]
    if case["model"] == "dcegm":
        rows = 33  # 16 shocks x 2 choices, 1 retired
        return {"bytes": b * T * (17 * w * 20 + rows * w * 40), "flops": b * T * rows * w * 40 * 16}
    if case["model"] == "hc":
        ns, na, fl = case["shock"] * w * case["hc"], 3 * case["cons"], 16
    else:
        k = 7 if case["model"] == "stochastic" else 1
        ns, na, fl = k * w * 2, 1.5 * case["cons"], 10
    if kind in ("sim", "sim_call"):
        n = case["subjects"]
        return {"bytes": b * T * (8 * ns + 44 * n), "flops": b * T * n * na * fl}
    return {"bytes": b * T * ns * 20, "flops": b * T * ns * na * fl}


# ---------------------------------------------------------------------------
# plain double precision
def _dev() -> str:
    return "cuda" if torch.cuda.is_available() else "cpu"


def _lin(a: float, b: float, n: int) -> torch.Tensor:
    return torch.from_numpy(np.linspace(a, b, n)).to(_dev())


def _tauchen7() -> tuple[np.ndarray, np.ndarray]:
    """Nodes and transition matrix of AR(1) log income, rho 0.9, sigma 0.1, 3 sd."""
    rho, sigma, n = 0.9, 0.1, 7
    z = np.linspace(-1, 1, n) * 3 * sigma / math.sqrt(1 - rho * rho)
    cdf = np.vectorize(lambda x: 0.5 * math.erfc(-x / math.sqrt(2)))
    mid = (z[:-1] + z[1:]) / 2
    F = cdf((mid[None, :] - rho * z[:, None]) / sigma)
    P = np.diff(np.concatenate([np.zeros((n, 1)), F, np.ones((n, 1))], axis=1), axis=1)
    return z, P


def _zs(w, v):
    return torch.where((w == 0) & ~torch.isfinite(v), torch.zeros_like(v), w * v)


def _read(V, x, lo, step):
    """Linear read with extrapolation of rows V (..., n) at x (..., m)."""
    n = V.shape[-1]
    c = (x - lo) / step
    i = c.floor().clamp(0, n - 2)
    u = c - i
    i = i.long()
    V = V.expand(*x.shape[:-1], n)
    return _zs(1 - u, V.gather(-1, i)) + _zs(u, V.gather(-1, i + 1))


class _Retirement:
    """The retirement models (deterministic, or with Tauchen income and CRRA
    utility) for a batch of parameter draws, one period at a time."""

    def __init__(self, case: dict, draws: list[dict]) -> None:
        d = _dev()
        self.T = case["periods"]
        self.sto = case["model"] == "stochastic"
        self.w, self.c = _lin(1, 400, case["wealth"]), _lin(1, 400, case["cons"])
        self.step = 399.0 / (case["wealth"] - 1)
        col = lambda k: torch.tensor([x[k] for x in draws], dtype=torch.float64, device=d)[:, None, None, None]  # noqa: E731
        self.beta = col("beta")
        self.R = 1 + col("r") if self.sto else torch.full_like(self.beta, 1.05)
        crra = col("crra")
        self.u = self.c ** (1 - crra) / (1 - crra) if self.sto else self.c.log().expand(len(draws), 1, 1, -1)
        if self.sto:
            z, P = _tauchen7()
        else:
            z, P = np.zeros(1), np.ones((1, 1))
        self.z, self.P = torch.from_numpy(z).to(d), torch.from_numpy(P).to(d)

    def q(self, w, pay, period, EVw, EVr, regime):
        """Q (B, incomes or rows, len(w), actions) of `regime`; `w` (..., m),
        EVw / EVr the expected values of the working / retired regimes by row
        (B, rows, n), of the terminal one in the last decision period."""
        save = self.R * (w[..., None] - self.c)
        ok = self.c <= w[..., None]
        out = []
        for work in ((1, 0) if regime == "working" else (0,)):
            x = save + pay * work
            EV = EVw if work else EVr
            q = self.u - 0.5 * work + self.beta * _read(EV[..., None, :], x, 1.0, self.step)
            out.append(torch.where(ok, q, torch.full_like(q, -math.inf)))
        return torch.cat(out, -1)

    def terminal(self, w):
        ok = self.c <= w[..., None]
        return torch.where(ok, self.u, torch.full_like(self.u, -math.inf)).amax(-1)

    def solve(self):
        B, K, n = self.beta.shape[0], len(self.z), len(self.w)
        w = self.w.expand(B, K, n)
        Vt = self.terminal(w)
        out = {"working": [], "retired": [], "terminal": [Vt]}
        Vw = Vr = Vt
        pay = (20.0 * self.z.exp())[None, :, None, None]
        for p in range(self.T - 2, -1, -1):
            EVw, EVr = self.P @ Vw, self.P @ Vr
            nw, nr = torch.empty_like(Vt), torch.empty_like(Vt)
            for k in range(K):  # one income at a time: memory
                s = slice(k, k + 1)
                a = (w[:, s], pay[:, s], p, EVw[:, s], EVr[:, s])
                nw[:, s] = self.q(*a, "working").amax(-1)
                nr[:, s] = self.q(*a, "retired").amax(-1)
            Vw, Vr = nw, nr
            out["working"].append(Vw)
            out["retired"].append(Vr)
        return {r: torch.stack(v[::-1], 1) for r, v in out.items()}


def _exact_hc(case: dict, seed: int) -> dict:
    d = _dev()
    T, nw, nh, ns = case["periods"], case["wealth"], case["hc"], case["shock"]
    w, h, c, hours = _lin(0, 1000, nw), _lin(1, 5, nh), _lin(1, 1000, case["cons"]), _lin(0, 1, 3)
    ninf = torch.tensor(-math.inf, dtype=torch.float64, device=d)
    out = {"alive": [], "terminal": []}
    for dr in _draws(case, seed):
        P = torch.from_numpy(np.random.default_rng(dr["seed"]).dirichlet(np.ones(ns), size=ns)).to(d)
        z = _lin(-0.5, 0.5, ns)
        u = c ** (1 - dr["crra"]) / (1 - dr["crra"])
        ok = c[None, :] <= w[:, None]
        V = torch.where(ok, u, ninf).amax(-1)[None, :, None].expand(ns, nw, nh).contiguous()
        res = [V]
        for _ in range(T - 1):
            fin = torch.isfinite(V)
            pos = (P > 0).to(P.dtype)
            EV = torch.einsum("kj,jwh->kwh", P, torch.where(fin, V, torch.zeros_like(V)))
            for bad, to in ((V == -math.inf, ninf), (V.isnan(), ninf * 0)):
                EV = torch.where(torch.einsum("kj,jwh->kwh", pos, bad.to(P.dtype)) > 0, to, EV)
            EV = EV / P.sum(1)[:, None, None]
            new = torch.full_like(V, -math.inf)
            for x in hours.tolist():
                ch = (0.95 * h + 0.1 * x - 1.0) / (4.0 / (nh - 1))
                i = ch.floor().clamp(0, nh - 2)
                t = ch - i
                i = i.long()
                row = _zs(1 - t, EV[:, :, i]) + _zs(t, EV[:, :, i + 1])  # (ns, nw, nh): axis h read at h'
                for k in range(ns):
                    pay = z[k].exp() * h * x  # (nh,)
                    x1 = (1 + dr["r"]) * (w[None, :, None] - c) + pay[:, None, None]  # (nh, nw, nc)
                    q = _read(row[k].t()[:, None, :], x1, 0.0, 1000.0 / (nw - 1))
                    q = (u - 0.5 * x) + dr["beta"] * q
                    best = torch.where(ok, q, ninf).amax(-1)  # (nh, nw)
                    new[k] = torch.maximum(new[k], best.t())
            V = new
            res.append(V)
        out["terminal"].append(res[0].reshape(1, -1))
        out["alive"].append(torch.stack(res[:0:-1]).reshape(T - 1, -1))
    return {r: torch.stack(v) for r, v in out.items()}


def _philox(subject, period, stream, key):
    """Philox-4x32-10 of the counters (subject, period, stream, 0)."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [subject.astype(np.uint64), np.full_like(subject, period, np.uint64), np.full_like(subject, stream, np.uint64),
         np.zeros_like(subject, np.uint64)]
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m32, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _normal(subject, period, stream, key) -> torch.Tensor:
    r = _philox(subject, period, stream, key)
    u = lambda a, b: (((a >> np.uint64(5)) << np.uint64(26) | (b >> np.uint64(6))).astype(np.float64) + 0.5) / 2.0**53  # noqa: E731
    return torch.from_numpy(np.sqrt(-2 * np.log(u(r[0], r[1]))) * np.cos(2 * np.pi * u(r[2], r[3]))).to(_dev())


def _exact_sim(case: dict, seed: int) -> list:
    d = _dev()
    draws, T, N = _draws(case, seed), case["periods"], case["subjects"]
    nan = float("nan")
    B = len(draws)
    z, P = _tauchen7()
    mk = lambda t: torch.full((B, t, N), nan, dtype=torch.float64, device=d)  # noqa: E731
    wealth, income, val, cons, labor = mk(T + 1), mk(T + 1), mk(T), mk(T), mk(T)
    sub = np.arange(N, dtype=np.uint64)
    Pm = torch.from_numpy(P).to(d)
    step = float(z[1] - z[0])
    for b, dr in enumerate(draws):
        mod = _Retirement(case, [dr])
        V = mod.solve()
        ic = _subjects(case, seed, b)
        w, y = (torch.from_numpy(ic[k]).to(d) for k in ("wealth", "income"))
        working = torch.ones(N, dtype=torch.bool, device=d)
        for p in range(T):
            wealth[b, p], income[b, p] = w, y
            if p == T - 1:
                q = mod.terminal(w[None, None])[0, 0]
                ok = mod.c <= w[:, None]
                a = torch.where(ok, mod.u[0, 0], torch.full((), -math.inf, device=d, dtype=torch.float64)).argmax(-1)
                val[b, p], cons[b, p] = q, mod.c[a]
                break
            EV = {r: Pm @ (V[r][0, p + 1] if p + 1 < T - 1 else V["terminal"][0, 0]) for r in ("working", "retired")}
            cy = (y - float(z[0])) / step
            lo = cy.floor().clamp(0, 5)
            t = (cy - lo)[:, None]
            lo = lo.long()
            nc = len(mod.c)
            for i0 in range(0, N, 2000):  # memory
                s = slice(i0, min(N, i0 + 2000))
                row = {r: ((1 - t[s]) * e[lo[s]] + t[s] * e[lo[s] + 1])[None] for r, e in EV.items()}
                pay = (20.0 * y[s].exp())[None, :, None, None]
                q = mod.q(w[s][None, :, None], pay, p, row["working"], row["retired"], "working")[0, :, 0]
                wk = working[s]
                q[:, :nc] = torch.where(wk[:, None], q[:, :nc], torch.full_like(q[:, :nc], -math.inf))
                qr = q[:, nc:]  # the retired regime's Q is the retiring choice's
                v, a = q.max(-1)
                val[b, p, s] = v
                ac = torch.where(wk, a, qr.argmax(-1))
                cc = mod.c[ac % nc]
                lab = torch.div(ac, nc, rounding_mode="floor").to(torch.float64)
                cons[b, p, s] = cc
                labor[b, p, s] = torch.where(wk, lab, torch.full_like(lab, nan))
                stay = wk & (lab == 0)
                w[s] = (1 + dr["r"]) * (w[s] - cc) + torch.where(stay, 20.0 * y[s].exp(), torch.zeros_like(cc))
                working[s] = stay
            y = 0.9 * y + 0.1 * _normal(sub, p, 1, seed * 1000 + b)
        wealth[b, T], income[b, T] = w, y
    return [{"states": {"wealth": wealth, "income": income}, "actions": {"consumption": cons, "labor_supply": labor},
             "regime": None, "value": val}]


def exact(case: dict, seed: int):
    """The values in plain double precision.  None for the policies (whole
    numbers), for DC-EGM (its envelope is the outcome of a sequential scan),
    and for the served moments and the simulations drawn from the reference's
    stream."""
    if case["kind"] in ("serve", "sim_call") or case["model"] == "dcegm":
        return None
    if case["kind"] == "sim":
        return _exact_sim(case, seed)
    if case["model"] == "hc":
        V = _exact_hc(case, seed)
    else:
        draws = _draws(case, seed)
        parts = [_Retirement(case, draws[i:i + 16]).solve() for i in range(0, len(draws), 16)]
        V = {r: torch.cat([p[r] for p in parts]) for r in parts[0]}
        V = {r: v.reshape(v.shape[0], v.shape[1], -1) for r, v in V.items()}
        if case["kind"] == "solve":
            shape = (7, case["wealth"]) if case["model"] == "stochastic" else (case["wealth"],)
            V = {r: v[0].reshape(v.shape[1], *shape) for r, v in V.items()}
    return {"V": V, "policy": None}
