"""What the engine's speed is measured on: the calls a user's program
makes, through the verbs of dust2_gb300, from one short particle filter to
batched and served filters, forward simulation, ODE sweeps, mixed-time
filters and gradients.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program has in hand before the call
    run(state)           one pass; returns its outputs
    exact(case, seed)    the outputs in plain 64-bit torch, where they are
                         computed numbers rather than random draws
    work(case)           bytes and floating-point operations of one pass

All inputs are synthetic: parameters and data are made from the seed with
numpy alone (epidemics are simulated by numpy's own binomial sampler).
"""

import math

import numpy as np
import torch

import dust2_gb300 as d

N_AGE = 16


# ---------------------------------------------------------------------------
# cases

def listed():
    return [
        # a user's first filter: dust2's example SIR (with its noise draw
        # in the comparison), one unit step per day; launches and
        # synchronisations are all of it
        {"name": "filter_sir_100", "kind": "filter", "model": "sir",
         "groups": 1, "low": 100, "high": 100, "n_obs": 30, "steps": 1},
        # one chain's likelihood of the benchmark SIR (1000 particles, 100
        # daily observations, dt = 1/4): too few particles for the device
        {"name": "filter_sir_1000", "kind": "filter", "model": "sir_cases",
         "groups": 1, "low": 1000, "high": 1000, "n_obs": 100, "steps": 4},
        # likelihoods of 64 regions with uneven particle counts, the
        # batched SIR benchmark
        {"name": "filter_sir_batched", "kind": "filter",
         "model": "sir_cases", "groups": 64, "low": 512, "high": 32768,
         "n_obs": 200, "steps": 4},
        # a user's own model class (the plugin adapter), a few groups,
        # missing data, and one sampled trajectory per group, as a
        # sampler's observer takes it
        {"name": "filter_sirs_trajectories", "kind": "filter",
         "model": "sirs", "groups": 6, "low": 1501, "high": 1501,
         "n_obs": 60, "steps": 2, "trajectories": True, "missing": True},
        # one chain's likelihood of the 16-age SEIR, odd particle count
        {"name": "filter_seir_3001", "kind": "filter", "model": "seir_age",
         "groups": 1, "low": 3001, "high": 3001, "n_obs": 60, "steps": 4},
        # the batched age-structured SEIR: 32 groups of 8192 particles
        {"name": "filter_seir_batched", "kind": "filter",
         "model": "seir_age", "groups": 32, "low": 8192, "high": 8192,
         "n_obs": 60, "steps": 4},
        # many chains' requests on one likelihood server, each with its
        # own particle count and data length
        {"name": "served_seir", "kind": "served", "model": "seir_age",
         "sessions": 32, "low": 512, "high": 16384, "n_obs": 90,
         "steps": 4},
        # forward projection: an ensemble simulated and one series kept
        {"name": "simulate_sir", "kind": "simulate", "model": "sir",
         "particles": 100003, "n_times": 60, "steps": 4},
        # parameter sweep of an ODE, weekly output
        {"name": "ode_sweep", "kind": "ode", "instances": 65536,
         "n_times": 28, "every": 7},
        # a small ODE ensemble with daily output: one launch's latency
        {"name": "ode_small", "kind": "ode", "instances": 300,
         "n_times": 100, "every": 1},
        # a mixed-time filter (ODE with daily stochastic updates)
        {"name": "filter_malaria", "kind": "filter", "model": "malaria",
         "groups": 2, "low": 1000, "high": 1000, "n_obs": 40, "steps": 1},
        # gradients of deterministic likelihoods (Hamiltonian samplers)
        {"name": "gradient_sir", "kind": "gradient", "groups": 64,
         "n_obs": 150},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


# particle-steps of a drawn filter at most: the cost of the largest
# listed filter of the same model or less
_MOST = {"sir": 1e8, "sir_cases": 4e8, "sirs": 6e7, "seir_age": 6e7,
         "malaria": 2e5}


def draw(rng):
    kind = rng.choice(["filter"] * 6 + ["served", "simulate", "ode",
                                        "gradient"])
    if kind == "filter":
        model = rng.choice(["sir", "sir_cases", "sir_cases", "sirs",
                            "seir_age", "seir_age", "malaria"])
        steps = 1 if model == "malaria" else rng.choice([1, 2, 4])
        n_obs = _log_int(rng, 20, 60 if model == "malaria" else 200)
        groups = _log_int(rng, 1, 4 if model == "malaria" else 64)
        most = _MOST[model] / (groups * n_obs * steps)
        high = max(2, min(_log_int(rng, 100, 32768), int(most)))
        low = rng.choice([high, max(2, high // rng.randint(2, 64))])
        if model == "malaria":
            low = high
        case = {"kind": kind, "model": model, "groups": groups, "low": low,
                "high": high, "n_obs": n_obs, "steps": steps}
        if low == high and model != "malaria" and rng.random() < 0.3:
            case["trajectories"] = True
        if rng.random() < 0.3:
            case["missing"] = True
        return case
    if kind == "served":
        high = _log_int(rng, 512, 16384)
        return {"kind": kind, "model": rng.choice(["seir_age", "sir_cases"]),
                "sessions": _log_int(rng, 4, 32),
                "low": max(100, high // rng.randint(1, 32)), "high": high,
                "n_obs": _log_int(rng, 20, 90), "steps": 4}
    if kind == "simulate":
        return {"kind": kind, "model": rng.choice(["sir", "sirs", "walk"]),
                "particles": _log_int(rng, 100, 100000),
                "n_times": _log_int(rng, 10, 60), "steps": rng.choice([1, 4])}
    if kind == "ode":
        return {"kind": kind, "instances": _log_int(rng, 100, 65536),
                "n_times": _log_int(rng, 5, 28), "every": rng.choice([1, 7])}
    return {"kind": kind, "groups": _log_int(rng, 1, 128),
            "n_obs": _log_int(rng, 20, 150)}


# ---------------------------------------------------------------------------
# inputs

def _counts(case, n):
    """Particle counts, log-uniform in [low, high]; a case's sizes are its
    own, whatever the seed."""
    rs = np.random.default_rng([n, case["low"], case["high"]])
    lo, hi = math.log(case["low"]), math.log(case["high"])
    return [int(round(math.exp(x))) for x in rs.uniform(lo, hi, n)]


def _contact():
    rs = np.random.default_rng(7)
    a = rs.gamma(2.0, 1.0, size=(N_AGE, N_AGE)) / N_AGE
    return np.triu(a) + np.triu(a, 1).T


def _sir_inputs(model, n, n_obs, steps, rs, big):
    """Parameters of n epidemics and their daily cases, simulated by
    numpy with `steps` steps a day and observed with Poisson noise."""
    pars, beta, gamma = [], np.empty(n), np.empty(n)
    pop, i0 = np.empty(n), np.empty(n)
    for g in range(n):
        pop[g] = 1e6 if big else float(rs.integers(1000, 20000))
        i0[g] = float(rs.integers(5, 101))
        beta[g] = rs.uniform(0.2, 0.5)
        gamma[g] = rs.uniform(0.05, 0.2)
        p = {"N": pop[g], "I0": i0[g], "beta": beta[g], "gamma": gamma[g]}
        if model == "sirs":
            p["omega"] = rs.uniform(0.01, 0.05)
        pars.append(p)
    dt = 1.0 / steps
    s, i = pop - i0, i0.copy()
    cases = np.zeros((n_obs, n))
    for t in range(n_obs):
        for _ in range(steps):
            n_si = rs.binomial(s.astype(int), 1 - np.exp(-beta * i / pop * dt))
            n_ir = rs.binomial(i.astype(int), 1 - np.exp(-gamma * dt))
            s, i = s - n_si, i + n_si - n_ir
            cases[t] += n_si
    return pars, rs.poisson(cases + 1e-6).astype(float)


def _seir_inputs(n, n_obs, steps, rs):
    c = _contact()
    rho = np.max(np.abs(np.linalg.eigvalsh(c)))
    r0 = rs.uniform(1.2, 3.0, n)
    pars = [{"R0": float(r), "sigma": 0.2, "gamma": 0.1, "size": 20,
             "I0": 5, "contact": c.ravel()} for r in r0]
    dt = 1.0 / steps
    pop = 62500.0
    s = np.full((n, N_AGE), pop - 5)
    e, i = np.zeros((n, N_AGE)), np.full((n, N_AGE), 5.0)
    cases = np.zeros((n_obs, n))
    for t in range(n_obs):
        for _ in range(steps):
            lam = (r0 * 0.1 / rho)[:, None] * (i / pop) @ c.T
            n_se = rs.binomial(s.astype(int), 1 - np.exp(-lam * dt))
            n_ei = rs.binomial(e.astype(int), 1 - np.exp(-0.2 * dt))
            n_ir = rs.binomial(i.astype(int), 1 - np.exp(-0.1 * dt))
            s, e, i = s - n_se, e + n_se - n_ei, i + n_ei - n_ir
            cases[t] += n_ei.sum(axis=1)
    mu = cases + 1e-6
    return pars, rs.negative_binomial(20, 20 / (20 + mu)).astype(float)


def _malaria_inputs(n, n_obs, rs):
    pars = [{"a": rs.uniform(0.25, 0.4), "r": rs.uniform(0.008, 0.015)}
            for _ in range(n)]
    tested = rs.integers(50, 400, (n_obs, n)).astype(float)
    positive = rs.binomial(tested.astype(int),
                           rs.uniform(0.6, 0.8, (1, n))).astype(float)
    return pars, tested, positive


def _columns(n_obs, n, series):
    """Data columns, one row per time and group."""
    out = {k: v.ravel() for k, v in series.items()}
    out["time"] = np.repeat(np.arange(1.0, n_obs + 1), n)
    if n > 1:
        out["group"] = np.tile(np.arange(1, n + 1), n_obs)
    return out


def _filter_inputs(case, n, rs):
    model, n_obs = case["model"], case["n_obs"]
    if model == "seir_age":
        pars, inc = _seir_inputs(n, n_obs, case["steps"], rs)
        series = {"incidence": inc}
    elif model == "malaria":
        pars, tested, positive = _malaria_inputs(n, n_obs, rs)
        series = {"tested": tested, "positive": positive}
    else:
        pars, inc = _sir_inputs(model, n, n_obs, case["steps"], rs,
                                model == "sir_cases" and n > 1)
        series = {"cases" if model == "sirs" else "incidence": inc}
    if case.get("missing"):
        gap = rs.uniform(size=(n_obs, n)) < 0.1
        series = {k: np.where(gap, np.nan, v) for k, v in series.items()}
    return pars, series


def _sweep_pars(n, rs):
    beta = rs.uniform(0.1, 0.5, n)
    gamma = rs.uniform(0.05, 0.2, n)
    i0 = rs.uniform(1, 100, n)
    return beta, gamma, i0


def _gradient_inputs(case, seed):
    rs = np.random.default_rng([seed, 4])
    pars, inc = _sir_inputs("sir", case["groups"], case["n_obs"], 1, rs,
                            False)
    return pars, inc


def prepare(case, seed):
    kind = case["kind"]
    rs = np.random.default_rng([seed, 1])
    if kind == "filter":
        n = case["groups"]
        pars, series = _filter_inputs(case, n, rs)
        even = case["low"] == case["high"]
        obj = d.dust_filter_create(
            getattr(d, case["model"])(), 0,
            _columns(case["n_obs"], n, series),
            n_particles=case["low"] if even else _counts(case, n),
            dt=1.0 / case["steps"], seed=seed)
        return {"kind": kind, "obj": obj, "pars": pars if n > 1 else pars[0],
                "trajectories": bool(case.get("trajectories"))}
    if kind == "served":
        n = case["sessions"]
        pars, series = _filter_inputs(case, n, rs)
        server = d.dust_likelihood_server(getattr(d, case["model"])(),
                                          hbm_budget=2e9)
        (name, values), = series.items()
        sessions = []
        days = np.random.default_rng(n).integers(
            max(1, case["n_obs"] // 3), case["n_obs"] + 1, n)
        for i, n_particles in enumerate(_counts(case, n)):
            n_obs = int(days[i])
            data = {"time": np.arange(1.0, n_obs + 1),
                    name: values[:n_obs, i]}
            sessions.append(server.open(pars[i], data, n_particles,
                                        dt=1.0 / case["steps"],
                                        seed=1000 * (seed % 10**6) + i))
        return {"kind": kind, "server": server, "sessions": sessions,
                "pars": pars}
    if kind == "simulate":
        if case["model"] == "walk":
            pars = {"sd": rs.uniform(0.5, 2)}
        else:
            pars = {"N": 1e5, "I0": 20, "beta": rs.uniform(0.2, 0.5),
                    "gamma": rs.uniform(0.05, 0.2)}
        sys = d.dust_system_create(getattr(d, case["model"])(), pars,
                                   n_particles=case["particles"],
                                   dt=1.0 / case["steps"], seed=seed)
        keep = [1] if case["model"] == "walk" else [2, 4]
        return {"kind": kind, "sys": sys, "keep": keep,
                "times": np.arange(1.0, case["n_times"] + 1)}
    if kind == "ode":
        n = case["instances"]
        beta, gamma, i0 = _sweep_pars(n, rs)
        pars = [{"I0": i0[k], "N": 1e6, "beta": beta[k], "gamma": gamma[k]}
                for k in range(n)]
        sys = d.dust_system_create(d.sirode(), pars, n_groups=n)
        times = case["every"] * np.arange(1.0, case["n_times"] + 1)
        return {"kind": kind, "sys": sys, "times": times, "keep": [2, 5]}
    pars, inc = _gradient_inputs(case, seed)
    n = case["groups"]
    obj = d.dust_unfilter_create(d.sir(), 0,
                                 _columns(case["n_obs"], n,
                                          {"incidence": inc}), dt=1)
    return {"kind": kind, "obj": obj, "pars": pars if n > 1 else pars[0]}


def run(state):
    kind = state["kind"]
    if kind == "filter":
        obj = state["obj"]
        ll = d.dust_likelihood_run(obj, state["pars"],
                                   save_trajectories=state["trajectories"])
        out = {"ll": ll, "state": d.dust_likelihood_last_state(obj)}
        if state["trajectories"]:
            out["trajectories"] = d.dust_likelihood_last_trajectories(
                obj, select_random_particle=True)
        return out
    if kind == "served":
        server = state["server"]
        tickets = [server.submit(s, p)
                   for s, p in zip(state["sessions"], state["pars"])]
        return np.array([server.wait(t)[0] for t in tickets])
    if kind in ("simulate", "ode"):
        sys = state["sys"]
        d.dust_system_set_time(sys, 0)
        d.dust_system_set_state_initial(sys)
        return d.dust_system_simulate(sys, state["times"],
                                      index_state=state["keep"])
    obj = state["obj"]
    ll = d.dust_likelihood_run(obj, state["pars"], adjoint=True)
    return {"ll": np.asarray(ll), "gradient":
            d.dust_likelihood_last_gradient(obj)}


# ---------------------------------------------------------------------------
# the same outputs in plain 64-bit arithmetic

def _exact_ode(case, seed):
    """The SIR equations by classical Runge-Kutta at 40 steps a day."""
    rs = np.random.default_rng([seed, 1])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    beta, gamma, i0 = (torch.tensor(x, dtype=torch.float64, device=dev)
                       for x in _sweep_pars(case["instances"], rs))
    scaled = beta / 1e6
    h = 1.0 / 40

    def slope(s, i):
        flow = scaled * s * i
        return flow, flow - gamma * i

    s, i = 1e6 - i0, i0.clone()
    out = []
    for day in range(1, case["n_times"] * case["every"] + 1):
        start = s.clone()
        for _ in range(40):
            a1, b1 = slope(s, i)
            a2, b2 = slope(s - h / 2 * a1, i + h / 2 * b1)
            a3, b3 = slope(s - h / 2 * a2, i + h / 2 * b2)
            a4, b4 = slope(s - h * a3, i + h * b3)
            s = s - h / 6 * (a1 + 2 * a2 + 2 * a3 + a4)
            i = i + h / 6 * (b1 + 2 * b2 + 2 * b3 + b4)
        if day % case["every"] == 0:
            out.append(torch.stack([i, start - s]).cpu().numpy())
    # (state, group, time) in dust2's column-major order
    return np.stack(out, axis=2)


def _exact_gradient(case, seed):
    pars, inc = _gradient_inputs(case, seed)

    def column(name):
        return torch.tensor([p[name] for p in pars], dtype=torch.float64)

    pop = column("N")
    beta, gamma, i0 = (column(x).requires_grad_()
                       for x in ("beta", "gamma", "I0"))
    s, i = pop - column("I0"), i0
    ll = torch.zeros_like(pop)
    for y in torch.tensor(inc, dtype=torch.float64):
        n_si = s * (1 - torch.exp(-beta * i / pop))
        n_ir = i * (1 - torch.exp(-gamma))
        s, i = s - n_si, i + n_si - n_ir
        lam = n_si + 1e-6
        ll = ll + y * torch.log(lam) - lam - torch.lgamma(y + 1)
    grad = torch.stack(torch.autograd.grad(ll.sum(), (beta, gamma, i0)))
    ll = ll.detach().numpy()
    grad = grad.numpy()
    if case["groups"] == 1:
        return {"ll": ll[0], "gradient": grad[:, 0]}
    return {"ll": ll, "gradient": grad}


def exact(case, seed):
    if case["kind"] == "ode":
        return _exact_ode(case, seed)
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    return None  # random draws


# ---------------------------------------------------------------------------
# work of one pass

# Floating-point operations of a particle-step: the models' and samplers'
# own (an elementary function counted once), and of a dopri5 step.
_FLOPS = {"sir": 60, "sir_cases": 60, "sirs": 90, "seir_age": 1739,
          "walk": 10, "malaria": 2000}
_STATE = {"sir": 5, "sir_cases": 4, "sirs": 4, "seir_age": 96, "walk": 1,
          "malaria": 20}
_ODE_STEP = 444


def work(case):
    kind = case["kind"]
    if kind in ("filter", "served"):
        n = case["groups"] if kind == "filter" else case["sessions"]
        low, high = case["low"], case["high"]
        mean = low if low == high else (high - low) / math.log(high / low)
        particles = n * mean
        n_obs = case["n_obs"] if kind == "filter" else case["n_obs"] * 2 / 3
        model = case["model"]
        state = 8 * _STATE[model] if kind == "filter" else 0
        # generators read and written, final state, data
        return {"bytes": particles * (64 + state) + 8 * n * n_obs,
                "flops": particles * n_obs * case["steps"] * _FLOPS[model]}
    if kind == "simulate":
        n = case["particles"]
        kept = 1 if case["model"] == "walk" else 2
        return {"bytes": n * (64 + 8 * kept * case["n_times"]),
                "flops": n * case["n_times"] * case["steps"] *
                _FLOPS[case["model"]]}
    if kind == "ode":
        n = case["instances"]
        # about one accepted step a day
        return {"bytes": n * (32 + 16 * case["n_times"]),
                "flops": n * case["n_times"] * case["every"] * _ODE_STEP}
    n = case["groups"]
    return {"bytes": 8 * n * (case["n_obs"] + 8),
            "flops": n * case["n_obs"] * 80}
