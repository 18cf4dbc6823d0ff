"""What a user of this package runs, as cases that can be timed.

A case names a path through the public entry points (``gpu_metropolis``,
``Session.run`` / ``run_da`` / ``loglik_batch`` / ``grad_batch`` /
``loglik_pointwise``, ``Surrogate.train_stages``), a model of
``gpumetropolis_b200.workloads`` and its sizes.  ``listed()`` holds one case per
path; ``draw()`` gives further ones over the same ranges: 1 to a few thousand
chains or points, some hundred to a million observations, 1 to 65 parameters,
the five models, the four proposal kinds, both engines, odd sizes included.

Sampler outputs follow discrete accept decisions, so they have no value "in 64
bits" of their own; the evaluators' outputs do (``exact``).
"""
from __future__ import annotations

import math

import numpy as np

from gpumetropolis_b200 import _native
from gpumetropolis_b200 import workloads as W
from gpumetropolis_b200.api import gpu_metropolis

_MODES = {"rwm": _native.MODE_RWM, "de": _native.MODE_DE, "chol": _native.MODE_CHOL,
          "mala": _native.MODE_MALA}
_ENGINES = {"auto": _native.ENGINE_AUTO, "interp": _native.ENGINE_INTERP}


def listed():
    return [
        # A whole fit of a one-parameter model on a small data set with the
        # adaptive warmup: the smallest problem of the test suite and of the
        # benchmark configurations (20,000 observations, 8 chains).
        dict(name="fit-gaussian", op="fit", model="gaussian", p=0, n_obs=20000, n_chains=8,
             n_iter=1000, method="rwm"),
        # A whole fit of an ordinary regression: adaptive warmup, then random
        # walks with a pooled Cholesky proposal.
        dict(name="fit-logistic", op="fit", model="logistic", p=16, n_obs=20011, n_chains=64,
             n_iter=400, method="rwm"),
        # The log-likelihood at one point, as an optimiser asks for it.
        dict(name="loglik-one-point", op="loglik", model="logistic", p=16, n_obs=4099,
             n_points=1, engine="auto"),
        # A batch of posterior draws evaluated on the interpreter engine (the
        # one that runs where the run-time compiler is not installed).
        dict(name="loglik-interpreter", op="loglik", model="logistic", p=16, n_obs=131072,
             n_points=512, engine="interp"),
        # Gradients of a batch of points (optimisers, Langevin moves by hand).
        dict(name="grad-logistic", op="grad", model="logistic", p=16, n_obs=65537, n_points=250,
             engine="auto"),
        # Pointwise log-likelihoods of posterior draws, the input of WAIC and LOO.
        dict(name="pointwise-poisson", op="pointwise", model="poisson", p=24, n_obs=16411,
             n_points=200, engine="auto"),
        # Random-walk sampling at the benchmark's size: 1,024 chains on 2^20
        # observations of a 17-parameter logistic regression.
        dict(name="rwm-logistic", op="sample", model="logistic", p=16, n_obs=1 << 20,
             n_chains=1024, n_iter=40, method="rwm"),
        # Differential evolution on a wide regression with heavy tails.
        dict(name="de-student", op="sample", model="student_t", p=64, n_obs=1 << 18,
             n_chains=2048, n_iter=20, method="de"),
        # Langevin sampling (value and gradient per step, Cholesky
        # preconditioner) of a count regression.
        dict(name="mala-poisson", op="sample", model="poisson", p=24, n_obs=1 << 18,
             n_chains=2048, n_iter=10, method="mala"),
        # Parallel tempering on a mixture: ladders of 16 temperatures, the
        # exchanges on the device.
        dict(name="pt-mixture", op="sample", model="mixture", p=0, n_obs=1 << 18,
             n_chains=2048, n_iter=40, method="pt"),
        # Two-stage sampling: a trained surrogate screens the proposals, the
        # survivors are evaluated exactly.
        dict(name="delayed-logistic", op="delayed", model="logistic", p=16, n_obs=1 << 19,
             n_chains=1024, n_iter=200, method="rwm"),
        # The surrogate's fit from exact pairs, with the default width, batch
        # and learning-rate schedule shape.
        dict(name="train-surrogate", op="train", model="logistic", p=16, n_pairs=65536,
             hidden=128, batch=4096, steps=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _model(rng, names):
    name = rng.choice(names)
    p = {"gaussian": 0, "mixture": 0, "logistic": 16, "poisson": 24,
         "student_t": 64}[name]
    return dict(model=name, p=p)


def draw(rng):
    op = rng.choice(["fit", "loglik", "loglik", "grad", "pointwise", "sample", "sample",
                     "sample", "delayed", "train"])
    if op == "fit":
        m = _model(rng, ["gaussian", "logistic", "poisson"])
        return dict(m, op=op, n_obs=_log(rng, 300, 40000), n_chains=rng.randint(4, 100),
                    n_iter=rng.randint(200, 1000), method="rwm")
    if op in ("loglik", "grad", "pointwise"):
        names = ["gaussian", "logistic", "poisson", "mixture", "student_t"]
        m = _model(rng, names)
        n_obs = _log(rng, 300, 131072)
        most = {"loglik": 1024, "grad": 512, "pointwise": max(1, 4000000 // n_obs)}[op]
        most = min(most, max(1, (1 << 26) // n_obs))
        c = dict(m, op=op, n_obs=n_obs, n_points=_log(rng, 1, min(most, 1024)), engine="auto")
        if op == "loglik" and rng.random() < 0.3:
            c["engine"] = "interp"
        return c
    if op == "sample":
        method = rng.choice(["rwm", "chol", "de", "mala", "pt"])
        m = _model(rng, {"pt": ["mixture"], "mala": ["logistic", "poisson"],
                         "de": ["logistic", "student_t"],
                         "chol": ["logistic", "poisson"]}.get(method,
                                                              ["gaussian", "logistic", "poisson"]))
        C = _log(rng, 6, 2048)
        if method == "pt":
            C = 16 * max(1, C // 16)
        # at most a quarter of the largest case's chains x observations x iterations
        n_obs = _log(rng, 1000, min(1 << 18, (1 << 29) // C))
        most = max(5, min(200, (1 << 32) // (C * n_obs) // (8 if method == "mala" else 1)))
        return dict(m, op=op, n_obs=n_obs, n_chains=C, n_iter=_log(rng, 5, max(6, most)),
                    method=method)
    if op == "delayed":
        return dict(op=op, model="logistic", p=16, n_obs=_log(rng, 1 << 14, 1 << 19),
                    n_chains=_log(rng, 100, 1024), n_iter=rng.randint(40, 200),
                    method=rng.choice(["rwm", "chol"]))
    return dict(op="train", model="logistic", p=16, n_pairs=_log(rng, 5000, 100000),
                hidden=rng.choice([128, 256]), batch=rng.choice([1024, 2048, 4096]),
                steps=rng.randint(30, 100))


# ---------------------------------------------------------------- preparation
def _workload(case, seed, n_obs=None):
    kw = {"p": case["p"]} if case["p"] else {}
    return W.make(case["model"], n_obs=n_obs or case["n_obs"], seed=1000 + seed, **kw)


def _centre(w):
    """The parameters near which the posterior sits."""
    t = w.truth
    if w.name == "gaussian":
        return np.array([t["post_mean"]])
    if w.name == "mixture":
        return np.array([math.log(t["w"] / (1 - t["w"])), t["mu1"], t["mu2"],
                         math.log(t["s1"]), math.log(t["s2"])])
    if w.name == "student_t":
        return np.append(t["beta"], math.log(t["sigma"]))
    return np.asarray(t["beta"], dtype=np.float64)


def _scale(w):
    """About a posterior standard deviation per parameter."""
    return {"gaussian": 2.0, "logistic": 2.5, "poisson": 1.7, "mixture": 3.0,
            "student_t": 2.2}[w.name] / math.sqrt(w.n_obs)


def _session(w, engine="auto"):
    m = w.model
    return _native.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts,
                           m.n_params, w.data, m.n_cols, w.n_obs, engine=_ENGINES[engine])


def _start(case, w, seed):
    """Starting states, step sizes and temperatures of a sampling run."""
    g = np.random.Generator(np.random.PCG64(77 + seed))
    C, d, s = case["n_chains"], w.model.n_params, _scale(w)
    init = _centre(w) + s * g.standard_normal((C, d))
    temps = np.ones(C)
    if case["method"] == "pt":
        ladder = min(16, C)
        temps = np.tile(64.0 ** (np.arange(ladder) / (ladder - 1)), C // ladder)
    k = {"mala": 1.65 / d ** (1 / 6)}.get(case["method"], 2.38 / math.sqrt(d))
    sd = (k * s * np.sqrt(temps))[:, None] * np.ones((C, d))
    L = None
    if case["method"] in ("chol", "mala"):
        low = 0.2 * np.tril(g.standard_normal((d, d)), -1) / math.sqrt(d)
        L = (k * s) * np.tile(np.eye(d) + low, (C, 1, 1))
    return init, sd, temps, L


def prepare(case, seed):
    op = case["op"]
    state = {"case": case, "seed": seed}
    if op == "train":
        # Exact pairs as a run records them: draws around the mode with the
        # log-likelihood there.
        w = _workload(case, seed, n_obs=2000)
        g = np.random.Generator(np.random.PCG64(55 + seed))
        pts = _centre(w) + 2 * _scale(w) * g.standard_normal((case["n_pairs"],
                                                              w.model.n_params))
        with _session(w) as s:
            state["ll"] = s.loglik_batch(pts)
        state["theta"] = pts
        cov = np.cov(pts, rowvar=False)
        state["white"] = np.linalg.inv(np.linalg.cholesky(cov))
        return state
    w = _workload(case, seed)
    if op == "fit":
        # The host's model and data are all that the caller has; the run-time
        # build of the model is once per program, so it is done here.
        state.update(model=w.model, data=w.data,
                     sd=np.full(w.model.n_params, 0.1))
        init = _centre(w) + _scale(w) * np.random.Generator(
            np.random.PCG64(66 + seed)).standard_normal((case["n_chains"], w.model.n_params))
        state["init"] = init
        gpu_metropolis(w.model, w.data[:64], init=init[:4], proposal_sd=state["sd"], n_iter=8,
                       warmup=4)
        return state
    state["session"] = s = _session(w, case.get("engine", "auto"))
    if op in ("loglik", "grad", "pointwise"):
        g = np.random.Generator(np.random.PCG64(88 + seed))
        pts = _centre(w) + _scale(w) * g.standard_normal((case["n_points"], w.model.n_params))
        state["points"] = pts.astype(np.float32).astype(np.float64)  # draws are float32
        s.engine  # the model's build, which every later call shares
        return state
    state["start"] = init, sd, temps, L = _start(case, w, seed)
    s.engine
    if op == "delayed":
        # Warmup as gpu_metropolis does it: exact iterations, their second
        # half recorded, then the fit on the device.
        C = case["n_chains"]
        n = max(8, -(-16384 // C))
        mode = _MODES[case["method"]]
        draws, _, _ = s.run(init, sd, temps, n, seed, mode, proposal_l=L)
        cur = draws.reshape((n, C, -1), order="F")[-1]
        s.record(1 << 20)
        draws, _, _ = s.run(cur, sd, temps, 2 * n, seed + 1, mode, proposal_l=L)
        cur = draws.reshape((2 * n, C, -1), order="F")[-1].astype(np.float64)
        net = _native.Surrogate(w.model.n_params, hidden=128, batch=4096, seed=1)
        s.train_surrogate(net, [(200, 3e-3), (200, 1e-3), (200, 3e-4)])
        s.record(0)
        state.update(net=net, start=(cur, 1.6 * sd, temps, None if L is None else 1.6 * L))
    return state


# ------------------------------------------------------------------ one pass
def run(state):
    c, seed = state["case"], state["seed"]
    op = c["op"]
    if op == "fit":
        fit = gpu_metropolis(state["model"], state["data"], init=state["init"],
                             proposal_sd=state["sd"], n_iter=c["n_iter"], method=c["method"],
                             seed=1 + seed)
        return {"draws": fit.draws, "accept": fit.accept_rate,
                "sd": fit.adaptation["final_proposal_sd"]}
    if op == "train":
        net = _native.Surrogate(state["theta"].shape[1], hidden=c["hidden"], batch=c["batch"],
                                seed=1)
        net.set_whitening(state["theta"].mean(axis=0), state["white"], float(state["ll"].mean()),
                          float(state["ll"].std()))
        n = c["steps"]
        losses = net.train_stages(state["theta"], state["ll"], [(n, 3e-3), (n, 1e-3), (n, 3e-4)])
        params = net.params()
        net.close()
        return {"losses": losses, "params": params}
    s = state["session"]
    if op == "loglik":
        return s.loglik_batch(state["points"])
    if op == "grad":
        return s.grad_batch(state["points"])
    if op == "pointwise":
        return s.loglik_pointwise(state["points"])
    init, sd, temps, L = state["start"]
    if op == "delayed":
        draws, acc, last, exact = s.run_da(state["net"], init, sd, temps, c["n_iter"], seed,
                                           _MODES[c["method"]], proposal_l=L)
        return {"draws": draws, "accept": acc, "last": last, "exact_evals": exact}
    method, d = c["method"], init.shape[1]
    if method == "pt":
        s.set_exchange(min(16, c["n_chains"]), 10)
    draws, acc, last = s.run(init, sd, temps, c["n_iter"], seed,
                             _MODES.get(method, _native.MODE_RWM),
                             2.38 / math.sqrt(2 * d), 1e-3, proposal_l=L)
    return {"draws": draws, "accept": acc, "last": last}


# ------------------------------------------------------- work and exact values
def work(case):
    if case["op"] == "train":
        d, H, B = (case["p"] + 1 + 63) // 64 * 64, case["hidden"], case["batch"]
        steps = 3 * case["steps"]
        flops = steps * B * (2 * d * H * 2 + 2 * H * H * 3)
        return {"bytes": case["n_pairs"] * (case["p"] + 2) * 8.0 + 4.0 * H * (d + H),
                "flops": float(flops)}
    cols = {"gaussian": 1, "mixture": 1}.get(case["model"], case["p"] + 1)
    np_ = {"gaussian": 1, "mixture": 5, "logistic": case["p"] + 1, "poisson": case["p"],
           "student_t": case["p"] + 1}[case["model"]]
    per = {"gaussian": 4, "mixture": 25, "logistic": 2 * np_ + 20, "poisson": 2 * np_ + 15,
           "student_t": 2 * np_ + 20}[case["model"]]
    n = case["n_obs"]
    data = 4.0 * n * cols
    if case["op"] in ("loglik", "grad", "pointwise"):
        P = case["n_points"]
        out = {"loglik": 1, "grad": np_, "pointwise": n}[case["op"]]
        return {"bytes": data + 8.0 * P * (np_ + out),
                "flops": float(P) * n * per * (2 if case["op"] == "grad" else 1)}
    C, T = case["n_chains"], case["n_iter"]
    evals = C * n * (T + 1.0) * (2 if case["method"] == "mala" else 1)
    if case["op"] == "delayed":
        evals *= 0.1  # the screened share
    if case["op"] == "fit":
        data *= 2  # the caller's 64-bit rows
    return {"bytes": data + 4.0 * C * T * np_ + 24.0 * C * np_, "flops": evals * per}


def exact(case, seed):
    if case["op"] not in ("loglik", "grad", "pointwise"):
        return None
    w = _workload(case, seed)
    g = np.random.Generator(np.random.PCG64(88 + seed))
    pts = _centre(w) + _scale(w) * g.standard_normal((case["n_points"], w.model.n_params))
    pts = pts.astype(np.float32).astype(np.float64)
    N, P, name, grad = w.n_obs, pts.shape[0], w.name, case["op"] == "grad"
    y = w.data[:, -1].astype(np.float64)
    X = w.data[:, :-1].astype(np.float64)
    if name == "logistic":
        X = np.concatenate([np.ones((N, 1)), X], axis=1)
    if name == "poisson":
        uniq, inv = np.unique(y, return_inverse=True)
        lfact = np.array([math.lgamma(v + 1.0) for v in uniq])[inv]
    rows = max(1, (1 << 22) // max(1, N))
    out = []
    for k in range(0, P, rows):
        q = pts[k:k + rows]
        if name == "gaussian":
            r = y[None] - q[:, :1]
            v, G = -r * r / 8, (r / 4).sum(axis=1, keepdims=True)
        elif name == "logistic":
            eta = q @ X.T
            v = y * eta - np.logaddexp(0.0, eta)
            G = (y - 1 / (1 + np.exp(-eta))) @ X if grad else None
        elif name == "poisson":
            eta = q @ X.T
            mu = np.exp(eta)
            v = y * eta - mu - lfact
            G = (y - mu) @ X if grad else None
        elif name == "student_t":
            sg = np.exp(q[:, -1:])
            z = (y - q[:, :-1] @ X.T) / sg
            u = 1 + z * z / 4
            v = (math.lgamma(2.5) - math.lgamma(2.0) - 0.5 * math.log(4 * math.pi) - q[:, -1:]
                 - 2.5 * np.log(u))
            if grad:
                e = 1.25 * z / u
                G = np.concatenate([(e / sg) @ X, (e * z - 1).sum(axis=1, keepdims=True)], axis=1)
        else:
            lw, m1, m2, l1, l2 = (q[:, j:j + 1] for j in range(5))
            z1, z2 = (y - m1) / np.exp(l1), (y - m2) / np.exp(l2)
            a = -0.5 * z1 * z1 - l1 - np.logaddexp(0.0, -lw)
            b = -0.5 * z2 * z2 - l2 - np.logaddexp(0.0, lw)
            v = np.logaddexp(a, b)
            if grad:
                ra, rb = np.exp(a - v), np.exp(b - v)
                sw = 1 / (1 + np.exp(-lw))
                G = np.stack([(ra * (1 - sw) - rb * sw).sum(axis=1),
                              (ra * z1 / np.exp(l1)).sum(axis=1),
                              (rb * z2 / np.exp(l2)).sum(axis=1),
                              (ra * (z1 * z1 - 1)).sum(axis=1),
                              (rb * (z2 * z2 - 1)).sum(axis=1)], axis=1)
        out.append(G if grad else v if case["op"] == "pointwise" else v.sum(axis=1))
    return np.concatenate(out).reshape(-1)
