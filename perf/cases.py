"""Timing cases of the engine: what its users call, from the smallest call to
full ensembles.

A case is a dict of plain values.  Its model is one of the generator's
families at the case's sizes with every rate constant scaled by a lognormal
factor of the seed (a model whose constants came from a fit), so another seed
is another model and another Philox key.  The cases call the package's public
Python entry points: ``Model.simulate``, ``Model.simulate_static``,
``Model.sensitivity``, ``simulate_batch`` and ``Model.eval_leap``.
"""
from __future__ import annotations

import numpy as np

from tau_leaping_gb300 import Model
from tau_leaping_gb300.model import simulate_batch


def _case(name, entry, family, **kw):
    c = dict(entry=entry, family=family, n_species=0, n_channels=0, gen_seed=0, pop_bits=32, x0_max=0, t_final=1.0,
             n=1, intervals=1, tracked=0, keep_samples=False, sets=0, max_steps=0)
    unknown = set(kw) - set(c)
    assert not unknown, unknown
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a handful of trajectories in a latency-bound
        # loop, through the entry point that never allocates
        _case("dimer_static", "static", "dimer", x0_max=100000, t_final=1.0, n=32, tracked=2),
        # the dimerisation-decay ensemble on a time grid, every species
        _case("dimer_ensemble", "simulate", "dimer", x0_max=100000, t_final=10.0, n=10000, intervals=10),
        # small populations: mostly direct-method steps; time series kept per
        # realization (what a user plots), a 12 x 20 network
        _case("small_series", "simulate", "toy", n_species=12, n_channels=20, gen_seed=5, x0_max=500, t_final=0.2,
              n=5000, intervals=20, tracked=4, keep_samples=True),
        # a mid-sized network with 64-bit populations and ragged sizes on a
        # large ensemble
        _case("net_ragged64", "simulate", "toy", n_species=45, n_channels=83, gen_seed=3, pop_bits=64, x0_max=10000,
              t_final=0.004, n=50001, tracked=3),
        # the headline network, a large ensemble to an early time
        _case("toy_large", "simulate", "toy", n_species=128, n_channels=256, gen_seed=7, x0_max=10000,
              t_final=0.0005, n=60000, tracked=2),
        # the same network, an ordinary ensemble, every species on a grid
        _case("toy_ordinary", "simulate", "toy", n_species=128, n_channels=256, gen_seed=7, x0_max=10000,
              t_final=0.002, n=4000, intervals=8),
        # cyclic chain of 1024 species, every species' statistics
        _case("chain_1024", "simulate", "chain", n_species=1024, t_final=1.0, n=8192),
        # colloidal aggregation, 31 250 channels, 64-bit populations
        _case("colloid_250", "simulate", "colloid", n_species=250, pop_bits=64, t_final=0.01, n=1216, tracked=2),
        # the same family past shared memory: the state lives in L2
        _case("colloid_400", "simulate", "colloid", n_species=400, pop_bits=64, t_final=0.004, n=304, tracked=2),
        # gradients of two species' means with respect to every rate
        _case("toy_gradient", "sensitivity", "toy", n_species=128, n_channels=256, gen_seed=7, x0_max=10000,
              t_final=0.002, n=4096, tracked=2),
        # a parameter sweep with gradients: rate sets of two models with
        # uneven end times in one launch
        _case("sweep_batch", "batch", "dimer", x0_max=100000, t_final=4.0, n=1024, sets=16, tracked=2),
        # leap quantities of many states (propensities, criticality, moments
        # and the step bound), as an analysis of a stored trajectory asks
        _case("leap_states", "eval", "toy", n_species=128, n_channels=256, gen_seed=7, x0_max=10000, n=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["dimer", "toy", "toy", "net", "net", "chain", "colloid", "gradient", "batch", "eval"])
    bits = rng.choice([32, 32, 64])
    if kind == "dimer":
        return _case(None, rng.choice(["simulate", "static"]), "dimer", pop_bits=bits, x0_max=_log_int(rng, 20000, 200000),
                     t_final=round(rng.uniform(0.5, 10.0), 3), n=_log_int(rng, 1, 20000),
                     intervals=rng.randint(1, 12), tracked=rng.randint(1, 3))
    if kind == "toy":  # the headline network, other ensembles
        n = _log_int(rng, 300, 60000)
        return _case(None, "simulate", "toy", n_species=128, n_channels=256, gen_seed=7, x0_max=10000, pop_bits=bits,
                     t_final=round(0.0005 * (60000 / n) ** 0.5, 6), n=n, intervals=rng.randint(1, 10),
                     tracked=rng.choice([1, 2, 17, 0]), keep_samples=rng.random() < 0.2 and n < 5000)
    if kind == "net":  # other networks; a step cap bounds the stiff ones
        N = _log_int(rng, 8, 300)
        n = _log_int(rng, 100, 60000)
        return _case(None, "simulate", "toy", n_species=N, n_channels=int(N * rng.uniform(1.0, 2.5)),
                     gen_seed=rng.randint(1, 99), x0_max=_log_int(rng, 1000, 50000), pop_bits=bits,
                     t_final=0.01, n=n, intervals=rng.randint(1, 5), tracked=rng.randint(1, min(N, 9)),
                     max_steps=300)
    if kind == "chain":
        N = _log_int(rng, 17, 2000)
        return _case(None, "simulate", "chain", n_species=N, pop_bits=bits, t_final=round(rng.uniform(0.3, 1.5), 3),
                     n=max(64, int(rng.uniform(0.1, 1.0) * 8e6 / N)), tracked=rng.choice([0, 1, 5]))
    if kind == "colloid":
        N = _log_int(rng, 24, 330)
        return _case(None, "simulate", "colloid", n_species=N, pop_bits=rng.choice([64, 64, 32]), t_final=0.005,
                     n=max(32, int(rng.uniform(0.2, 1.0) * 1.2e8 / (N * N))), intervals=rng.randint(1, 3), tracked=2)
    if kind == "gradient":
        return _case(None, "sensitivity", "toy", n_species=128, n_channels=256, gen_seed=7, x0_max=10000,
                     t_final=round(rng.uniform(0.0002, 0.002), 6), n=_log_int(rng, 200, 4096),
                     tracked=rng.randint(1, 4))
    if kind == "batch":
        return _case(None, "batch", "dimer", x0_max=_log_int(rng, 20000, 200000), t_final=round(rng.uniform(1.0, 4.0), 3),
                     n=_log_int(rng, 64, 1024), sets=rng.randint(2, 16), tracked=2)
    return _case(None, "eval", "toy", n_species=128, n_channels=256, gen_seed=7, x0_max=10000,
                 n=_log_int(rng, 16, 2048))


def _model(c, rng):
    kw = dict(pop_bits=c["pop_bits"])
    if c["family"] != "dimer":
        kw["n_species"] = c["n_species"]
    if c["family"] == "toy":
        kw.update(n_channels=c["n_channels"], seed=c["gen_seed"], x0_min=0, x0_max=c["x0_max"])
    elif c["family"] == "dimer":
        kw.update(x0_min=c["x0_max"], x0_max=c["x0_max"])
    base = Model.generate(c["family"], **kw)
    d = base.desc()
    base.close()
    d["rate"] = d["rate"] * rng.lognormal(0.0, 0.05, size=len(d["rate"]))
    return Model.from_arrays(**d, pop_bits=c["pop_bits"]), d


def _tracked(c, m):
    return list(range(c["tracked"] or m.n_species))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    m, d = _model(case, rng)
    s = {"case": case, "model": m, "tracked": _tracked(case, m), "seed": int(rng.integers(1, 1 << 62))}
    if case["entry"] == "static":
        # the entry point wants the tables resident: one call uploads them
        m.simulate(1e-6, 1, tracked=[0])
    elif case["entry"] == "batch":
        toy = Model.generate("toy")
        sets, few = case["sets"], max(1, case["sets"] // 4)
        s["items"] = [
            dict(model=m, t_final=case["t_final"], n=case["n"], seed=s["seed"], tracked=s["tracked"],
                 rate_sets=d["rate"][None, :] * rng.lognormal(0.0, 0.2, size=(sets, m.n_channels)),
                 t_final_sets=case["t_final"] * rng.uniform(0.1, 1.0, size=sets), sensitivity=True),
            dict(model=toy, t_final=0.002, n=max(1, case["n"] // 4), seed=s["seed"], tracked=[0, 4],
                 rate_sets=toy.desc()["rate"][None, :] * rng.lognormal(0.0, 0.2, size=(few, toy.n_channels)),
                 t_final_sets=0.002 * rng.uniform(0.5, 1.0, size=few), sensitivity=True)]
    elif case["entry"] == "eval":
        s["x"] = (d["x0"][None, :] * rng.uniform(0.0, 2.0, size=(case["n"], m.n_species))).astype(np.int64)
        s["rate"] = d
    return s


def run(state):
    c, m = state["case"], state["model"]
    if c["entry"] == "eval":
        return m.eval_leap(state["x"])
    if c["entry"] == "sensitivity":
        r = m.sensitivity(c["t_final"], c["n"], seed=state["seed"], tracked=state["tracked"])
        return {k: r[k] for k in ("grad", "stderr", "mean_final", "leaps", "ssa_steps")}
    if c["entry"] == "batch":
        out = simulate_batch(state["items"])
        return [{k: o[k] for k in ("mean", "stddev", "grad", "stderr", "mean_final", "leaps", "ssa_steps")} for o in out]
    if c["entry"] == "static":
        r = m.simulate_static(c["t_final"], c["n"], seed=state["seed"], intervals=c["intervals"],
                              tracked=state["tracked"])
    else:
        r = m.simulate(c["t_final"], c["n"], seed=state["seed"], intervals=c["intervals"], tracked=state["tracked"],
                       keep_samples=c["keep_samples"], max_steps=c["max_steps"], allow_truncation=True)
    out = {"times": r.times, "mean": r.mean, "stddev": r.stddev, "leaps": r.leaps, "ssa": r.ssa_steps,
           "rejections": r.rejections, "truncated": r.truncated}
    if c["keep_samples"]:
        out["samples"] = r.samples
    return out


# Element operations of one realization-step: per channel a propensity and a
# Poisson draw, per net entry the two moment FMAs and the integer update.
def _ops(m):
    return 2 * m.n_channels + 3 * m.nnz_net


def work(case):
    """Operations from a pilot's steps per realization; bytes: the model once,
    the samples written and read once by the statistics, the results."""
    c = dict(case)
    m, _ = _model(c, np.random.default_rng(1))
    tr = _tracked(c, m)
    tables = 12 * m.n_channels + 8 * m.nnz_net + 8 * m.n_species
    if c["entry"] == "eval":
        # populations in; propensities, criticality, moments and bounds out
        return {"bytes": float(c["n"] * (8 * m.n_species + 5 * m.n_channels + 8 * m.n_species + 12) + tables),
                "flops": float(c["n"] * (3 * m.n_channels + 4 * m.nnz_net))}
    sets, share = max(1, c["sets"]), 0.55 if c["entry"] == "batch" else 1.0  # mean end time over the sets
    n = min(c["n"], 32)
    r = m.simulate(c["t_final"], n, seed=1, tracked=[0], max_steps=c["max_steps"], allow_truncation=True)
    steps = (r.leaps + r.ssa_steps) / n * c["n"] * sets * share
    flops = steps * _ops(m)
    width = 8 if m.pop_bits == 64 else 4
    samples = sets * c["n"] * (c["intervals"] + 1) * len(tr) * width
    if c["entry"] in ("sensitivity", "batch"):
        samples += 4 * sets * c["n"] * m.n_channels  # scores
        flops += 3 * steps * m.n_channels
    if c["entry"] == "batch":
        toy = Model.generate("toy")
        few, nt = max(1, c["sets"] // 4), max(1, c["n"] // 4)
        r = toy.simulate(0.0015, 32, seed=1, tracked=[0])
        flops += (r.leaps + r.ssa_steps) / 32 * few * nt * (_ops(toy) + 3 * toy.n_channels)
        samples += 4 * few * nt * toy.n_channels
    return {"bytes": float(2 * samples + tables), "flops": float(flops)}


def exact(case, seed):
    """Leap quantities in FP64 (Cao, Gillespie, Petzold 2006); the simulations'
    outputs are statistics of integer trajectories that FP32 steps draw."""
    if case["entry"] != "eval":
        return None
    s = prepare(case, seed)
    m, x, rate = s["model"], s["x"], s["rate"]["rate"].astype(np.float32).astype(np.float64)
    t = m.tables()
    order, s0, s1 = (t[k].astype(np.int64) for k in ("order", "s0", "s1"))
    xf = x.astype(np.float64)
    x0, x1 = xf[:, s0], xf[:, s1]
    a = rate * np.where(order == 0, 1.0, x0)
    a = np.abs(np.where(order == 2, a * x1, np.where(order == 3, a * (x0 - 1) * 0.5, a)))
    nc = 5
    crit = (order != 0) & ((x0 < np.where(order == 3, 2 * nc, nc)) | ((order == 2) & (x1 < nc)))
    N = m.n_species
    V = np.zeros((N, m.n_channels))
    d = s["rate"]
    for j in range(m.n_channels):
        for q in range(d["col_ptr"][j], d["col_ptr"][j + 1]):
            V[d["row_ind"][q], j] += d["stoich"][q]
    anc = np.where(crit, 0.0, a)
    mu, s2 = anc @ V.T, anc @ (V * V).T
    kind = np.zeros(N, np.int64)
    for j in range(m.n_channels):
        if order[j] == 1:
            kind[s0[j]] = max(kind[s0[j]], 1)
        elif order[j] == 2:
            kind[s0[j]], kind[s1[j]] = max(kind[s0[j]], 2), max(kind[s1[j]], 2)
        elif order[j] == 3:
            kind[s0[j]] = 3
    with np.errstate(divide="ignore", invalid="ignore"):
        g = np.where(kind == 3, np.where(xf >= 2, 2 + 1 / (xf - 1), 3.0), kind.astype(np.float64))
        num = np.maximum(float(np.float32(0.03)) * xf / g, 1.0)
        b = np.minimum(np.where(mu != 0, num / np.abs(mu), np.inf), np.where(s2 != 0, num * num / s2, np.inf))
    tau = np.min(np.where(kind > 0, b, np.inf), axis=1)
    return {"a": a, "crit": None, "mu": mu, "sigma2": s2, "tau1": tau, "a0": a.sum(axis=1)}
