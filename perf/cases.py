"""The calls this framework is measured on.

Every case is one call of a public entry point -- ``solve()``, an annealer's
``run_reads`` or ``BatchRunner`` -- on a problem that ``prepare`` has in hand:
host arrays, or a model object whose device copy the user's program keeps.
The outputs are everything the call hands back: sampled states (whole numbers),
their energies and the traces.

Ranges (``draw`` spans them): 12 to 2000 spins dense, 512 to 4096 sparse, 200
to 1200 higher-order; 1 to 256 reads; 4 to 64 Trotter slices; couplings +-1 and
real; all four ``solve()`` methods, classical parallel tempering, cluster
sweeps and instance sets.
"""
from __future__ import annotations

import math

import numpy as np

import qlatanneal_b200 as qa
from qlatanneal_b200.instances import dense_real, geometric_betas, regular3, sk_dense


def listed():
    return [
        # one read of a small QUBO with every default of solve(): the call of
        # an interactive session or of a decomposition solver's inner loop;
        # one ring on one SM, all latency
        dict(name="solve_qubo_tiny", kind="solve_qubo", n=24, reads=1, steps=50, spb=20, wls=5, P=32),
        # the ordinary call: a real-valued QUBO as an array, defaults, some reads
        dict(name="solve_qubo", kind="solve_qubo", n=200, reads=32, steps=50, spb=20, wls=5, P=32),
        # a larger, ragged real QUBO with fewer sweeps
        dict(name="solve_qubo_large", kind="solve_qubo", n=900, reads=100, steps=40, spb=2, wls=1, P=16),
        # classical annealing of a spin glass: many short chains
        dict(name="sa_sk", kind="sa_sk", n=256, reads=64, steps=100, spb=10),
        # classical annealing with real couplings, solve()'s default schedule
        dict(name="sa_real", kind="sa_real", n=1000, reads=128, steps=50, spb=4),
        # the dense SQA workload of the benchmark
        dict(name="sqa_sk", kind="sqa_sk", n=512, reads=256, steps=1000, spb=1, wls=1, P=32),
        # the largest dense +-1 instances, a ragged size
        dict(name="sqa_sk_large", kind="sqa_sk", n=2000, reads=128, steps=100, spb=1, wls=1, P=16),
        # parallel tempering over Trotter rings on a sparse graph
        dict(name="sqapt_sparse", kind="sqapt_sparse", n=2048, reads=32, rungs=32, steps=10, spb=20, wls=5, P=16,
             swap=5),
        # a set of sparse instances of uneven size in one call
        dict(name="sqapt_sparse_set", kind="sqapt_set", n=4096, n_min=512, models=6, reads=16, rungs=16, steps=40,
             spb=1, wls=1, P=16, swap=10),
        # higher-order models (three-body terms, real two-body couplings)
        dict(name="sqa_hubo", kind="sqa_hubo", n=1024, reads=128, steps=60, spb=1, wls=1, P=16),
        # the susceptibility-guided schedule: pilot scan and production
        dict(name="sqa_chi", kind="sqa_chi", n=300, reads=32, steps=100, spb=20, points=16, scan=30, burn=10, P=32),
        # classical parallel tempering, swaps after every step: many launches
        dict(name="pt_sk", kind="pt_sk", n=128, reads=32, rungs=24, steps=100, spb=5, swap=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sites(c):
    """Site attempts of one pass (a worldline proposal counts its P sites)."""
    n = c["n"] if c["kind"] != "sqapt_set" else sum(_set_sizes(c))
    P, rungs = c.get("P", 1), c.get("rungs", 1)
    sweeps = c["steps"] * (c["spb"] + c.get("wls", 0) + c.get("cls", 0))
    if c["kind"] == "sqa_chi":
        sweeps += c["points"] * (c["scan"] + c["burn"])
    return n * P * rungs * c["reads"] * sweeps


def _cost(c):
    """Relative time of a case within its kind: attempts, and per accepted
    flip of a dense real model the n fields it changes."""
    dense = c["kind"] in ("solve_qubo", "sa_real")
    # the sweeps of a read are sequential: few reads do not make a pass short
    width = max(1, c["reads"] * c.get("rungs", 1))
    return _sites(c) / width * max(width, 64) * (1.0 + c["n"] / 256.0 if dense else 1.0)


def draw(rng):
    kind = rng.choice(["solve_qubo", "solve_qubo", "sa_sk", "sa_real", "sqa_sk", "sqa_sk", "sqapt_sparse",
                       "sqapt_set", "sqa_hubo", "sqa_chi", "pt_sk", "sqa_cluster"])
    if kind == "solve_qubo":
        c = dict(n=_log_int(rng, 12, 1000), reads=_log_int(rng, 1, 128), steps=rng.choice([30, 50, 80]),
                 spb=rng.choice([1, 2, 5, 20]), wls=rng.choice([0, 1, 5]), P=rng.choice([8, 16, 20, 32]))
    elif kind == "sa_sk":
        c = dict(n=_log_int(rng, 20, 512), reads=_log_int(rng, 1, 256), steps=rng.randint(20, 100),
                 spb=rng.randint(1, 20))
    elif kind == "sa_real":
        c = dict(n=_log_int(rng, 50, 1500), reads=_log_int(rng, 1, 256), steps=50, spb=rng.randint(1, 20))
    elif kind == "sqa_sk":
        c = dict(n=_log_int(rng, 60, 2000), reads=_log_int(rng, 1, 256), steps=rng.randint(50, 1000),
                 spb=rng.choice([1, 1, 2, 5]), wls=rng.choice([0, 1, 1, 2]), P=rng.choice([4, 8, 16, 24, 32, 64]))
    elif kind == "sqapt_sparse":
        c = dict(n=2 * _log_int(rng, 256, 2048), reads=_log_int(rng, 1, 32), rungs=rng.randint(4, 32),
                 steps=rng.randint(5, 20), spb=rng.randint(1, 20), wls=rng.randint(0, 5), P=rng.choice([8, 16, 32]),
                 swap=rng.choice([1, 5, 10]))
    elif kind == "sqapt_set":
        c = dict(n=2 * _log_int(rng, 512, 2048), n_min=512, models=rng.randint(2, 8), reads=_log_int(rng, 1, 16),
                 rungs=rng.randint(4, 16), steps=rng.randint(10, 40), spb=1, wls=1, P=16, swap=10)
    elif kind == "sqa_hubo":
        c = dict(n=_log_int(rng, 200, 1200), reads=_log_int(rng, 1, 128), steps=rng.randint(20, 100), spb=1,
                 wls=rng.choice([0, 1]), P=rng.choice([8, 16, 16, 20]))
    elif kind == "sqa_chi":
        c = dict(n=_log_int(rng, 60, 600), reads=_log_int(rng, 1, 32), steps=100, spb=rng.choice([5, 10, 20]),
                 points=16, scan=30, burn=10, P=rng.choice([16, 32]))
    elif kind == "pt_sk":
        c = dict(n=_log_int(rng, 30, 400), reads=_log_int(rng, 1, 32), rungs=rng.randint(4, 32),
                 steps=rng.randint(20, 100), spb=rng.randint(1, 10), swap=rng.choice([1, 2, 10]))
    else:  # cluster sweeps along imaginary time, real couplings on a sparse graph
        c = dict(n=2 * _log_int(rng, 30, 250), reads=_log_int(rng, 1, 32), steps=rng.randint(10, 40),
                 spb=rng.choice([1, 5]), wls=rng.choice([0, 1]), cls=1, P=rng.choice([8, 16, 32]))
    c = dict(kind=kind, **c)
    # no dearer than the dearest listed case of its kind: fewer steps, then
    # fewer reads, then fewer spins
    caps = [_cost(x) for x in listed() if x["kind"] == kind]
    cap = max(caps) if caps else 3e7
    while _cost(c) > cap:
        if c["steps"] > 10 and kind != "sqa_chi":
            c["steps"] = max(10, c["steps"] * 3 // 4)
        elif c["spb"] > 1:
            c["spb"] = max(1, c["spb"] * 3 // 4)
        elif c["reads"] > 1 and c["reads"] * c.get("rungs", 1) > 64:
            c["reads"] = max(1, c["reads"] * 3 // 4)
        else:
            c["n"] = max(c.get("n_min", 12), (c["n"] * 3 // 8) * 2)
    return c


def _set_sizes(c):
    """Even sizes spread over [n_min, n], largest first."""
    k = c["models"]
    return [2 * int(round((c["n_min"] + (c["n"] - c["n_min"]) * (k - 1 - i) / max(k - 1, 1)) / 2)) for i in range(k)]


def _qubo(n, seed):
    """A dense real QUBO: off-diagonal weights in (-1, 1), linear terms on the diagonal."""
    rng = np.random.default_rng(seed)
    Q = np.triu(rng.uniform(-1.0, 1.0, (n, n)), 1)
    Q[np.diag_indices(n)] = rng.normal(0.0, 1.0, n)
    return Q


def _hubo(n, seed):
    """3n three-body terms (+-1), 2n two-body terms (uniform in (-1, 1)) and linear terms N(0, 0.2^2)."""
    rng = np.random.default_rng(seed)

    def tuples(k, count):
        got = np.empty((0, k), np.int64)
        while len(got) < count:
            t = np.sort(rng.integers(0, n, (2 * count, k)), axis=1)
            t = t[np.all(t[:, 1:] != t[:, :-1], axis=1)]
            got = np.unique(np.concatenate([got, t]), axis=0)
        return got[rng.permutation(len(got))[:count]].tolist()

    terms = {tuple(t): float(w) for t, w in zip(tuples(3, 3 * n), rng.choice([-1.0, 1.0], 3 * n))}
    terms.update({tuple(t): float(w) for t, w in zip(tuples(2, 2 * n), rng.uniform(-1.0, 1.0, 2 * n))})
    terms.update({(i,): float(w) for i, w in enumerate(rng.normal(0.0, 0.2, n))})
    return terms


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = dict(case=case, seed=1 + seed)
    if kind == "solve_qubo":
        st["Q"] = _qubo(c["n"], seed)  # the user's array: solve() takes it from here
        st["schedule"] = qa.auto_schedule_sqa(c["steps"])
        return st
    if kind in ("sa_sk", "sqa_sk", "sqa_chi", "pt_sk"):
        h, J = sk_dense(c["n"], seed, h_sigma=0.1 if kind == "sqa_sk" else 0.0)
        st["model"] = qa.DenseIsing(h, J)
    elif kind == "sa_real":
        st["model"] = qa.DenseIsing(*dense_real(c["n"], seed))
    elif kind == "sqapt_sparse":
        st["model"] = qa.SparseIsing(*regular3(c["n"], seed), c["n"])
    elif kind == "sqapt_set":
        st["models"] = [qa.SparseIsing(*regular3(n, seed + 1000 * k), n) for k, n in enumerate(_set_sizes(c))]
        st["runner"] = qa.BatchRunner()
    elif kind == "sqa_hubo":
        st["model"] = qa.HigherOrderIsing(_hubo(c["n"], seed), c["n"])
    elif kind == "sqa_cluster":
        h, edges = regular3(c["n"], seed)
        w = np.random.default_rng(seed + 1).uniform(-1.0, 1.0, len(edges))
        st["model"] = qa.SparseIsing(h, [(i, j, float(x)) for (i, j, _), x in zip(edges, w)], c["n"])
    steps = c["steps"]
    if kind == "sa_sk":
        st["schedule"] = qa.AnnealSchedule.from_betas(geometric_betas(0.1, 5.0, steps))
    elif kind == "sa_real":
        st["schedule"] = qa.auto_schedule_sa(steps)
    elif kind == "sqa_sk":
        st["schedule"] = qa.SQASchedule.from_vectors(np.full(steps, 0.5 * c["P"]), np.linspace(3.0, 0.01, steps))
    elif kind == "sqa_hubo":
        st["schedule"] = qa.SQASchedule.from_vectors(np.linspace(0.1, 4.0, steps), np.linspace(2.0, 0.02, steps))
    elif kind == "sqa_chi":
        st["schedule"] = qa.auto_schedule_sqa(steps, gamma_start=3.0)
    elif kind == "sqa_cluster":
        st["schedule"] = qa.auto_schedule_sqa(steps)
    elif kind in ("sqapt_sparse", "sqapt_set"):
        st["betas"] = 0.2 * (4.0 / 0.2) ** (np.arange(c["rungs"]) / (c["rungs"] - 1))
        st["gammas"] = np.linspace(2.5, 0.05, c["rungs"])
    elif kind == "pt_sk":
        st["annealer"] = qa.ParallelTemperingAnnealer(st["model"], geometric_betas(0.05, 2.0, c["rungs"]))
    return st


def _solved(r):
    return dict(samples=np.stack(r.samples), energies=np.array(r.energies), best=r.best_sample,
                best_energy=r.best_energy, trace=np.array(r.trace))


def _tempered(res):
    return dict(best=np.stack([r.best_state.as_array() for r in res]),
                best_energies=np.array([r.best_energy for r in res]),
                final=np.stack([s.as_array() for r in res for s in r.final_states]),
                final_energies=np.array([r.final_energies for r in res]),
                average_energy=np.array([r.average_energy_trace for r in res]),
                swaps=np.array([r.swap_acceptance_trace for r in res]))


def run(state):
    c, kind, seed = state["case"], state["case"]["kind"], state["seed"]
    if kind == "solve_qubo":
        return _solved(qa.solve(state["Q"], reads=c["reads"], sweeps_per_beta=c["spb"], worldline_sweeps=c["wls"],
                                trotter_slices=c["P"], schedule=state["schedule"], seed=seed, return_bits=True))
    if kind in ("sa_sk", "sa_real"):
        return _solved(qa.solve(state["model"], method="sa", reads=c["reads"], sweeps_per_beta=c["spb"],
                                schedule=state["schedule"], seed=seed))
    if kind in ("sqa_sk", "sqa_hubo", "sqa_cluster"):
        return _solved(qa.solve(state["model"], method="sqa", reads=c["reads"], sweeps_per_beta=c["spb"],
                                worldline_sweeps=c["wls"], cluster_sweeps=c.get("cls", 0), trotter_slices=c["P"],
                                schedule=state["schedule"], seed=seed))
    if kind == "sqa_chi":
        return _solved(qa.solve(state["model"], method="sqa_chi", reads=c["reads"], sweeps_per_beta=c["spb"],
                                trotter_slices=c["P"], schedule=state["schedule"], optimal_num_steps=c["steps"],
                                optimal_beta=4.0, chi_scan_points=c["points"], chi_scan_sweeps=c["scan"],
                                chi_scan_burn=c["burn"], seed=seed))
    if kind == "sqapt_sparse":
        return _solved(qa.solve(state["model"], method="sqapt", reads=c["reads"], sweeps_per_beta=c["spb"],
                                worldline_sweeps=c["wls"], trotter_slices=c["P"], pt_steps=c["steps"],
                                swap_interval=c["swap"], pt_betas=state["betas"], pt_gammas=state["gammas"],
                                schedule=qa.auto_schedule_sqa(), seed=seed))
    if kind == "sqapt_set":
        res = state["runner"].sqapt(state["models"], state["betas"], state["gammas"], c["P"], c["spb"], c["wls"],
                                    c["steps"], c["swap"], reads=c["reads"], seed=seed)
        return [_tempered(reads) for reads in res]
    res = state["annealer"].run_reads(c["spb"], c["steps"], c["swap"], reads=c["reads"], seed=seed)
    return _tempered(res)


# Arithmetic no sweep can do without, per site attempt: h + g, the sign, the
# product with 2 beta / P, the Trotter term and its subtraction, the threshold
# (one operation) and the comparison.
_FLOPS_PER_SITE = 7


def work(case):
    c, kind = case, case["kind"]
    sizes = _set_sizes(c) if kind == "sqapt_set" else [c["n"]]
    total = 0
    for n in sizes:
        if kind in ("solve_qubo", "sa_real"):
            total += 8 * (n * n + n)  # float64 couplings and fields
        elif kind in ("sa_sk", "sqa_sk", "sqa_chi", "pt_sk"):
            total += n * n // 8 + 8 * n  # a sign per coupling, the fields
        elif kind == "sqa_hubo":
            total += 3 * n * 14 + 2 * n * 16 + 8 * n  # spins (2 bytes each) and coefficient of each term
        else:
            total += 3 * n // 2 * 12 + 8 * n  # an edge: two spins and a weight
        reads, steps = c["reads"], c["steps"]
        total += reads * (n + 8 + 8 * steps)  # best states, energies, traces
        if kind in ("sqapt_set", "pt_sk"):
            total += reads * (c["rungs"] * (n + 8) + 8 * steps)
    return {"bytes": int(total), "flops": int(_FLOPS_PER_SITE * _sites(c))}


def exact(case, seed):
    """Every output is a sample of a Markov chain (or the energy of one): it
    follows from the whole sequence of accept / reject decisions on the
    engine's own random numbers, so no output has a value of its own in 64
    bits that plain numpy could give."""
    return None
