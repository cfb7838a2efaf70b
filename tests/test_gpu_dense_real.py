"""ring_dense_kernel (dense models with real couplings) against the CPU
restatement and against the flip-by-flip generic kernel, which it replaces
(QA_DISABLE_DENSE brings that one back).  Both round every field update and
every sum alike, so spins, energies, traces and counters must be equal.
"""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from qlatanneal_b200.instances import dense_real
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu

# block edges (31, 32, 33), row edges (n % 4, groups of 128 columns: two at a time
# up to 256, four beyond), one slice, two, a number that is no multiple of
# the warps, more than one slice a warp
CASES = [(1, 4, 1, 1), (31, 1, 1, 0), (65, 1, 1, 2), (32, 2, 1, 1), (33, 3, 2, 1), (64, 16, 1, 2), (127, 17, 1, 1), (129, 5, 1, 1),
         (257, 33, 1, 1), (130, 64, 1, 1), (514, 8, 1, 1),
         (256, 3, 1, 1), (388, 4, 1, 1), (641, 3, 1, 1), (770, 2, 1, 1)]


@pytest.mark.parametrize("order", ["reference", "checkerboard"])
@pytest.mark.parametrize("n,P,spb,wls", CASES)
def test_sqa_matches_oracle(oracle, order, n, P, spb, wls):
    model = qa.DenseIsing(*dense_real(n, 10 + n))
    om = oracle_model(oracle, model)
    steps, reads, seed = 6, 2, 91
    # hot (most moves accepted) to cold
    betas = P * np.geomspace(0.02, 3.0, steps) / np.sqrt(n)
    gammas = np.linspace(2.0, 0.05, steps)
    ann = qa.SQAAnnealer(model, qa.SQASchedule.from_vectors(betas, gammas), P)
    try:
        qa.set_update_order(order)
        oracle.set_update_order(order)
        res = ann.run_reads(spb, wls, reads=reads, seed=seed)
        for r in range(reads):
            best, _, trace, _ = oracle.sqa_run(om, betas, gammas, P, 1, spb, wls, seed, r)
            np.testing.assert_array_equal(res[r].best_state.as_array(), best)
            np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
            # reported from the float64 coefficients, not the tracked float32 ones
            assert res[r].best_energy == pytest.approx(oracle.energy64(om, best), rel=1e-12, abs=1e-12)
    finally:
        qa.set_update_order("reference")
        oracle.set_update_order("reference")


def _both(monkeypatch, call):
    a = call()
    monkeypatch.setenv("QA_DISABLE_DENSE", "1")
    b = call()
    monkeypatch.delenv("QA_DISABLE_DENSE")
    return a, b


@pytest.mark.parametrize("n,reads", [(40, 3), (70, 400), (300, 160)])  # 8 and 16 warps, rotated launches
@pytest.mark.parametrize("method", ["sqa", "sqapt", "sqa_chi", "optimal", "qubo"])
def test_equals_generic_kernel(monkeypatch, method, n, reads):
    h, J = dense_real(n, 3)
    model, P, seed = qa.DenseIsing(h, J), 9, 5

    def call():
        if method == "sqa":
            s = qa.SQASchedule.from_vectors(np.linspace(0.2, 6.0, 12), np.linspace(2.0, 0.05, 12))
            ann = qa.SQAAnnealer(model, s, P, 2)
            res = ann.run_reads(1, 1, reads=reads, seed=seed)
        elif method == "sqapt":
            ann = qa.SQAParallelTemperingAnnealer(model, np.geomspace(0.3, 4.0, 4), np.linspace(2.0, 0.1, 4), P)
            res = ann.run_reads(1, 1, 6, 2, reads=max(1, reads // 4), seed=seed)
        elif method == "sqa_chi":
            ann = qa.SQAChiAnnealer(model, P)
            res = ann.run_chi_reads(2.0, 3.0, 0.05, 8, 2, 4, 6, 2, reads=max(1, reads // 4), seed=seed)
        elif method == "optimal":  # bond samples, and couplings J_perp far above the thermal scale
            ann = qa.SQAAnnealer(model, qa.auto_schedule_sqa(4), P)
            res = ann.run_optimal_reads(4.0, 0.1, 1e4, 0.0, num_steps=10, sweeps_per_step=2, worldline_sweeps=1,
                                        calib_probes=3, calib_sweeps=2, reads=max(1, reads // 4), seed=seed)
        else:
            Q = np.triu(np.random.default_rng(8).uniform(-1, 1, (n, n)))
            r = qa.solve(Q, reads=reads, sweeps_per_beta=2, worldline_sweeps=1, trotter_slices=P, seed=seed,
                         schedule=qa.auto_schedule_sqa(6))
            return [np.stack(r.samples), np.array(r.energies), np.array(r.trace)]
        st = ann.last_stats
        name = "average_energy_trace" if method == "sqapt" else "energy_trace"
        return [np.stack([x.best_state.as_array() for x in res]), np.array([x.best_energy for x in res]),
                np.array([getattr(x, name) for x in res]),
                np.array([st.slice_attempts, st.slice_accepts, st.worldline_attempts, st.worldline_accepts])]

    a, b = _both(monkeypatch, call)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


def test_huge_couplings_keep_the_generic_kernel(monkeypatch):
    """2 J beyond float32: the product overflows before the sum, as it did."""
    h, J = dense_real(24, 4)
    J *= 1.2e38
    model = qa.DenseIsing(h, J)
    s = qa.SQASchedule.from_vectors([1e-38, 2e-38], [1.0, 0.5])
    a, b = _both(monkeypatch, lambda: qa.SQAAnnealer(model, s, 4).run_reads(1, 1, reads=3, seed=2))
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x.best_state.as_array(), y.best_state.as_array())


def test_batch_of_uneven_models_equals_single_runs():
    """Exact energies (16 states a CTA) where a CTA's states belong to two models."""
    models = [qa.DenseIsing(*dense_real(n, 20 + n)) for n in (130, 65, 97, 300)]
    s = qa.SQASchedule.from_vectors([0.5, 2.0, 6.0], [2.0, 1.0, 0.1])
    both = qa.BatchRunner().sqa(models, s, 3, reads=5, worldline_sweeps=1, seed=4)
    sa = qa.BatchRunner().anneal(models, qa.AnnealSchedule.from_betas([0.2, 1.0]), 2, reads=5, seed=4)
    for m, x, y in zip(models, both, sa):
        for got, want in ((x, qa.SQAAnnealer(m, s, 3).run_reads(1, 1, reads=5, seed=4)),
                          (y, qa.Annealer(m, qa.AnnealSchedule.from_betas([0.2, 1.0])).run_reads(2, 5, seed=4))):
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a.best_state.as_array(), b.best_state.as_array())
                assert a.best_energy == b.best_energy
                np.testing.assert_array_equal(a.energy_trace, b.energy_trace)
