"""ring_hubo_kernel (terms of at most four spins) against the CPU restatement and
against the generic kernel (QA_DISABLE_HUBO): equal, real coefficients included."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu


def model(n, seed, per_spin):
    """Terms of two to four spins with real coefficients; with many terms a spin a
    target repeats within a flip's updates and they fill several chunks."""
    rng = np.random.default_rng(seed)
    terms = {}
    for d in (2, 3, 4):
        for _ in range(per_spin * n // d if n >= d else 0):
            terms[tuple(sorted(rng.choice(n, size=d, replace=False).tolist()))] = float(rng.normal())
    terms.update({(i,): float(w) for i, w in enumerate(rng.normal(0.0, 0.3, n))})
    return qa.HigherOrderIsing(terms, n)


# few spins and many terms (every lane touches the others), block edges, one to 64
# slices, slices that are no multiple of the warps
CASES = [(4, 3, 1, 1, 2), (20, 2, 1, 2, 9), (33, 17, 1, 1, 3), (64, 33, 2, 0, 2), (65, 1, 1, 1, 4), (100, 64, 1, 1, 1),
         (300, 8, 1, 1, 3)]


@pytest.mark.parametrize("order", ["reference", "checkerboard"])
@pytest.mark.parametrize("n,P,spb,wls,per", CASES)
def test_sqa_matches_oracle(oracle, order, n, P, spb, wls, per):
    m = model(n, n, per)
    om = oracle_model(oracle, m)
    steps, reads, seed = 5, 2, 31
    betas, gammas = P * np.geomspace(0.02, 1.5, steps), np.linspace(2.0, 0.05, steps)
    ann = qa.SQAAnnealer(m, qa.SQASchedule.from_vectors(betas, gammas), P)
    try:
        qa.set_update_order(order)
        oracle.set_update_order(order)
        res = ann.run_reads(spb, wls, reads=reads, seed=seed)
        acc = np.zeros(4, np.int64)
        for r in range(reads):
            best, _, trace, cnt = oracle.sqa_run(om, betas, gammas, P, 1, spb, wls, seed, r)
            acc += np.asarray(cnt[:4], np.int64)
            np.testing.assert_array_equal(res[r].best_state.as_array(), best)
            np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
        st = ann.last_stats
        assert [st.slice_attempts, st.slice_accepts, st.worldline_attempts, st.worldline_accepts] == acc.tolist()
    finally:
        qa.set_update_order("reference")
        oracle.set_update_order("reference")


@pytest.mark.parametrize("method", ["sqapt", "sqa_chi", "optimal", "many"])
def test_equals_generic_kernel(monkeypatch, method):
    m, seed = model(70, 3, 3), 5

    def call():
        if method == "sqapt":
            ann = qa.SQAParallelTemperingAnnealer(m, np.geomspace(0.3, 4.0, 4), np.linspace(2.0, 0.1, 4), 9)
            res = ann.run_reads(2, 1, 8, 4, reads=40, seed=seed)
            return [x for r in res for x in (r.best_state.as_array(), np.array(r.final_energies),
                                             np.array(r.average_energy_trace))]
        if method == "sqa_chi":
            ann = qa.SQAChiAnnealer(m, 9)
            res = ann.run_chi_reads(2.0, 3.0, 0.05, 8, 2, 4, 6, 2, reads=3, seed=seed)
        elif method == "optimal":
            ann = qa.SQAAnnealer(m, qa.auto_schedule_sqa(4), 9)
            res = ann.run_optimal_reads(4.0, 0.1, 2.0, 0.0, num_steps=10, sweeps_per_step=2, worldline_sweeps=1,
                                        calib_probes=3, calib_sweeps=2, reads=3, seed=seed)
        else:  # more rings than SMs: rotated launches
            ann = qa.SQAAnnealer(m, qa.auto_schedule_sqa(210), 5)
            res = ann.run_reads(1, 1, reads=160, seed=seed)
        return [x for r in res for x in (r.best_state.as_array(), np.array(r.energy_trace))]

    a = call()
    monkeypatch.setenv("QA_DISABLE_HUBO", "1")
    for x, y in zip(a, call()):
        np.testing.assert_array_equal(x, y)
