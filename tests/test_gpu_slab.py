"""ring_slab_kernel (sparse models in neighbour records) against the CPU
restatement, and against ring_sparse_kernel (QA_DISABLE_SLAB) for the methods
that share it.  Integer couplings: everything is exact, so everything is equal.
"""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from qlatanneal_b200.instances import regular3
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu


def ring_model(n, seed, real_h=True):
    """A cycle with chords: up to four neighbours, couplings up to +-127, real
    fields; neighbours in one block and (ascending order) in neighbouring ones."""
    rng = np.random.default_rng(seed)
    edges = {(min(i, (i + 1) % n), max(i, (i + 1) % n)) for i in range(n) if n > 1 and i != (i + 1) % n}
    edges |= {(i, i + n // 2) for i in range(n // 2) if n > 5}
    w = rng.choice([-127.0, -3.0, -1.0, 1.0, 2.0, 127.0], size=len(edges))
    h = rng.normal(0.0, 0.7, n) if real_h else np.zeros(n)
    return qa.SparseIsing(h, [(a, b, float(v)) for (a, b), v in zip(sorted(edges), w)], n)


# one spin, a short block, block and 128-position edges, several groups of 128
# positions a warp and fewer than warps; one slice to 64, odd numbers, both word sizes
CASES = [(1, 3, 1, 1), (2, 1, 2, 0), (31, 2, 1, 1), (32, 5, 1, 2), (33, 33, 1, 1), (127, 4, 2, 1), (128, 31, 1, 1),
         (129, 32, 1, 1), (200, 64, 1, 1), (640, 7, 1, 1), (1500, 16, 1, 1)]


@pytest.mark.parametrize("order", ["reference", "checkerboard"])
@pytest.mark.parametrize("n,P,spb,wls", CASES)
def test_sqa_matches_oracle(oracle, order, n, P, spb, wls):
    model = ring_model(n, n) if n % 2 or n < 4 else qa.SparseIsing(*regular3(n, n), n)
    om = oracle_model(oracle, model)
    steps, reads, seed = 6, 2, 17
    betas = P * np.geomspace(0.01, 2.0, steps)  # most moves accepted, then few
    gammas = np.linspace(2.0, 0.05, steps)
    ann = qa.SQAAnnealer(model, qa.SQASchedule.from_vectors(betas, gammas), P)
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


@pytest.mark.parametrize("n,reads", [(64, 2), (300, 100)])
@pytest.mark.parametrize("method", ["sqapt", "sqa_chi", "optimal", "pt", "set"])
def test_equals_sparse_kernel(monkeypatch, method, n, reads):
    model, seed = ring_model(n, 3, real_h=False), 5

    def call():
        if method == "sqapt":
            ann = qa.SQAParallelTemperingAnnealer(model, np.geomspace(0.3, 4.0, 4), np.linspace(2.0, 0.1, 4), 9)
            res = ann.run_reads(2, 1, 8, 4, reads=reads, seed=seed)
        elif method == "sqa_chi":
            ann = qa.SQAChiAnnealer(model, 9)
            res = ann.run_chi_reads(2.0, 3.0, 0.05, 8, 2, 4, 6, 2, reads=reads, seed=seed)
        elif method == "optimal":
            ann = qa.SQAAnnealer(model, qa.auto_schedule_sqa(4), 9)
            res = ann.run_optimal_reads(4.0, 0.1, 2.0, 0.0, num_steps=10, sweeps_per_step=2, worldline_sweeps=1,
                                        calib_probes=3, calib_sweeps=2, reads=reads, seed=seed)
        elif method == "pt":
            ann = qa.ParallelTemperingAnnealer(model, np.geomspace(0.05, 2.0, 4))
            res = ann.run_reads(2, 6, 2, reads=reads, seed=seed)
        else:  # uneven models, each on its own plan
            models = [ring_model(k, k) for k in (n, 40, 129)]
            out = qa.BatchRunner().sqapt(models, np.geomspace(0.3, 4.0, 4), np.linspace(2.0, 0.1, 4), 9, 1, 1, 6, 3,
                                         reads=max(2, reads // 4), seed=seed)
            return [x for rr in out for r in rr for x in (r.best_state.as_array(), np.array(r.final_energies),
                                                          np.array(r.average_energy_trace))]
        return [x for r in res for x in (r.best_state.as_array(), np.array([r.best_energy]))] + [
            np.array([getattr(r, "average_energy_trace", None) or r.energy_trace for r in res])]

    a = call()
    monkeypatch.setenv("QA_DISABLE_SLAB", "1")
    for x, y in zip(a, call()):
        np.testing.assert_array_equal(x, y)
