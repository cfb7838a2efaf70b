"""sa_dense_kernel (dense SA: +-1 couplings in bits, other couplings in float32
rows) against the CPU restatement: spins, traces and counters equal."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from qlatanneal_b200.instances import dense_real, sk_dense
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu


# short blocks, block and 128-column edges, more than 512 and 1024 columns (pieces of a row)
@pytest.mark.parametrize("n", [1, 31, 33, 128, 130, 511, 516, 1029])
@pytest.mark.parametrize("kind", ["pm1", "real"])
def test_sa_matches_oracle(oracle, kind, n):
    h, J = sk_dense(n, n, h_sigma=0.2) if kind == "pm1" else dense_real(n, n)
    model = qa.DenseIsing(h, J)
    om = oracle_model(oracle, model)
    # infinite temperature (every move accepted, no limit) to cold
    betas = np.concatenate([[0.0], np.geomspace(1e-3, 3.0, 5) / np.sqrt(n)])
    reads, spb, seed = 2, 2, 23
    ann = qa.Annealer(model, qa.AnnealSchedule.from_betas(betas))
    res = ann.run_reads(spb, reads=reads, seed=seed)
    acc = 0
    for r in range(reads):
        best, _, trace, cnt = oracle.sa_run(om, betas, spb, seed, r)
        acc += cnt[1]
        np.testing.assert_array_equal(res[r].best_state.as_array(), best)
        np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
        assert res[r].best_energy == pytest.approx(oracle.energy64(om, best), rel=1e-12, abs=1e-12)
    assert ann.last_stats.slice_accepts == acc


def test_batch_of_uneven_models():
    models = [qa.DenseIsing(*dense_real(n, n)) for n in (40, 300, 129)]
    sched = qa.AnnealSchedule.from_betas([0.05, 0.3, 1.0])
    for m, x in zip(models, qa.BatchRunner().anneal(models, sched, 3, reads=4, seed=9)):
        for a, b in zip(x, qa.Annealer(m, sched).run_reads(3, 4, seed=9)):
            np.testing.assert_array_equal(a.best_state.as_array(), b.best_state.as_array())
            np.testing.assert_array_equal(a.energy_trace, b.energy_trace)
