"""Infinite fields, couplings near the end of float32 and beta = 0 on the dense
and sparse kernels, against the CPU restatement: a field that overflows and a
product that is not a number decide as they do there."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 130, 600])
def test_sa_overflowing_fields(oracle, n):
    """Finite couplings whose sums overflow: infinite fields, at beta = 0 (the
    product is not a number: rejected) and above (accepted or rejected for good)."""
    rng = np.random.default_rng(n)
    J = np.triu(rng.choice([-8e37, 8e37], (n, n)), 1)
    model = qa.DenseIsing(rng.normal(0.0, 1.0, n), J + J.T)
    om = oracle_model(oracle, model)
    betas, spb, seed = np.array([0.0, 1e-39, 0.0, 1e-38, 1.0]), 2, 5
    ann = qa.Annealer(model, qa.AnnealSchedule.from_betas(betas))
    res = ann.run_reads(spb, reads=3, seed=seed)
    acc = 0
    for r in range(3):
        best, _, trace, cnt = oracle.sa_run(om, betas, spb, seed, r)
        acc += cnt[1]
        np.testing.assert_array_equal(res[r].best_state.as_array(), best)
        np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
    assert ann.last_stats.slice_accepts == acc
