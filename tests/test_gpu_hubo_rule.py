"""Higher-order models where the rule of the warps of a ring changes: results as the
CPU restatement gives them in both update orders."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from test_gpu_hubo import model
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu


# rings just beyond what the SMs hold with a phase's warps and with a warp per slice, P of
# one, odd, more slices than warps, a P that 16 is no multiple of
@pytest.mark.parametrize("order", ["reference", "checkerboard"])
@pytest.mark.parametrize("n,P,reads", [(33, 7, 149), (33, 7, 593), (40, 16, 296), (40, 16, 297), (30, 1, 2400), (45, 33, 149),
                                       (64, 11, 300), (20, 64, 450)])
def test_matches_oracle(oracle, order, n, P, reads):
    m = model(n, n, 2)
    om = oracle_model(oracle, m)
    steps, seed = 3, 41
    betas, gammas = P * np.geomspace(0.02, 1.5, steps), np.linspace(2.0, 0.05, steps)
    ann = qa.SQAAnnealer(m, qa.SQASchedule.from_vectors(betas, gammas), P)
    try:
        qa.set_update_order(order)
        oracle.set_update_order(order)
        res = ann.run_reads(1, 1, reads=reads, seed=seed)
        for r in sorted({0, reads // 2, reads - 1}):
            best, _, trace, _ = oracle.sqa_run(om, betas, gammas, P, 1, 1, 1, seed, r)
            np.testing.assert_array_equal(res[r].best_state.as_array(), best)
            np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
    finally:
        qa.set_update_order("reference")
        oracle.set_update_order("reference")
