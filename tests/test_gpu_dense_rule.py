"""The checkerboard order of dense models with real couplings where the rule of
the warps changes (rings against SMs, slices of a phase against an SM's 16 warps,
two blocks of spins): results as the CPU restatement gives them."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from qlatanneal_b200.instances import dense_real
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu


# a phase's warps, half of an odd number of slices, one slice, rings just beyond what
# the SMs hold (148 SMs: 149, 297, 593 rings), the last n of ring_kernel and the first beyond
@pytest.mark.parametrize("n,P,reads", [(64, 7, 149), (64, 7, 593), (65, 7, 593), (64, 17, 149), (65, 33, 149), (40, 16, 296),
                                       (40, 16, 297), (30, 1, 2400), (66, 1, 2400), (260, 9, 300)])
def test_checkerboard_matches_oracle(oracle, n, P, reads):
    model = qa.DenseIsing(*dense_real(n, n))
    om = oracle_model(oracle, model)
    steps, seed = 4, 37
    betas, gammas = P * np.geomspace(0.02, 3.0, steps) / np.sqrt(n), np.linspace(2.0, 0.05, steps)
    ann = qa.SQAAnnealer(model, qa.SQASchedule.from_vectors(betas, gammas), P)
    try:
        qa.set_update_order("checkerboard")
        oracle.set_update_order("checkerboard")
        res = ann.run_reads(1, 1, reads=reads, seed=seed)
        for r in sorted({0, reads // 2, reads - 1}):
            best, _, trace, _ = oracle.sqa_run(om, betas, gammas, P, 1, 1, 1, seed, r)
            np.testing.assert_array_equal(res[r].best_state.as_array(), best)
            np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
    finally:
        qa.set_update_order("reference")
        oracle.set_update_order("reference")


@pytest.mark.parametrize("n,P,reads,warps", [
    (84, 20, 371, 5),    # 3 rings an SM, 10 slices in two rounds: one wave (8 warps: two rounds as well, two waves)
    (84, 20, 148, 16),   # no more rings than SMs
    (400, 24, 450, 4),   # 4 rings an SM, as many as shared memory holds
    (66, 12, 1200, 3)])
def test_warps_by_waves_and_rounds(n, P, reads, warps):
    from qlatanneal_b200 import _lib, autotune
    eng = _lib.Engine.get(None)
    assert autotune._ring_warps(eng, qa.DenseIsing(*dense_real(n, 1)), P, reads, True, False) == warps
