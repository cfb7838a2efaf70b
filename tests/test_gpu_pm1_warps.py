"""Dense +-1 rings in qanneal's order run one warp per slice where there are no
more rings than SMs, else half as many for more than 16 slices.  A read's
result does not depend on it: the first reads of a large call equal a small
call's, and the oracle's.
"""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from qlatanneal_b200.instances import sk_dense
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,P", [(33, 17), (70, 32), (129, 31), (300, 24), (64, 16)])
def test_few_and_many_rings_agree(oracle, n, P):
    model = qa.DenseIsing(*sk_dense(n, 4 + n))
    om = oracle_model(oracle, model)
    steps, seed = 6, 17
    betas = P * np.geomspace(0.02, 2.0, steps) / np.sqrt(n)
    gammas = np.linspace(2.0, 0.05, steps)
    ann = qa.SQAAnnealer(model, qa.SQASchedule.from_vectors(betas, gammas), P)
    few = ann.run_reads(2, 1, reads=3, seed=seed)
    many = ann.run_reads(2, 1, reads=400, seed=seed)
    try:
        oracle.set_update_order("reference")
        for r in range(3):
            best, _, trace, _ = oracle.sqa_run(om, betas, gammas, P, 1, 2, 1, seed, r)
            for res in (few[r], many[r]):
                np.testing.assert_array_equal(res.best_state.as_array(), best)
                np.testing.assert_array_equal(np.asarray(res.energy_trace), trace)
    finally:
        oracle.set_update_order("reference")


@pytest.mark.parametrize("n,P,warps", [(5, 32, 16), (32, 24, 12), (33, 24, 24), (32, 16, 16)])
def test_one_block_has_no_wavefront(n, P, warps):
    """Models of one block of 32 spins gain nothing from a warp for each slice."""
    from qlatanneal_b200 import _lib, autotune
    eng, model = _lib.Engine.get(None), qa.DenseIsing(*sk_dense(n, 1))
    assert autotune._ring_warps(eng, model, P, 3, False, False) == warps
