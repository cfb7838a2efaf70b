"""The checkerboard order of sparse models in neighbour records, either side of
the line between ring_sparse_kernel and ring_slab_kernel: results as the CPU
restatement gives them."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from test_gpu_parity_sa_sqa import oracle_model
from test_gpu_slab import ring_model

pytestmark = pytest.mark.gpu


# (spins, slices, reads): P = 31 .. 64 where the slab kernel takes one ring (both word
# sizes), the last spin counts before it does, and many rings of a small model
@pytest.mark.parametrize("n,P,reads", [(213, 31, 1), (221, 32, 1), (513, 33, 2), (461, 64, 1), (460, 64, 1), (212, 31, 1),
                                       (100, 16, 2), (101, 16, 2), (40, 32, 700), (16, 1, 2)])
def test_checkerboard_matches_oracle(oracle, n, P, reads):
    model = ring_model(n, n)
    om = oracle_model(oracle, model)
    steps, seed = 4, 29
    betas, gammas = P * np.geomspace(0.01, 2.0, steps), np.linspace(2.0, 0.05, steps)
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


# both sides of the line: slices of a phase side by side (P = 1, odd and even P) and in
# qanneal's order (13 spins, or fewer with many rings)
@pytest.mark.parametrize("n,P,reads,order", [
    (32, 1, 2, "checkerboard"), (33, 1, 2, "reference"), (16, 5, 2, "checkerboard"), (17, 5, 2, "checkerboard"),
    (124, 16, 2, "checkerboard"), (125, 16, 2, "checkerboard"), (13, 6, 2, "reference"), (14, 6, 2, "reference"),
    (8, 20, 40, "reference"), (8, 20, 900, "reference")])
def test_small_models_match_oracle(oracle, n, P, reads, order):
    model = ring_model(n, n)
    om = oracle_model(oracle, model)
    steps, seed = 4, 31
    betas, gammas = P * np.geomspace(0.01, 2.0, steps), np.linspace(2.0, 0.05, steps)
    ann = qa.SQAAnnealer(model, qa.SQASchedule.from_vectors(betas, gammas), P)
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
