"""Classical parallel tempering of +-1 models in one launch (pt_chains_kernel)."""
import numpy as np
import pytest

import qlatanneal_b200 as qa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,reads,spb,steps,swap", [(1, 2, 1, 1, 3, 1), (31, 3, 5, 2, 7, 2), (33, 32, 2, 1, 5, 1),
                                                      (129, 5, 40, 3, 9, 10), (400, 8, 3, 1, 4, 3), (64, 33, 2, 1, 4, 1)])
def test_parallel_tempering_one_launch(monkeypatch, n, R, reads, spb, steps, swap):
    """pt_chains_kernel (+-1 models, up to 32 rungs, the whole run in one launch)
    equals a launch per swap interval (QA_DISABLE_PT_CHAINS; always with 33)."""
    rng = np.random.default_rng(n)
    J = np.triu(rng.choice([-1.0, 1.0], (n, n)), 1)
    model = qa.DenseIsing(rng.normal(0, 0.3, n), J + J.T, 0.5)
    ann = qa.ParallelTemperingAnnealer(model, np.geomspace(1e-3, 3.0, R))  # hot chains accept nearly every move

    def call():
        res = ann.run_reads(spb, steps, swap, reads=reads, seed=11)
        st = ann.last_stats
        return [x for r in res for x in (r.best_state.as_array(), r.best_energy, np.array(r.final_energies),
                                         np.stack([s.as_array() for s in r.final_states]),
                                         np.array(r.average_energy_trace), np.array(r.swap_acceptance_trace))] + [
            np.array([st.slice_attempts, st.slice_accepts])]

    a = call()
    monkeypatch.setenv("QA_DISABLE_PT_CHAINS", "1")
    for x, y in zip(a, call()):
        np.testing.assert_array_equal(x, y)
