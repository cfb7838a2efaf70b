"""Dense SA with more reads than the multi-warp form holds at once: one warp a
read, and sa_kernel for small models with real couplings.  A read's result does
not depend on it."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from qlatanneal_b200.instances import dense_real, sk_dense
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu


# either side of n = 18, of n = 96, of the 128 uniforms a warp draws and of 512 columns of a row; more
# reads than one warp a read holds (32 an SM at most) and fewer
@pytest.mark.parametrize("kind,n,reads", [("pm1", 20, 5000), ("pm1", 129, 2500), ("real", 40, 1200), ("real", 40, 2600),
                                          ("real", 95, 2000), ("real", 96, 2000), ("real", 300, 900),
                                          ("real", 514, 600), ("pm1", 1310, 700), ("real", 17, 800),
                                          ("real", 18, 800)])
def test_many_reads_match_oracle(oracle, kind, n, reads):
    model = qa.DenseIsing(*(sk_dense(n, n, h_sigma=0.2) if kind == "pm1" else dense_real(n, n)))
    om = oracle_model(oracle, model)
    betas = np.concatenate([[0.0], np.geomspace(1e-3, 3.0, 4) / np.sqrt(n)])
    ann = qa.Annealer(model, qa.AnnealSchedule.from_betas(betas))
    res = ann.run_reads(2, reads=reads, seed=23)
    few = ann.run_reads(2, reads=64, seed=23)
    for r in (0, reads // 2, reads - 1):
        best, _, trace, _ = oracle.sa_run(om, betas, 2, 23, r)
        np.testing.assert_array_equal(res[r].best_state.as_array(), best)
        np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
    for a, b in zip(res, few):
        np.testing.assert_array_equal(a.best_state.as_array(), b.best_state.as_array())
        assert a.best_energy == b.best_energy and a.energy_trace == b.energy_trace
