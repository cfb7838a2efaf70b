"""The update records of higher-order models: the same memory whatever the terms
share, and the same results where a target has many more records than the others
(chunks of one record), where targets run on from one round of records into the
next, and where a spin has none."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from test_gpu_parity_sa_sqa import oracle_model

pytestmark = pytest.mark.gpu


def shared_pair(n, terms, seed=1):
    """Four-body terms that all hold spins 0 and 1."""
    rng = np.random.default_rng(seed)
    out = {}
    while len(out) < terms:
        a, b = sorted((2 + rng.choice(n - 2, 2, replace=False)).tolist())
        out[(0, 1, a, b)] = float(rng.normal())
    return qa.HigherOrderIsing(out, n)


def uneven(n, seed=2):
    """Spins without a term, with one, and with several of 2 to 4 spins."""
    rng = np.random.default_rng(seed)
    out = {(0, 1): 0.5}
    for d, k in ((2, 2 * n), (3, n), (4, n)):
        for _ in range(k):
            out[tuple(sorted((2 + rng.choice(n // 2, size=d, replace=False)).tolist()))] = float(rng.normal())
    return qa.HigherOrderIsing(out, n)


def test_memory_of_terms_that_share_a_pair():
    """600000 records of 16 bytes; a round of records a pair member padded to 32 took 107 MB."""
    import torch
    model = shared_pair(1000, 50000)
    ann = qa.SQAAnnealer(model, qa.SQASchedule.from_vectors([1.0], [1.0]), 2)
    free = torch.cuda.mem_get_info()[0]
    ann.run_reads(1, 0, reads=1, seed=1)
    assert free - torch.cuda.mem_get_info()[0] < 48 << 20


@pytest.mark.parametrize("generic", [False, True])
@pytest.mark.parametrize("make,args", [(shared_pair, (40, 300)), (shared_pair, (130, 90)), (uneven, (90,)), (uneven, (40,))])
def test_sqa_matches_oracle(monkeypatch, oracle, make, args, generic):
    if generic:
        monkeypatch.setenv("QA_DISABLE_HUBO", "1")
    m = make(*args)
    om = oracle_model(oracle, m)
    P, steps, seed = 5, 5, 31
    betas, gammas = P * np.geomspace(0.02, 1.5, steps), np.linspace(2.0, 0.05, steps)
    ann = qa.SQAAnnealer(m, qa.SQASchedule.from_vectors(betas, gammas), P)
    res = ann.run_reads(2, 1, reads=2, seed=seed)
    oracle.set_update_order("reference")
    for r in range(2):
        best, _, trace, _ = oracle.sqa_run(om, betas, gammas, P, 1, 2, 1, seed, r)
        np.testing.assert_array_equal(res[r].best_state.as_array(), best)
        np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
