"""Infinite fields, couplings near the end of float32 and beta = 0 on the dense
and sparse kernels, against the CPU restatement: a field that overflows and a
product that is not a number decide as they do there."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from qlatanneal_b200.instances import dense_real, regular3, sk_dense
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


def pairs(n, seed=3):
    """Spins coupled in pairs by +-2e38: a field is one coupling, finite, while 2 J is
    not.  Rounding the product first makes the partner's field infinite after a flip;
    one fused multiply-add would give its finite negative."""
    rng = np.random.default_rng(seed)
    J = np.zeros((n, n))
    for i in range(0, n - 1, 2):
        J[i, i + 1] = J[i + 1, i] = rng.choice([-2e38, 2e38])
    return qa.DenseIsing(np.zeros(n), J)


@pytest.mark.parametrize("n", [40, 300])
def test_sa_couplings_whose_double_overflows(oracle, n):
    model = pairs(n)
    om = oracle_model(oracle, model)
    betas, spb, seed = np.array([1e-39, 2e-39, 5e-39, 1e-38]), 2, 7
    ann = qa.Annealer(model, qa.AnnealSchedule.from_betas(betas))
    for reads in (3, 1000):
        res = ann.run_reads(spb, reads=reads, seed=seed)
        acc = 0
        for r in range(3):
            best, _, trace, cnt = oracle.sa_run(om, betas, spb, seed, r)
            acc += cnt[1]
            np.testing.assert_array_equal(res[r].best_state.as_array(), best)
            np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
        if reads == 3:
            assert 0 < acc == ann.last_stats.slice_accepts


@pytest.mark.parametrize("order", ["reference", "checkerboard"])
@pytest.mark.parametrize("n,P", [(40, 4), (300, 3)])
def test_sqa_couplings_whose_double_overflows(oracle, order, n, P):
    model = pairs(n)
    om = oracle_model(oracle, model)
    betas, gammas, seed = P * np.array([1e-39, 2e-39, 5e-39]), np.array([1e39, 1e38, 1e38]), 7
    ann = qa.SQAAnnealer(model, qa.SQASchedule.from_vectors(betas, gammas), P)
    try:
        qa.set_update_order(order)
        oracle.set_update_order(order)
        res = ann.run_reads(2, 1, reads=2, seed=seed)
        acc = np.zeros(4, np.int64)
        for r in range(2):
            _, _, trace, cnt = oracle.sqa_run(om, betas, gammas, P, 1, 2, 1, seed, r)
            acc += np.asarray(cnt[:4], np.int64)
            np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
        st = ann.last_stats
        assert acc[1] > 0
        assert [st.slice_attempts, st.slice_accepts, st.worldline_attempts, st.worldline_accepts] == acc.tolist()
    finally:
        qa.set_update_order("reference")
        oracle.set_update_order("reference")


def with_infinite_h(kind, n):
    rng = np.random.default_rng(n)
    if kind == "sparse":
        h, edges = regular3(n, n)
        h[rng.permutation(n)[:3]] = [np.inf, -np.inf, np.inf]
        return qa.SparseIsing(h, edges, n)
    h, J = sk_dense(n, n) if kind == "pm1" else dense_real(n, n)
    h[rng.permutation(n)[:3]] = [np.inf, -np.inf, np.inf]
    return qa.DenseIsing(h, J)


@pytest.mark.parametrize("order", ["reference", "checkerboard"])
@pytest.mark.parametrize("kind,n,P", [("real", 40, 5), ("real", 300, 3), ("pm1", 70, 4), ("sparse", 130, 3), ("sparse", 300, 40)])
def test_sqa_infinite_fields(oracle, order, kind, n, P):
    """beta = 0 times an infinite field is not a number: the move is rejected."""
    model = with_infinite_h(kind, n)
    om = oracle_model(oracle, model)
    betas, gammas, seed = P * np.array([0.0, 0.02, 1.0]), np.array([2.0, 1.0, 0.1]), 7
    ann = qa.SQAAnnealer(model, qa.SQASchedule.from_vectors(betas, gammas), P)
    try:
        qa.set_update_order(order)
        oracle.set_update_order(order)
        res = ann.run_reads(2, 1, reads=2, seed=seed)
        acc = np.zeros(4, np.int64)
        for r in range(2):
            _, _, trace, cnt = oracle.sqa_run(om, betas, gammas, P, 1, 2, 1, seed, r)
            acc += np.asarray(cnt[:4], np.int64)
            np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
        st = ann.last_stats
        assert acc[1] > 0
        assert [st.slice_attempts, st.slice_accepts, st.worldline_attempts, st.worldline_accepts] == acc.tolist()
    finally:
        qa.set_update_order("reference")
        oracle.set_update_order("reference")


@pytest.mark.parametrize("kind,n,reads", [("pm1", 70, 3), ("real", 40, 3), ("real", 300, 3), ("real", 40, 1500)])
def test_sa_infinite_h(oracle, kind, n, reads):
    model = with_infinite_h(kind, n)
    om = oracle_model(oracle, model)
    betas, spb, seed = np.array([0.0, 0.02, 1.0]), 2, 7
    ann = qa.Annealer(model, qa.AnnealSchedule.from_betas(betas))
    res = ann.run_reads(spb, reads=reads, seed=seed)
    acc = 0
    for r in range(reads):
        _, _, trace, cnt = oracle.sa_run(om, betas, spb, seed, r)
        acc += cnt[1]
        np.testing.assert_array_equal(np.asarray(res[r].energy_trace), trace)
    assert 0 < acc == ann.last_stats.slice_accepts


def test_pt_chains_infinite_h(monkeypatch):
    model = with_infinite_h("pm1", 70)
    ann = qa.ParallelTemperingAnnealer(model, np.geomspace(1e-3, 2.0, 5))
    out = []
    for _ in range(2):
        res = ann.run_reads(2, 6, 2, reads=3, seed=11)
        out.append([x for r in res for x in (np.array(r.final_energies), np.array(r.average_energy_trace),
                                             np.array(r.swap_acceptance_trace))] + [np.array(ann.last_stats.slice_accepts)])
        monkeypatch.setenv("QA_DISABLE_PT_CHAINS", "1")
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
