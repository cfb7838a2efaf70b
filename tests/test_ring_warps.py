"""warps_per_ring: what each kernel makes of it, and no launch shape timed twice by
the autotuner."""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from qlatanneal_b200 import autotune
from qlatanneal_b200.instances import dense_real, hubo_random, regular3, sk_dense


def test_distinct_keeps_one_candidate_per_launch():
    cands = [dict(warps_per_ring=w) for w in (8, 16, 32)]
    assert autotune._distinct(cands, lambda c: min(8, c["warps_per_ring"]), {4}) == cands[:1]
    assert autotune._distinct(cands, lambda c: c["warps_per_ring"], {16}) == [cands[0], cands[2]]


@pytest.mark.gpu
@pytest.mark.parametrize("kind,model,most", [
    ("pm1", lambda: qa.DenseIsing(*sk_dense(64, 1)), 32), ("real", lambda: qa.DenseIsing(*dense_real(64, 1)), 16),
    ("hubo", lambda: qa.HigherOrderIsing(hubo_random(64, 1), 64), 16),
    ("sparse", lambda: qa.SparseIsing(*regular3(600, 1), 600), 8)])
def test_overrides_reach_the_kernel(kind, model, most):
    from qlatanneal_b200 import _lib
    eng, m = _lib.Engine.get(None), model()
    P, sched = 32, qa.SQASchedule.from_vectors(np.linspace(2.0, 30.0, 6), np.linspace(2.0, 0.05, 6))
    ann = qa.SQAAnnealer(m, sched, P)
    want = ann.run_reads(1, 1, reads=3, seed=4)
    try:
        for w in (1, 3, 5, 8, 16, 32):
            autotune.set_tuning(eng, dict(warps_per_ring=w))
            assert autotune._ring_warps(eng, m, P, 3, False, False) == min(w, most)
            for a, b in zip(want, ann.run_reads(1, 1, reads=3, seed=4)):
                np.testing.assert_array_equal(a.best_state.as_array(), b.best_state.as_array())
                assert a.energy_trace == b.energy_trace
        entry = autotune.tune_sqa(ann, 1, 1, reads=3, timing_steps=4)
        shapes = []
        for c in entry["candidates"]:
            if c["tuning"]["rotate"] == -1 and c["tuning"]["field_form"] == -1:
                autotune.set_tuning(eng, c["tuning"])
                shapes.append(autotune._ring_warps(eng, m, P, 3, False, False))
        # (the +-1 forms stage times the fastest warps once more with form -1)
        assert len(set(shapes)) >= len(shapes) - (1 if kind in ("pm1", "real") else 0)
    finally:
        autotune.set_tuning(eng, None)
