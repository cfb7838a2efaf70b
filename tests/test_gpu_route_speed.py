"""A call that a special kernel takes is not slower than the general path it took
before (the switch in the second column brings that back).  Where the rules of
the dispatch put the line wrong the special path took 1.3 to 6 times as long;
the bound is 1.25 on the fastest of six runs of each side, taken in turn.
"""
import numpy as np
import pytest

import qlatanneal_b200 as qa
from qlatanneal_b200.instances import dense_real, regular3

pytestmark = pytest.mark.gpu


def sa_real(n, reads):
    """Chains in flight, not the time of one chain, bound many reads."""
    betas = np.geomspace(0.3, 3.0, 20) * 1.7 / np.sqrt(n)
    ann = qa.Annealer(qa.DenseIsing(*dense_real(n, 1)), qa.AnnealSchedule.from_betas(betas))
    return ann, lambda: ann.run_reads(5, reads=reads, seed=1)


def sparse_checkerboard(n, P, reads):
    """Few spins, many slices, slices side by side."""
    qa.set_update_order("checkerboard")
    ann = qa.SQAAnnealer(qa.SparseIsing(*regular3(n, 1), n),
                         qa.SQASchedule.from_vectors(P * np.linspace(0.1, 2.0, 10), np.linspace(2.0, 0.05, 10)), P)
    return ann, lambda: ann.run_reads(5, 1, reads=reads, seed=1)


def sparse_small(n, P, reads, order):
    """A sweep a step: the energies of a step count as well."""
    qa.set_update_order(order)
    ann = qa.SQAAnnealer(qa.SparseIsing(*regular3(n, 1), n),
                         qa.SQASchedule.from_vectors(P * np.linspace(0.1, 2.5, 40), np.linspace(2.0, 0.05, 40)), P)
    return ann, lambda: ann.run_reads(1, 0, reads=reads, seed=1)


def dense_checkerboard(n, P, reads):
    """Many rings: the slices of a phase at work on all SMs, not the chain of one."""
    qa.set_update_order("checkerboard")
    ann = qa.SQAAnnealer(qa.DenseIsing(*dense_real(n, 1)), qa.SQASchedule.from_vectors(
        P * np.linspace(0.1, 3.0, 6) / np.sqrt(n), np.linspace(2.0, 0.05, 6)), P)
    return ann, lambda: ann.run_reads(3, 0, reads=reads, seed=1)


def hubo_rings(n, P, reads, order):
    """Pair terms on a ring: little to do at a flip, many rings."""
    qa.set_update_order(order)
    terms = {tuple(sorted((i, (i + 1) % n))): 1.0 - 2.0 * (i % 3 == 0) for i in range(n)}
    ann = qa.SQAAnnealer(qa.HigherOrderIsing(terms, n), qa.SQASchedule.from_vectors(
        P * np.linspace(0.1, 2.0, 6), np.linspace(2.0, 0.05, 6)), P)
    return ann, lambda: ann.run_reads(2, 0, reads=reads, seed=1)


SHAPES = [
    (sa_real, "QA_DISABLE_DENSE", (24, 4000)),
    (sa_real, "QA_DISABLE_DENSE", (64, 2000)),
    (sa_real, "QA_DISABLE_DENSE", (256, 4000)),
    (sparse_checkerboard, "QA_DISABLE_SLAB", (40, 32, 1)),
    (sparse_checkerboard, "QA_DISABLE_SLAB", (40, 64, 200)),
    (sparse_checkerboard, "QA_DISABLE_SLAB", (128, 64, 32)),
    (sparse_checkerboard, "QA_DISABLE_SLAB", (512, 32, 32)),
    (sparse_checkerboard, "QA_DISABLE_SLAB", (128, 16, 600)),
    (sparse_small, "QA_DISABLE_SLAB", (104, 16, 44, "checkerboard")),
    (sparse_small, "QA_DISABLE_SLAB", (20, 8, 700, "checkerboard")),
    (sparse_small, "QA_DISABLE_SLAB", (14, 1, 1, "checkerboard")),
    (sparse_small, "QA_DISABLE_SLAB", (8, 20, 14, "reference")),
    (sparse_small, "QA_DISABLE_SLAB", (10, 16, 2, "reference")),
    (dense_checkerboard, "QA_DISABLE_DENSE", (12, 8, 3000)),
    (dense_checkerboard, "QA_DISABLE_DENSE", (24, 12, 600)),
    (dense_checkerboard, "QA_DISABLE_DENSE", (64, 5, 1000)),
    (dense_checkerboard, "QA_DISABLE_DENSE", (200, 8, 600)),
    (hubo_rings, "QA_DISABLE_HUBO", (200, 16, 600, "checkerboard")),
    (hubo_rings, "QA_DISABLE_HUBO", (64, 8, 1000, "checkerboard")),
    (hubo_rings, "QA_DISABLE_HUBO", (200, 4, 600, "reference")),
]


@pytest.mark.parametrize("make,switch,shape", SHAPES, ids=lambda v: getattr(v, "__name__", None))
def test_not_slower_than_the_general_path(monkeypatch, make, switch, shape):
    ann, call = make(*shape)
    special, general = [], []
    try:
        for _ in range(7):
            call()
            special.append(ann.last_stats.sweep_ms)
            monkeypatch.setenv(switch, "1")
            call()
            general.append(ann.last_stats.sweep_ms)
            monkeypatch.delenv(switch)
    finally:
        qa.set_update_order("reference")
    assert min(special[1:]) <= 1.25 * min(general[1:])
