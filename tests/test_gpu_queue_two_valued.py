"""Queues of jobs with two-valued, few-valued and constant columns, by list
growth (lists off alignment) and by row lists, against the oracle: the pieces of
two-valued features have a scan of their own in list growth."""
import numpy as np
import pytest

from cudatree_b200 import _lib
from cudatree_b200.forest_queue import fit_forests
from oracle import cudatree_oracle as O

from .test_gpu_fit import _assert_same_trees

pytestmark = pytest.mark.gpu


def _job(n, f, c, seed):
    rng = np.random.default_rng(seed)
    y = rng.integers(0, c, size=n)
    x = rng.normal(size=(n, f)).astype(np.float32)
    x[:, 0] += 0.5 * y
    for k in range(1, f):
        if k % 3 == 1:
            x[:, k] = rng.random(n) < 0.2 + 0.5 * (y % 2)
        elif k % 6 == 2:
            x[:, k] = rng.integers(0, 3, size=n)
        elif k % 7 == 3:
            x[:, k] = 4.0
    return x, y


@pytest.mark.parametrize("shift", [0, 8])
@pytest.mark.parametrize("specs", [[(2, 2, 2), (30, 3, 2), (700, 9, 4)], [(1500, 30, 3), (3, 4, 2), (5000, 70, 8)],
                                   [(4000, 12, 9), (9000, 5, 2), (1, 3, 1)], [(66000, 8, 3), (80000, 5, 2)]])
def test_queue_matches_oracle(cuda_device, monkeypatch, shift, specs):
    lists = _lib.Lists
    monkeypatch.setattr(_lib, "Lists", lambda a, b, *rest: lists(a and a + shift, b and b + shift, *rest))
    jobs = [_job(*s, seed=17 * k + len(specs)) for k, s in enumerate(specs)]
    for options in (None, {"subtree_cutoff": 0, "scan_piece": 512}, {"subtree_cutoff": 128}):
        forests = fit_forests(jobs, n_estimators=2, seeds=range(len(jobs)), fit_options=options)
        for k, ((x, y), f) in enumerate(zip(jobs, forests)):
            _assert_same_trees(f._trees, O.fit_forest(x, y, n_estimators=2, seed=k).trees)
