"""Fits and small queues of several threads at once, each call of another shape
(so that every thread makes and destroys loop graphs beside the
others), give the trees of the same calls one after another."""
import threading

import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier
from cudatree_b200.forest_queue import fit_forests

pytestmark = pytest.mark.gpu


def _call(k):
    rng = np.random.default_rng(k)
    n, f, c = 200 + 397 * k, 3 + k % 11, 2 + k % 5
    y = rng.integers(0, c, size=n)
    x = (rng.normal(size=(n, f)) + 0.4 * y[:, None]).astype(np.float32)
    if k % 4 == 3:
        return [t for g in fit_forests([(x, y), (x[: n // 2], y[: n // 2])], n_estimators=2, seeds=[k, k + 1])
                for t in g._trees]
    return RandomForestClassifier(n_estimators=3, seed=k).fit(x, y)._trees


def test_threads_with_graphs_of_their_own(cuda_device):
    calls = range(36)
    alone = [_call(k) for k in calls]
    got, errors = {}, []

    def caller(t):
        try:
            for k in [*range(t, len(calls), 3), *range((t + 1) % 3, len(calls), 3)]:
                got[t, k] = _call(k)
        except BaseException as e:  # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=caller, args=(t,)) for t in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and len(got) == 2 * len(calls)
    for (_, k), trees in got.items():
        assert len(trees) == len(alone[k])
        for a, b in zip(trees, alone[k]):
            np.testing.assert_array_equal(a.left_children, b.left_children)
            np.testing.assert_array_equal(a.feature_threshold_array, b.feature_threshold_array)
            np.testing.assert_array_equal(a.values_array, b.values_array)


def test_fit_waits_for_its_own_stream_only(cuda_device, monkeypatch):
    """A device-wide wait is forbidden while any stream captures: with one in fit,
    a thread that was making its loop graph was left with a broken one."""
    import torch

    def refuse(*a):
        raise AssertionError("device-wide wait")

    monkeypatch.setattr(torch.cuda, "synchronize", refuse)
    assert len(_call(2)) == 3 and len(_call(3)) == 4
