"""Two callers of the forest queue at once, each with its own seeds, get the
forests of solo fits."""
import threading

import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier
from cudatree_b200.forest_queue import fit_forests

from .test_gpu_queue import _blobs, _same

pytestmark = pytest.mark.gpu


def test_two_callers_at_once(cuda_device):
    jobs = [_blobs(300 + 401 * k, 6 + k, 2 + k, 80 + k) for k in range(5)]
    got, errors = {}, []

    def caller(c):
        try:
            for r in range(3):
                got[c, r] = fit_forests(jobs, n_estimators=3, seeds=range(100 * c + 10 * r, 100 * c + 10 * r + 5))
        except BaseException as e:  # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=caller, args=(c,)) for c in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for (c, r), forests in got.items():
        for k, ((x, y), f) in enumerate(zip(jobs, forests)):
            _same(f, RandomForestClassifier(n_estimators=3, seed=100 * c + 10 * r + k).fit(x, y))
    assert len(got) == 6 and np.all([len(f) == 5 for f in got.values()])
