"""Votes of forests of many small trees, with one tree group and several and in
both forms of the walk, against the oracle's walk."""
import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier
from oracle import cudatree_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("n,trees", [(60, 1000), (220, 500), (220, 1400)])
def test_many_small_trees_match_oracle(cuda_device, n, trees):
    rng = np.random.default_rng(n)
    x, y = rng.normal(size=(n, 5)).astype(np.float32), rng.integers(0, 3, size=n)
    kw = dict(n_estimators=trees, seed=n, max_features=2)
    forest, ref = RandomForestClassifier(**kw).fit(x, y), O.fit_forest(x, y, **kw)
    q = rng.normal(size=(2500, 5)).astype(np.float32)
    for rows in (3, 200, 1023, 1024, 2500):
        np.testing.assert_array_equal(forest.predict_proba(q[:rows]), O.predict_proba(ref, q[:rows]))
