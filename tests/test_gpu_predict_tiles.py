"""Row tiles and tree groups of the forest walk: tiles of a few rows, and
forests of less than, just over and several times the trees that a block walks
at once, with one group (direct vote) and several (vote table), against the
oracle's walk; the server's batch walk gives the same."""
import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier
from cudatree_b200.serving import ForestServer
from oracle import cudatree_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trees,f,c", [(3, 9, 5), (33, 9, 5), (49, 9, 5), (129, 9, 5), (40, 700, 60)])
def test_row_tiles_and_tree_groups_match_oracle(cuda_device, trees, f, c):
    rng = np.random.default_rng(trees)
    x = rng.normal(size=(1200, f)).astype(np.float32)
    y = rng.integers(0, c, size=1200)  # noise: deep trees
    kw = dict(n_estimators=trees, seed=trees, max_features=3)
    forest, ref = RandomForestClassifier(**kw).fit(x, y), O.fit_forest(x, y, **kw)
    q = rng.normal(size=(3001, f)).astype(np.float32)
    pred, proba = O.predict(ref, q), O.predict_proba(ref, q)
    srv = ForestServer(max_features=1024)
    try:
        fid = srv.add_forest(forest)
        for rows in (1, 2, 5, 31, 33, 200, 1023, 1024, 3001):
            np.testing.assert_array_equal(forest.predict(q[:rows]), pred[:rows])
            np.testing.assert_array_equal(forest.predict_proba(q[:rows]), proba[:rows])
            np.testing.assert_array_equal(srv.predict(fid, q[:rows]), pred[:rows])
    finally:
        srv.close()
