"""The two forms of the forest walk: few walks in flight for one round of trees
and for small groups, more for groups that are far beyond L1 (CPU: the
library's rule), and the same votes from both at the rule's edge (GPU)."""
import ctypes as C

import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier, _lib
from oracle import cudatree_oracle as O


def _few(group, tree_bytes, rows_per_tile=32):
    fn = getattr(_lib.load(), "_ZN2ct21predict_few_in_flightEjjm")
    fn.restype, fn.argtypes = C.c_bool, [C.c_uint32, C.c_uint32, C.c_uint64]
    return fn(rows_per_tile, group, tree_bytes)


@pytest.mark.parametrize("group,tree_bytes,few", [
    (32, 75_000, True), (32, 600, True),                       # one round
    (100, 1_200, True), (100, 5_600, True), (300, 1_900, True), (1000, 200, True),
    (300, 4_000, False), (1000, 1_200, False), (1000, 5_600, False), (5000, 200, False),
    (33, 75_000, False), (100, 8_400, False)])                 # rounds of trees beyond L1
def test_form(group, tree_bytes, few):
    assert _few(group, tree_bytes) == few


@pytest.mark.gpu
@pytest.mark.parametrize("n,trees", [(60, 1000), (220, 500), (220, 1400)])
def test_many_small_trees_match_oracle(cuda_device, n, trees):
    rng = np.random.default_rng(n)
    x, y = rng.normal(size=(n, 5)).astype(np.float32), rng.integers(0, 3, size=n)
    kw = dict(n_estimators=trees, seed=n, max_features=2)
    forest, ref = RandomForestClassifier(**kw).fit(x, y), O.fit_forest(x, y, **kw)
    q = rng.normal(size=(2500, 5)).astype(np.float32)
    for rows in (3, 1023, 2500):
        np.testing.assert_array_equal(forest.predict_proba(q[:rows]), O.predict_proba(ref, q[:rows]))
