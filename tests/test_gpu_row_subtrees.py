"""Several launches of row-list growth's warp subtrees in one fit."""
import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier, _lib
from oracle import cudatree_oracle as O

from .test_gpu_fit import _assert_same_trees

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["host", "host_then_graph"])
def test_every_launch_grows_all_of_its_subtrees(cuda_device, how):
    """Steps of 4,000 nodes fill the subtree list (two steps' worth) many times
    over.  A launch of more subtrees than the chip holds warps (3,552) claims
    the others from a counter, which has to start anew for each launch."""
    rng = np.random.default_rng(3)
    n, trees = 60000, 8
    x = rng.normal(size=(n, 3)).astype(np.float32)
    y = rng.integers(0, 2, size=n)
    kw = dict(n_estimators=trees, max_features=1, bootstrap=False, seed=5)
    one_launch = RandomForestClassifier(**kw).fit(x, y)  # every level in the graph, one list of subtrees
    forest = RandomForestClassifier(**kw)
    forest.step_nodes = 4000
    if how == "host":
        forest.host_level_loop = True
    else:
        forest.graph_samples = 8 * n // 3  # the wide levels run from the host
    forest.fit(x, y)
    if how == "host":
        assert forest.last_fit_stats["launches"][_lib.KERNEL_GROUPS.index("subtree")] > 3
    for a, b in zip(forest._trees, one_launch._trees):
        np.testing.assert_array_equal(a.left_children, b.left_children)
        np.testing.assert_array_equal(a.feature_idx_array, b.feature_idx_array)
        np.testing.assert_array_equal(a.feature_threshold_array, b.feature_threshold_array)
        np.testing.assert_array_equal(a.values_array, b.values_array)
    _assert_same_trees(forest._trees[:2], O.fit_forest(x, y, **{**kw, "n_estimators": 2}).trees)
