"""Algorithmic bytes of row-list growth's kernel groups, against the sizes of the
nodes of the trees it grew: orders of the selected features and moved rows of
large splits count as partition, marks and moved rows of small splits as mark."""
import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier, _lib

pytestmark = pytest.mark.gpu


def _node_sizes(tree, x):
    """Rows that reach each node of a tree grown without bootstrap."""
    n = np.zeros(tree.n_nodes, np.int64)
    at = np.zeros(x.shape[0], np.int64)
    alive = np.arange(x.shape[0])
    while alive.size:
        n += np.bincount(at[alive], minlength=tree.n_nodes)
        alive = alive[tree.left_children[at[alive]] != 0]
        k = at[alive]
        left = x[alive, tree.feature_idx_array[k]] <= tree.feature_threshold_array[k]
        at[alive] = np.where(left, tree.left_children[k], tree.right_children[k])
    return n


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("n,per_row", [(30000, 8), (700000, 20)])
def test_bytes_follow_the_node_sizes(cuda_device, n, per_row, host):
    """30,000 rows: every order is a bitmap (8 bytes per row).  700,000: the nodes
    of 9,217 to 10,900 rows are too sparse for one (20 bytes per row)."""
    m, few = 3, 10000
    rng = np.random.default_rng(n)
    if per_row == 8:
        x = rng.normal(size=(n, 5)).astype(np.float32)
        y = rng.integers(0, 3, size=n)
    else:
        # one split leaves `few` rows, whose first split is a large node's too
        u = rng.permutation(n).astype(np.float32)
        x = np.stack([u, u + rng.normal(size=n).astype(np.float32), rng.normal(size=n).astype(np.float32)], axis=1)
        y = np.where(u < few, rng.integers(0, 3, size=n), 0)
    f = RandomForestClassifier(1, max_features=m, bootstrap=False, seed=3)
    f.host_level_loop = host
    f.fit(x, y)
    tree = f._trees[0]
    size = _node_sizes(tree, x)
    inner = tree.left_children != 0
    steps = size[inner & (size > 32)]  # (smaller nodes are warp subtrees)
    ordered = size[(size > 9216) & inner]
    sparse = 8 * ordered < -(-n // 128) * 16 + 16
    assert ordered.size > 1 and sparse.any() == (per_row == 20)
    got = dict(zip(_lib.KERNEL_GROUPS, f.last_fit_stats["bytes"]))
    assert got["partition"] == m * (ordered * np.where(sparse, 20, 8)).sum() + 8 * steps[steps > 512].sum()
    assert got["mark"] == 8 * steps.sum() + 4 * steps[steps <= 512].sum()
