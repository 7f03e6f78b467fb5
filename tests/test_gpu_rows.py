"""Row-list growth (one row list per tree, sorted orders made on demand)
against the oracle, at the edges of its node-size classes: the warp subtrees
(32 rows), one warp (512), the two CTA sizes (2,048 and 9,216), bitmaps of one
and of several slices (32,768 rows), and every kind of feature column."""
import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier
from oracle import cudatree_oracle as O

from .test_gpu_fit import _assert_same_trees

pytestmark = pytest.mark.gpu


def _columns(n, c, seed, onehot=5):
    """Continuous, tied, few-valued, one-hot, constant and wide-ranged
    columns (infinities and negative zeros among them), labels that depend on
    some of them."""
    rng = np.random.default_rng(seed)
    y = rng.integers(0, c, size=n)
    x = rng.normal(size=(n, 8 + onehot)).astype(np.float32)
    x[:, 0] += 0.3 * y
    x[:, 1] = np.round(x[:, 1] + 0.1 * y, 1)
    x[:, 2] = rng.integers(0, 3, size=n) + (y == 0)
    x[:, 3] = 2.5
    x[:, 4] = np.where(np.abs(x[:, 4]) < 0.2, -0.0, x[:, 4] * 1e6)
    x[:: 97, 4] = np.inf
    x[1:: 101, 4] = -np.inf
    x[:, 5] *= 1e-5  # neighbours closer than the candidate gap
    x[:, 8:] = 0.0
    x[np.arange(n), 8 + rng.integers(0, onehot, size=n)] = 1.0
    return x, y


@pytest.mark.parametrize("n,c", [(2, 2), (32, 3), (33, 3), (511, 7), (512, 8), (513, 9), (2047, 2), (2048, 8),
                                 (2049, 30), (4097, 1), (9216, 7), (9217, 7), (9217, 12), (32768, 3), (33000, 8),
                                 (66001, 2), (66001, 70)])
def test_node_size_edges_match_oracle(cuda_device, n, c):
    """Without bootstrap the root holds exactly n rows, in every kind of column."""
    x, y = _columns(n, c, n + c)
    kw = dict(n_estimators=2 if n < 30000 else 1, bootstrap=False, seed=n, max_features=6)
    forest = RandomForestClassifier(**kw).fit(x, y)
    _assert_same_trees(forest._trees, O.fit_forest(x, y, **kw).trees)


@pytest.mark.parametrize("kw", [dict(min_samples_split=40), dict(subtree_cutoff=0), dict(subtree_cutoff=7),
                                dict(max_features=20), dict(max_features=1)])
@pytest.mark.parametrize("virtual", [True, False])
def test_options_match_oracle(cuda_device, kw, virtual):
    """Options, with and without virtual two-valued features (12 one-hot columns)."""
    x, y = _columns(12000, 5, 3, onehot=12)
    forest = RandomForestClassifier(n_estimators=2, seed=4, **kw)
    forest.virtual_features = virtual
    forest.fit(x, y)
    ref = O.fit_forest(x, y, n_estimators=2, seed=4,
                       **{k: v for k, v in kw.items() if k != "subtree_cutoff"})
    _assert_same_trees(forest._trees, ref.trees)


@pytest.mark.parametrize("n,few", [(300000, 12000), (590000, 9219), (700000, 9800)])
@pytest.mark.parametrize("c", [2, 6, 8, 9])
def test_crowded_runs_of_ranks_match_oracle(cuda_device, n, few, c):
    """The first split leaves a node of `few` rows that are neighbours in two
    columns: one run of ranks holds them all (the first size), or the node is
    too sparse for a bitmap (the others; at the last, 8 and 9 classes take
    list growth).  Its descendants pass every size class with the sorts that
    many ranks take."""
    rng = np.random.default_rng(n + c)
    u = rng.permutation(n).astype(np.float32)
    x = np.stack([u, u + rng.normal(size=n).astype(np.float32), rng.normal(size=n).astype(np.float32)]
                 + [np.ones(n, np.float32)] * 5, axis=1)
    y = np.where(u < few, (x[:, 2] * 3 + rng.integers(0, 2, size=n) + (u > few / 3)).astype(np.int64) % c, 0)
    kw = dict(n_estimators=1, bootstrap=False, seed=c, max_features=3)
    forest = RandomForestClassifier(**kw).fit(x, y)
    _assert_same_trees(forest._trees, O.fit_forest(x, y, **kw).trees)


def test_identical_rows_become_impure_leaves(cuda_device):
    """A large node that cannot split: its leaf takes the class of its first
    row in feature 0's order."""
    rng = np.random.default_rng(5)
    x = np.repeat(rng.normal(size=(6, 4)).astype(np.float32), 3000, axis=0)
    y = rng.integers(0, 4, size=x.shape[0])
    kw = dict(n_estimators=3, seed=9, max_features=2)
    forest = RandomForestClassifier(**kw).fit(x, y)
    _assert_same_trees(forest._trees, O.fit_forest(x, y, **kw).trees)


def test_misaligned_lists_take_list_growth(cuda_device):
    """List buffers that are not 16-byte aligned cannot hold the row lists and
    sorted planes: the fit keeps every feature's list and grows the same trees."""
    import ctypes as C

    import torch

    from cudatree_b200 import _lib
    from cudatree_b200.random_forest import fetch_tree_columns
    from . import gpu_utils as G
    x, y = _columns(20000, 4, 8)
    gp = G.GpuProblem(x, y, 4, 4, bootstrap=True, seed=3)
    gl = G.GpuLists(gp, 2)
    raw = [torch.zeros(2 * 2 * gp.n, dtype=torch.int32, device=G.dev()) for _ in range(5)]
    nn = torch.zeros(2, dtype=torch.int32, device=G.dev())
    tb = _lib.TreeBuffers(*[r.data_ptr() for r in raw], nn.data_ptr(), 2 * gp.n)
    opts = _lib.FitOptions(_lib.CT_FIT_BATCHED, 0, 32, 0)
    ws = C.c_size_t()
    _lib.call("ct_fit_workspace_size", C.byref(gp.prob), 2, C.byref(opts), C.byref(ws))
    work = G.dev_bytes(ws.value)
    out = []
    for misalign in (0, 2):
        gl.lists.si0 = gl.si[0].data_ptr() + misalign
        _lib.call("ct_fit", C.byref(gp.prob), C.byref(gl.lists), 0, 2, C.byref(opts), C.byref(tb), work.data_ptr(),
                  ws.value, G.stream())
        out.append(fetch_tree_columns(tb, nn, 2, G.dev()))
    for a, b in zip([out[0][0], *out[0][1]], [out[1][0], *out[1][1]]):
        np.testing.assert_array_equal(a, b)
