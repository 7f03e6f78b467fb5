"""Sorted planes of row-list growth that lie in the fit's workspace: lists with
more slots or a longer stride than the fit's trees and rows, and a last batch
of fewer trees than the lists hold, grow the oracle's trees and write nothing
behind the workspace."""
import ctypes as C

import numpy as np
import pytest
import torch

from cudatree_b200 import RandomForestClassifier, _lib
from cudatree_b200.random_forest import fetch_tree_columns
from oracle import cudatree_oracle as O

from . import gpu_utils as G
from .test_gpu_fit import _assert_same_trees

pytestmark = pytest.mark.gpu
GUARD = 1 << 20  # bytes behind the workspace and the lists that must stay as they were


def _data(n, f, c, seed):
    rng = np.random.default_rng(seed)
    y = rng.integers(0, c, size=n)
    x = (rng.normal(size=(n, f)) + 0.4 * y[:, None]).astype(np.float32)
    x[:, 1] = np.round(x[:, 1], 1)
    return x, y


def _assert_columns(counts, cols, ref):
    assert counts.tolist() == [t.n_nodes for t in ref]
    names = ("left", "right", "feature", "threshold", "value")
    for col, name in zip(cols, names):
        np.testing.assert_array_equal(col, np.concatenate([getattr(t, name) for t in ref]), err_msg=name)


# features, selected: no plane fits behind the row lists (5, 6 of 16 bits), one (9) or two (13) per
# buffer do; the others lie in the workspace
@pytest.mark.parametrize("f,m", [(5, 3), (6, 6), (9, 3), (9, 9), (13, 4), (13, 12)])
@pytest.mark.parametrize("extra_slots,extra_stride", [(0, 0), (35, 0), (0, 4099), (3, 513)])
def test_lists_larger_than_the_fit(cuda_device, f, m, extra_slots, extra_stride):
    n, trees = 20000, 2
    x, y = _data(n, f, 3, f)
    gp = G.GpuProblem(x, y, 3, m, bootstrap=True, seed=7)
    slots, stride = trees + extra_slots, n + extra_stride
    size = slots * f * stride * gp.ib
    si = [torch.full((size + GUARD,), 0x5A, dtype=torch.uint8, device=G.dev()) for _ in range(2)]
    mark = G.dev_bytes(_lib.mark_bytes(stride, slots))
    lists = _lib.Lists(si[0].data_ptr(), si[1].data_ptr(), mark.data_ptr(), stride, slots)
    raw = [torch.zeros(trees * 2 * n, dtype=torch.int32, device=G.dev()) for _ in range(5)]
    nn = torch.zeros(trees, dtype=torch.int32, device=G.dev())
    tb = _lib.TreeBuffers(*[r.data_ptr() for r in raw], nn.data_ptr(), 2 * n)
    opts = _lib.FitOptions(_lib.CT_FIT_BATCHED, 0, 32, 0)
    ws = C.c_size_t()
    _lib.call("ct_fit_workspace_size", C.byref(gp.prob), trees, C.byref(opts), C.byref(ws))
    work = torch.full((ws.value + GUARD,), 0x5A, dtype=torch.uint8, device=G.dev())
    _lib.call("ct_fit", C.byref(gp.prob), C.byref(lists), 0, trees, C.byref(opts), C.byref(tb), work.data_ptr(),
              ws.value, G.stream())
    counts, cols = fetch_tree_columns(tb, nn, trees, G.dev())
    for buf, used in ((work, ws.value), (si[0], size), (si[1], size)):
        assert bool((buf[used:] == 0x5A).all())
    _assert_columns(counts, cols, O.fit_forest(x, y, n_estimators=trees, max_features=m, seed=7).trees)


def test_last_batch_of_fewer_trees(cuda_device):
    """3 trees grown 2 at a time: the second call has lists of two slots for one tree."""
    x, y = _data(12000, 8, 4, 2)
    forest = RandomForestClassifier(n_estimators=3, max_features=3, seed=11)
    forest.fit_init(x, y)
    trees = forest._fit_trees_k(0, 3, "batched", forest.bfs_threshold, 2)
    forest.fit_release()
    _assert_same_trees(trees, O.fit_forest(x, y, n_estimators=3, max_features=3, seed=11).trees)
