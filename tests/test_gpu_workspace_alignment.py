"""A workspace at 8 bytes off a 16-byte boundary, which list growth takes and
row-list growth's 16-byte words do not, still grows the oracle's trees: a fit,
and a queue of two jobs."""
import ctypes as C

import numpy as np
import pytest
import torch

from cudatree_b200 import _lib
from cudatree_b200.random_forest import fetch_tree_columns
from oracle import cudatree_oracle as O

from . import gpu_utils as G

pytestmark = pytest.mark.gpu
BOOTSTRAP = _lib.KERNEL_GROUPS.index("bootstrap")
TREES = 2


def _data(n, f, c, seed):
    rng = np.random.default_rng(seed)
    y = rng.integers(0, c, size=n)
    return (rng.normal(size=(n, f)) + 0.5 * y[:, None]).astype(np.float32), y


def _buffers(slots, capacity):
    raw = [torch.zeros(slots * capacity, dtype=torch.int32, device=G.dev()) for _ in range(5)]
    nn = torch.zeros(slots, dtype=torch.int32, device=G.dev())
    return _lib.TreeBuffers(*[r.data_ptr() for r in raw], nn.data_ptr(), capacity), nn, raw


def _assert_oracle(counts, cols, trees):
    assert counts.tolist() == [t.n_nodes for t in trees]
    for col, name in zip(cols, ("left", "right", "feature", "threshold", "value")):
        np.testing.assert_array_equal(col, np.concatenate([getattr(t, name) for t in trees]), err_msg=name)


# launches of the bootstrap group: two per fit (row lists), three per tree (list growth)
@pytest.mark.parametrize("shift,launches", [(0, 2), (8, 3 * TREES), (16, 2)])
@pytest.mark.parametrize("n", [600, 20000])
def test_fit(cuda_device, n, shift, launches):
    x, y = _data(n, 6, 3, 4)
    gp = G.GpuProblem(x, y, 3, 3, bootstrap=True, seed=8)
    gl = G.GpuLists(gp, TREES)
    tb, nn, _raw = _buffers(TREES, 2 * n)
    opts = _lib.FitOptions(_lib.CT_FIT_BATCHED, 0, 32, 0)
    ws = C.c_size_t()
    _lib.call("ct_fit_workspace_size", C.byref(gp.prob), TREES, C.byref(opts), C.byref(ws))
    work = G.dev_bytes(ws.value + shift)
    _lib.call("ct_fit", C.byref(gp.prob), C.byref(gl.lists), 0, TREES, C.byref(opts), C.byref(tb),
              work.data_ptr() + shift, ws.value, G.stream())
    assert _lib.fit_stats()["launches"][BOOTSTRAP] == launches
    counts, cols = fetch_tree_columns(tb, nn, TREES, G.dev())
    _assert_oracle(counts, cols, O.fit_forest(x, y, n_estimators=TREES, max_features=3, seed=8).trees)


@pytest.mark.parametrize("shift,launches", [(0, 2 * 2), (8, 3 * 2 * TREES)])
def test_queue(cuda_device, shift, launches):
    data = [_data(900, 5, 2, 1), _data(12000, 7, 4, 2)]
    gps = [G.GpuProblem(x, y, int(y.max()) + 1, 3, bootstrap=True, seed=20 + k) for k, (x, y) in enumerate(data)]
    lists = [G.GpuLists(gp, TREES) for gp in gps]
    jobs = (_lib.FitJob * 2)()
    for job, gp, gl in zip(jobs, gps, lists):
        job.problem, job.lists, job.n_trees = gp.prob, gl.lists, TREES
    tb, nn, _raw = _buffers(2 * TREES, 2 * max(gp.n for gp in gps))
    opts = _lib.FitOptions(_lib.CT_FIT_BATCHED, 0, 32, 0)
    ws = C.c_size_t()
    _lib.call("ct_fit_queue_workspace_size", jobs, 2, C.byref(opts), C.byref(ws))
    work = G.dev_bytes(ws.value + shift)
    _lib.call("ct_fit_queue", jobs, 2, C.byref(opts), C.byref(tb), work.data_ptr() + shift, ws.value, G.stream())
    assert _lib.fit_stats()["launches"][BOOTSTRAP] == launches
    counts, cols = fetch_tree_columns(tb, nn, 2 * TREES, G.dev())
    ref = [t for k, (x, y) in enumerate(data)
           for t in O.fit_forest(x, y, n_estimators=TREES, max_features=3, seed=20 + k).trees]
    _assert_oracle(counts, cols, ref)
