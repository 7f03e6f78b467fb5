"""Workspace that row-list growth asks for (CPU: the size functions need no GPU)."""
import ctypes as C

import pytest

from cudatree_b200 import _lib


def _workspace(n, f, c, m, trees):
    p = _lib.Problem(None, None, None, n, f, c, 2 if n <= 0xFFFF else 4, 1 if c <= 255 else 2, m, 1, 1, 0)
    o = _lib.FitOptions(_lib.CT_FIT_BATCHED, 0, 32, 0)
    ws = C.c_size_t()
    _lib.call("ct_fit_workspace_size", C.byref(p), trees, C.byref(o), C.byref(ws))
    return ws.value


# 32-bit indices hold (4 F - 8) / 8 planes behind the row list of each buffer: 49 of 100 features, 26 of 54, 8 of 18
@pytest.mark.parametrize("n,f,c,there", [(1_000_000, 100, 2, 98), (581_012, 54, 7, 52), (500_000, 18, 2, 16)])
def test_only_planes_past_the_list_buffers_take_workspace(n, f, c, there):
    trees = 100
    plane = 8 * trees * n
    fits, one_more = _workspace(n, f, c, there, trees), _workspace(n, f, c, there + 1, trees)
    # the plane and the piece lists of one more selected feature (less where list growth needs the most)
    assert 0 < one_more - fits < 1.5 * plane
    assert _workspace(n, f, c, f, trees) - fits < 1.5 * plane * (f - there)


def test_all_features_selected_fit_beside_their_lists():
    """1,000,000 x 100, all selected, 100 trees: 80 GB of index lists and the
    workspace stay well inside one GPU."""
    assert _workspace(1_000_000, 100, 2, 100, 100) < 20e9
    assert _workspace(60_000, 784, 1000, 784, 100) < 160e9
