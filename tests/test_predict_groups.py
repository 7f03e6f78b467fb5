"""Tree groups of a prediction (CPU: the library's size function): every tree is
in a group, and a launch of many rows stays within a grid's blocks."""
import ctypes as C

import pytest

from cudatree_b200 import _lib

GRID_MOST = 2**31 - 1


def _group_size(n_trees, n_nodes, node_bytes, rows_per_tile, tiles):
    fn = getattr(_lib.load(), "_ZN2ct18predict_group_sizeEjmmjj")
    fn.restype, fn.argtypes = C.c_uint32, [C.c_uint32, C.c_uint64, C.c_size_t, C.c_uint32, C.c_uint32]
    return fn(n_trees, n_nodes, node_bytes, rows_per_tile, tiles)


@pytest.mark.parametrize("rows", [1, 1000, 65536, 10**7, 2**31, 2**32 - 1])
@pytest.mark.parametrize("n_trees,nodes_per_tree", [(1, 50), (100, 700), (1000, 800), (5000, 2000), (40000, 3000)])
@pytest.mark.parametrize("rows_per_tile", [1, 8, 32])
def test_groups_cover_the_trees_within_a_grid(rows, n_trees, nodes_per_tree, rows_per_tile):
    tiles = -(-rows // rows_per_tile)
    if tiles > GRID_MOST:
        pytest.skip("more tiles than blocks with one group: refused at any size of group")
    g = _group_size(n_trees, n_trees * nodes_per_tree, 8, rows_per_tile, tiles)
    assert 1 <= g <= n_trees
    assert -(-n_trees // g) * tiles <= GRID_MOST
