"""Tree groups of a prediction and the form of its walk (CPU: the library's rule):
every tree is in a group, a launch of many rows stays within a grid's blocks,
and calls where the vote table and the rows read again cost more than groups
gain keep one group."""
import ctypes as C

import pytest

from cudatree_b200 import _lib

GRID_MOST = 2**31 - 1


class _Plan(C.Structure):
    _fields_ = [("group", C.c_uint32), ("few_in_flight", C.c_bool)]


def _plan(n_trees, tree_bytes, rows, features=10, classes=2, votes=True):
    fn = getattr(_lib.load(), "_ZN2ct12predict_planEjmmjjjb")
    fn.restype = _Plan
    fn.argtypes = [C.c_uint32, C.c_uint64, C.c_size_t, C.c_uint32, C.c_uint32, C.c_uint32, C.c_bool]
    return fn(n_trees, n_trees * max(1, tree_bytes // 8), 8, rows, features, classes, votes)


def _rows_per_tile(rows, features, classes):
    r = 32
    while r > 1 and (r // 2 >= rows or r * classes * 4 > 65536 or r * features * 4 > 32768):
        r //= 2
    return r


@pytest.mark.parametrize("rows", [1, 1000, 65536, 10**7, 2**31, 2**32 - 1])
@pytest.mark.parametrize("n_trees,tree_bytes", [(1, 400), (100, 5600), (1000, 6400), (5000, 16000), (40000, 24000)])
@pytest.mark.parametrize("features", [4, 900, 60000])
def test_groups_cover_the_trees_within_a_grid(rows, n_trees, tree_bytes, features):
    tiles = -(-rows // _rows_per_tile(rows, features, 2))
    if tiles > GRID_MOST:
        pytest.skip("more tiles than blocks with one group: refused at any size of group")
    g = _plan(n_trees, tree_bytes, rows, features).group
    assert 1 <= g <= n_trees
    assert -(-n_trees // g) * tiles <= GRID_MOST


# calls measured with one group and with several (us): the faster is taken
@pytest.mark.parametrize("n_trees,tree_bytes,rows,features,classes,grouped", [
    (202, 16_900, 4618, 1023, 2, False), (308, 16_100, 63762, 896, 300, False), (36, 8_400, 18225, 192, 7, False),
    (53, 13_200, 16020, 14, 300, False), (128, 1_400, 6289, 393, 3, False), (57, 700, 13936, 5, 10, False),
    (500, 75_000, 65536, 54, 7, True), (100, 24_000, 2048, 54, 7, True), (1000, 4_800, 7848, 20, 2, True),
    (1174, 9_100, 16633, 476, 300, True), (250, 60_000, 2358, 54, 7, True), (500, 20_000, 40, 54, 7, True)])
def test_groups_where_they_pay(n_trees, tree_bytes, rows, features, classes, grouped):
    assert (_plan(n_trees, tree_bytes, rows, features, classes).group < n_trees) == grouped


@pytest.mark.parametrize("rows", [1, 500, 5000, 10**6])
def test_no_groups_without_a_vote_table(rows):
    assert _plan(700, 30_000, rows, votes=False).group == 700


@pytest.mark.parametrize("n_trees,tree_bytes,rows,features,classes,few", [
    (32, 75_000, 65536, 10, 2, True), (500, 75_000, 65536, 54, 7, True),            # one round
    (100, 1_200, 65536, 20, 2, True), (300, 1_900, 65536, 20, 2, True),             # small groups, every SM at work
    (279, 1_000, 63112, 165, 100, False), (54, 8_400, 901, 24, 7, False)])          # no room for six blocks; few blocks
def test_form(n_trees, tree_bytes, rows, features, classes, few):
    assert _plan(n_trees, tree_bytes, rows, features, classes).few_in_flight == few
