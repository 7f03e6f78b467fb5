"""A root of one class splits on the first candidate of its lowest feature, as
every form does, also where its whole order is one piece of the scan."""
import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier
from oracle import cudatree_oracle as O

from .test_gpu_fit import _assert_same_trees

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("piece", [0, 16384])
@pytest.mark.parametrize("label", [0, 1])
def test_root_of_one_class(cuda_device, piece, label):
    """270 trees of 64 selected features make enough pieces for a level to keep
    pieces of 16,384 positions, so all 12,000 rows are one."""
    x = np.random.default_rng(1).normal(size=(12000, 64)).astype(np.float32)
    y = np.full(12000, label)
    forest = RandomForestClassifier(270, max_features=64, bootstrap=False, seed=3)
    forest._tuned = {"scan_piece": piece}
    forest.fit(x, y)
    ref = O.fit_forest(x, y, n_estimators=1, max_features=64, bootstrap=False, seed=3).trees
    for tree in forest._trees[::53]:
        _assert_same_trees([tree], ref)
