"""The device's candidate test itself (is_candidate_sorted): neighbours of every
magnitude whose gap lies at, just below and just above 1e-5 are split, or not, as
the double test x + 1e-5 < x_next has it."""
import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier
from oracle import cudatree_oracle as O

from . import gpu_utils as G
from .test_gpu_fit import _assert_same_trees

pytestmark = pytest.mark.gpu


def _neighbours():
    """(x, x_next) with x <= x_next: a few float steps apart, and around the gaps that decide."""
    rng = np.random.default_rng(11)
    base = np.concatenate([rng.normal(size=300), rng.normal(size=300) * 1e-5, rng.uniform(-300, 300, 300),
                           rng.normal(size=100) * 1e6, rng.normal(size=40) * 1e30, rng.normal(size=40) * 1e-30,
                           [0.0, -0.0, np.inf, -np.inf, 127.99999, 128.0, -128.0, 3.4e38, -3.4e38,
                            1e-45]]).astype(np.float32)
    pairs = [(base, np.full_like(base, np.inf)), (np.full_like(base, -np.inf), base), (base, base)]
    for steps in (1, 2, 3, 7, 100):
        up = base.copy()
        for _ in range(steps):
            up = np.nextafter(up, np.float32(np.inf))
        pairs.append((base, up))
    for gap in (9.9998e-6, 9.9999e-6, 1e-5, 1.00001e-5, 1.00002e-5, 1e-4, 1.0):
        centre = (base.astype(np.float64) + gap).astype(np.float32)
        for k in range(-4, 5):
            near = centre.copy()
            for _ in range(abs(k)):
                near = np.nextafter(near, np.float32(np.inf if k > 0 else -np.inf))
            pairs.append((base, near))
    a, b = np.concatenate([p[0] for p in pairs]), np.concatenate([p[1] for p in pairs])
    ok = b >= a
    return a[ok], b[ok]


def test_two_row_nodes_split_as_the_double_test_says(cuda_device):
    a, b = _neighbours()
    k = a.size
    x = np.stack([a, b], axis=1).reshape(-1, 1)  # rows 2 i and 2 i + 1 are node i
    gp = G.GpuProblem(x, np.tile([0, 1], k), 2, 1)
    gl = G.GpuLists(gp)
    gl.put(0, np.arange(2 * k, dtype=np.int64)[None, :])
    nodes = G.node_array([dict(slot=0, start=2 * i, n=2, raw_id=i, key=i, impurity=1.0, buf=0) for i in range(k)])
    res, _, _ = G.split_nodes(gp, gl, nodes, np.ones((k, 2)))
    exact = a.astype(np.float64) + 0.00001 < b.astype(np.float64)
    assert 0.2 < exact.mean() < 0.9
    np.testing.assert_array_equal(res["feature"] == 0, exact)


@pytest.mark.parametrize("n,c", [(30, 3), (400, 3), (400, 12), (1500, 3), (6000, 12), (12000, 3), (12000, 12)])
def test_row_lists_skip_the_same_candidates(cuda_device, n, c):
    """Columns whose sorted neighbours lie about 1e-5 apart, through the node sizes of row-list growth."""
    rng = np.random.default_rng(n + c)
    steps = rng.choice([0.0, 9.9e-6, 9.99999e-6, 1e-5, 1.000001e-5, 1.01e-5, 3e-5], size=(n, 3))
    x = (np.cumsum(steps, axis=0) + [0.0, 1.0, -0.05]).astype(np.float32)
    x = np.stack([rng.permutation(x[:, k]) for k in range(3)], axis=1)
    y = rng.integers(0, c, size=n)
    kw = dict(n_estimators=2, max_features=2, bootstrap=False, seed=c)
    _assert_same_trees(RandomForestClassifier(**kw).fit(x, y)._trees, O.fit_forest(x, y, **kw).trees)
