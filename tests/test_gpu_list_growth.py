"""List growth (every feature's sorted list kept per node) in the batched form.
It grows the tables that row-list growth does not take; here the list buffers
start 8 bytes off a 16-byte boundary, which sends any fit to it.  Its options,
subtree sizes, entry widths, feature kinds and level loops, and its queue, grow
the oracle's trees."""
import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier, _lib, synthetic
from cudatree_b200.forest_queue import fit_forests
from oracle import cudatree_oracle as O

from .test_gpu_fit import _assert_same_trees, _synthetic, _two_valued_data
from .test_gpu_queue import _blobs

pytestmark = pytest.mark.gpu
BOOTSTRAP = _lib.KERNEL_GROUPS.index("bootstrap")


@pytest.fixture(autouse=True)
def lists_off_alignment(monkeypatch):
    lists = _lib.Lists

    def shifted(si0, si1, *rest):  # (both buffers are padded by 64 bytes)
        return lists(si0 and si0 + 8, si1 and si1 + 8, *rest)

    monkeypatch.setattr(_lib, "Lists", shifted)


def _fit(x, y, tuned=None, **kw):
    """A fit and the check that it kept the lists: their bootstrap takes launches per tree."""
    attrs = {k: kw.pop(k) for k in ("virtual_features", "host_level_loop", "step_nodes", "graph_samples") if k in kw}
    f = RandomForestClassifier(**kw)
    f._tuned = tuned
    for k, v in attrs.items():
        setattr(f, k, v)
    f.fit(x, y)
    assert f.last_fit_stats["launches"][BOOTSTRAP] == (3 if f.bootstrap else 1) * f.n_estimators
    return f


@pytest.mark.parametrize("n,f,c", [(70000, 6, 5), (30000, 7, 3)])
def test_partition_options(cuda_device, n, f, c):
    """Every partition shape, huge-segment threshold and small-segment cutoff;
    32-bit entries and 16-bit ones."""
    x, y = _synthetic(n, f, c, 61)
    ref = O.fit_forest(x, y, n_estimators=2, seed=61)
    options = [(s, h, 0) for s in range(4) for h in (0, 16384, 0xFFFFFFFF)]
    options += [(0, 0, 1024), (1, 16384, 2048), (2, 0, 4096), (0, 0xFFFFFFFF, 65536)]
    for shape, huge, small in options:
        g = _fit(x, y, {"part_shape": shape, "huge_rows": huge, "small_rows": small}, n_estimators=2, seed=61)
        _assert_same_trees(g._trees, ref.trees)


@pytest.mark.parametrize("mss", [1, 3])
def test_subtree_cutoffs(cuda_device, mss):
    """Subtrees of one row per lane (to 32) and of four (to 128), noise labels."""
    x, _ = _synthetic(1500, 24, 5, 31)
    y = np.random.default_rng(1031).integers(0, 5, size=1500)
    ref = O.fit_forest(x, y, n_estimators=3, min_samples_split=mss, seed=77)
    for cut in (0, 8, 32, 64, 128):
        f = _fit(x, y, n_estimators=3, min_samples_split=mss, seed=77, subtree_cutoff=cut)
        _assert_same_trees(f._trees, ref.trees)


@pytest.mark.parametrize("n,f,c", [(4096, 8, 16), (4097, 8, 16), (66000, 6, 3), (2000, 5, 1), (3000, 9, 300)])
def test_entry_widths(cuda_device, n, f, c):
    """16-bit entries filled by row and label, without room for the label, 32-bit
    ones, one class, and 16-bit labels."""
    x, y = _synthetic(n, f, c, 11)
    _assert_same_trees(_fit(x, y, n_estimators=2, seed=5)._trees, O.fit_forest(x, y, n_estimators=2, seed=5).trees)


@pytest.mark.parametrize("n,c,piece", [(700, 3, 0), (9000, 5, 0), (9000, 12, 1024), (70000, 7, 4096)])
@pytest.mark.parametrize("bootstrap", [True, False])
def test_two_valued_features(cuda_device, n, c, piece, bootstrap):
    x, y = _two_valued_data(n, c, 17)
    kw = dict(n_estimators=2, max_features=4, seed=29, bootstrap=bootstrap)
    f = _fit(x, y, {"scan_piece": piece, "subtree_cutoff": 32}, **kw)
    _assert_same_trees(f._trees, O.fit_forest(x, y, **kw).trees)


@pytest.mark.parametrize("n", [3000, 40000, 70000])
@pytest.mark.parametrize("virtual", [True, False])
def test_virtual_features(cuda_device, n, virtual):
    x, y = synthetic.covtype_like(n=n, seed=n)
    kw = dict(n_estimators=2, max_features=7, seed=n)
    _assert_same_trees(_fit(x, y, virtual_features=virtual, **kw)._trees, O.fit_forest(x, y, **kw).trees)


@pytest.mark.parametrize("f", [65, 130, 300])
def test_constant_feature_masks(cuda_device, f):
    """One mask word per 64 features, kept when one feature in eight is two-valued."""
    rng = np.random.default_rng(f)
    n = 2500
    y = rng.integers(0, 4, size=n)
    x = (rng.normal(size=(n, f)) + 0.8 * y[:, None] * (np.arange(f) % 5 == 0)).astype(np.float32)
    x[:, 1::4] = rng.integers(0, 2, size=(n, len(range(1, f, 4))))
    x[:, 3::8] = rng.integers(0, 3, size=(n, len(range(3, f, 8))))
    for j in (2, 64, f - 1):
        x[:, j] = 7.0
    kw = dict(n_estimators=2, max_features=9, seed=f)
    _assert_same_trees(_fit(x, y, **kw)._trees, O.fit_forest(x, y, **kw).trees)


@pytest.mark.parametrize("step_nodes", [0, 7])
@pytest.mark.parametrize("cut", [32, 128])
def test_level_loops(cuda_device, step_nodes, cut):
    """Every level in the graph, the first ones from the host, all from the host."""
    x, y = _synthetic(5000, 10, 6, 41)
    ref = O.fit_forest(x, y, n_estimators=3, seed=43)
    for host, graph_samples in ((False, 0xFFFFFFFF), (False, 3000), (True, 0)):
        f = _fit(x, y, n_estimators=3, seed=43, subtree_cutoff=cut, host_level_loop=host, step_nodes=step_nodes,
                 graph_samples=graph_samples)
        _assert_same_trees(f._trees, ref.trees)


def test_queue(cuda_device):
    """Jobs of both entry widths, of up to 130 features and of one to 40 classes share list-growth levels."""
    specs = [(20, 5, 1), (900, 70, 5), (3000, 30, 3), (70000, 6, 4), (40, 3, 2), (5000, 130, 40), (1500, 12, 7)]
    jobs = [_blobs(n, f, c, 300 + k, ties=k % 2 == 0) for k, (n, f, c) in enumerate(specs)]
    seeds = [500 + k for k in range(len(jobs))]
    for (x, y), seed, g in zip(jobs, seeds, fit_forests(jobs, n_estimators=3, seeds=seeds)):
        assert g.last_fit_stats["launches"][BOOTSTRAP] % 9 == 0  # three per tree of its group (row lists: two per job)
        _assert_same_trees(g._trees, O.fit_forest(x, y, n_estimators=3, seed=seed).trees)
