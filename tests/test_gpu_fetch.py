"""Read-back of raw trees: breadth-first renumbering on the device against the
host's (ct_tree_canonicalize), for shuffled raw ids, trees deeper than the
device walk's level limit, the smaller scratch of the host path, and malformed
trees."""
import ctypes as C

import numpy as np
import pytest
import torch

from cudatree_b200 import _lib

from . import gpu_utils as G

pytestmark = pytest.mark.gpu


def _tree(n_inner, seed, chain=False):
    """A raw tree with shuffled ids (the root keeps id 0)."""
    rng = np.random.default_rng(seed)
    n = 2 * n_inner + 1
    left, right = np.zeros(n, np.int64), np.zeros(n, np.int64)
    leaves, made = [0], 1
    for _ in range(n_inner):
        k = len(leaves) - 1 if chain else int(rng.integers(len(leaves)))
        p = leaves.pop(k)
        left[p], right[p] = made, made + 1
        leaves += [made, made + 1]
        made += 2
    perm = np.concatenate([[0], 1 + rng.permutation(n - 1)])
    out = {"left": np.zeros(n, np.uint32), "right": np.zeros(n, np.uint32)}
    out["left"][perm] = np.where(left > 0, perm[left], 0)
    out["right"][perm] = np.where(right > 0, perm[right], 0)
    out["feature"] = rng.integers(0, 60000, n).astype(np.uint32)
    out["threshold"] = rng.normal(size=n).astype(np.float32)
    out["value"] = rng.integers(0, 1000, n).astype(np.uint32)
    return out


def _fetch(trees, scratch_bytes=None):
    cap = max(t["left"].size for t in trees) + 3
    counts = np.array([t["left"].size for t in trees], np.uint32)
    total = int(counts.sum())
    bufs = []
    for name in ("left", "right", "feature", "threshold", "value"):
        a = np.full((len(trees), cap), 7, trees[0][name].dtype)
        for i, t in enumerate(trees):
            a[i, :counts[i]] = t[name]
        bufs.append(G.to_dev(a))
    nn = G.to_dev(counts)
    tb = _lib.TreeBuffers(*[b.data_ptr() for b in bufs], nn.data_ptr(), cap)
    sb = int(_lib.load().ct_fetch_trees_scratch(total, len(trees))) if scratch_bytes is None else scratch_bytes
    scratch = torch.zeros(sb, dtype=torch.uint8, device=G.dev())
    cols = [np.empty(total, dt) for dt in (np.uint32, np.uint32, np.uint16, np.float32, np.uint32)]
    _lib.call("ct_fetch_trees", C.byref(tb), len(trees), counts.ctypes.data, scratch.data_ptr(), sb,
              *[c.ctypes.data for c in cols], G.stream())
    return counts, cols


def _canonical(t):
    n = t["left"].size
    cols = [np.empty(n, dt) for dt in (np.uint32, np.uint32, np.uint16, np.float32, np.uint32)]
    _lib.call("ct_tree_canonicalize", *[t[k].ctypes.data for k in ("left", "right", "feature", "threshold", "value")],
              n, *[c.ctypes.data for c in cols])
    return cols


@pytest.mark.parametrize("sizes,chain", [([0], False), ([1, 0, 2], False), ([255, 256, 257, 3], False),
                                         ([5000, 1, 70000], False), ([4094], True), ([4100, 6], True)])
def test_renumbering_matches_the_host(cuda_device, sizes, chain):
    trees = [_tree(k, i, chain) for i, k in enumerate(sizes)]
    want = [np.concatenate(c) for c in zip(*[_canonical(t) for t in trees])]
    total = sum(t["left"].size for t in trees)
    for scratch in (None, 20 * total + 4 * (len(trees) + 1) + 256):
        _, got = _fetch(trees, scratch)
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("kind", ["cycle", "out_of_range", "unreachable", "shared"])
def test_malformed_trees_are_refused(cuda_device, kind):
    t = _tree(20, 3)
    inner = np.flatnonzero(t["left"])
    leaf = np.flatnonzero(t["left"] == 0)
    if kind == "cycle":
        t["left"][inner[-1]] = inner[1]
    elif kind == "out_of_range":
        t["right"][inner[2]] = 41
    elif kind == "unreachable":
        t["left"][inner[3]] = t["right"][inner[3]] = 0
    else:
        t["left"][inner[2]] = t["left"][inner[4]]
    assert leaf.size
    with pytest.raises(_lib.CudaTreeError):
        _fetch([_tree(3, 1), t])
