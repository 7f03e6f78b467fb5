"""Timed cases of the framework: whole fits, forest growth on resident data,
the forest queue, and prediction, from the smallest calls to the largest.

Kinds of case (all through public entry points):

* ``fit``      RandomForestClassifier(...).fit(x, y): host arrays in, trees out
* ``grow``     ct_fit + ct_fetch_trees on data already resident and presorted,
               with buffers a program keeps between fits: the growth alone
* ``queue``    fit_forests: many small forests through shared level steps
* ``predict``  forest.predict / predict_proba on host rows, or
               ct_predict(_compact) on resident rows (``resident``)

Data kinds: ``covtype`` (10 Gaussian columns and two one-hot groups, 54
columns, 7 classes), ``digits`` (small integers, 10 balanced classes),
``wide`` (many noise columns, 50 informative ones) and ``blobs`` (Gaussian
class means, every fourth column rounded so that values tie).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from cudatree_b200 import RandomForestClassifier, _lib, synthetic
from cudatree_b200.forest_queue import fit_forests


# ------------------------------------------------------------------- cases
def _fit(name, data, n, f, c, trees, **kw):
    case = {"name": name, "kind": "fit", "data": data, "n": n, "f": f, "c": c, "trees": trees,
            "max_features": 0, "bootstrap": True, "min_samples_split": 1, "pinned": False}
    case.update(kw)
    return case


def listed():
    return [
        # the smallest fit a user runs: a table of flowers, default arguments;
        # launches, allocations and host work are all of it
        _fit("fit_iris", "blobs", 150, 4, 3, 10),
        # the reference's digits benchmark: every row kept, integer-valued
        # columns, many of them constant in a node
        _fit("fit_digits", "digits", 1797, 64, 10, 50, max_features=8, bootstrap=False),
        # one ordinary job: a ragged shape, 16-bit lists that cannot carry labels
        _fit("fit_blobs", "blobs", 7919, 129, 23, 10),
        # more than 255 classes (two-byte labels) and a raised min_samples_split
        _fit("fit_many_classes", "blobs", 6007, 40, 300, 20, min_samples_split=5),
        # one tree per call, as a caller that grows its trees one by one does
        _fit("grow_one_tree", "covtype", 100003, 54, 7, 1, kind="grow", max_features=7),
        # the headline benchmark: 100 trees of the covtype-shaped table
        _fit("grow_covtype", "covtype", 581012, 54, 7, 100, kind="grow", max_features=7),
        # a table of continuous columns only, two classes
        _fit("grow_continuous", "blobs", 200003, 28, 2, 50, kind="grow"),
        # many columns, many classes: the reference's wide benchmark
        _fit("grow_wide", "wide", 10000, 3000, 100, 200, kind="grow", max_features=55),
        # a queue of uneven small forests, fitted together
        {"name": "queue", "kind": "queue", "jobs": 24, "lo": 500, "hi": 20000, "f_hi": 256, "trees": 10},
        # one request of a few rows against a resident 100-tree forest
        {"name": "predict_few_rows", "kind": "predict", "data": "covtype", "n": 50021, "f": 54, "c": 7, "trees": 100,
         "rows": 3, "proba": False, "resident": False},
        # a full serving batch against a 500-tree forest, rows on the device
        {"name": "predict_batch", "kind": "predict", "data": "covtype", "n": 581012, "f": 54, "c": 7, "trees": 500,
         "rows": 65536, "proba": False, "resident": True},
        # class fractions of wide rows, many classes
        {"name": "predict_proba_wide", "kind": "predict", "data": "wide", "n": 4001, "f": 3000, "c": 100, "trees": 60,
         "rows": 4099, "proba": True, "resident": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "covtype", "continuous", "wide", "queue", "predict", "predict"])
    if kind == "fit":
        n, f = _log_int(rng, 60, 30000), _log_int(rng, 3, 200)
        if rng.random() < 0.3:
            case = _fit("", "digits", n, f, 10, rng.randint(5, 50))
        else:
            case = _fit("", "blobs", n, f, _log_int(rng, 2, 400), rng.randint(3, 30))
        case["c"] = min(case["c"], n)
        case["bootstrap"] = rng.random() < 0.8
        case["min_samples_split"] = rng.choice([1, 1, 2, 7])
        case["max_features"] = rng.choice([0, 0, max(1, f // 3)])
    elif kind == "covtype":
        case = _fit("", "covtype", _log_int(rng, 20000, 400000), 54, 7, _log_int(rng, 1, 100), kind="grow",
                    max_features=7)
    elif kind == "continuous":
        case = _fit("", "blobs", _log_int(rng, 30000, 200000), rng.randint(5, 40), rng.randint(2, 12),
                    _log_int(rng, 2, 40), kind="grow")
    elif kind == "wide":
        case = _fit("", "wide", _log_int(rng, 2000, 10000), _log_int(rng, 400, 2500), rng.randint(2, 100),
                    _log_int(rng, 4, 120), kind="grow")
    elif kind == "queue":
        case = {"kind": "queue", "jobs": rng.randint(4, 20), "lo": 500, "hi": _log_int(rng, 2000, 20000),
                "f_hi": _log_int(rng, 24, 256), "trees": rng.randint(2, 10)}
    else:
        wide = rng.random() < 0.3
        case = {"kind": "predict", "data": "wide" if wide else "covtype", "f": 1500 if wide else 54,
                "n": _log_int(rng, 1000, 4000) if wide else _log_int(rng, 5000, 200000), "c": 100 if wide else 7,
                "trees": _log_int(rng, 5, 60 if wide else 200), "rows": _log_int(rng, 1, 5000 if wide else 65536),
                "proba": rng.random() < 0.4, "resident": rng.random() < 0.4}
        if case["resident"]:
            case["proba"] = False
    case.pop("name", None)
    return case


# -------------------------------------------------------------------- data
def _blobs(n, f, c, seed):
    rng = np.random.default_rng(seed)
    y = np.concatenate([np.arange(min(c, n)), rng.integers(0, c, size=max(0, n - c))])
    rng.shuffle(y)
    means = rng.normal(0.0, 1.0, size=(c, f)).astype(np.float32)
    x = rng.standard_normal((n, f), dtype=np.float32) + means[y]
    x[:, ::4] = np.round(x[:, ::4], 1)
    return x, y.astype(np.int64)


def _data(kind, n, f, c, seed):
    if kind == "covtype":
        return synthetic.covtype_like(n, seed=1000 + seed)
    if kind == "digits":
        return synthetic.digits_like(n, f, c, seed=1000 + seed)
    if kind == "wide":
        return synthetic.wide(n, f, c, seed=1000 + seed)
    return _blobs(n, f, c, 1000 + seed)


def _forest(case, seed, **kw):
    return RandomForestClassifier(case["trees"], max_features=case.get("max_features") or None,
                                  min_samples_split=case.get("min_samples_split", 1),
                                  bootstrap=case.get("bootstrap", True), seed=2000 + seed, **kw)


def _bytes(n):
    return torch.empty(int(n) + 64, dtype=torch.uint8, device="cuda")


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _workspace(fn, *args):
    ws = C.c_size_t()
    _lib.call(fn, *args, C.byref(ws))
    return ws.value


def _node_bound(case):
    """Room for a case's nodes, the same for every seed: twice the rows of a
    tree is the most there can be; the covtype-shaped and two-class tables
    stay far below."""
    per_tree = {"covtype": case["n"] // 4 + 64, "wide": case["n"]}.get(case["data"], 2 * case["n"])
    return case["trees"] * per_tree


def _node_columns(trees, bound):
    """Host arrays a program keeps for its trees: nodes per tree, then left
    and right child, feature, threshold and value of every node, tree after
    tree (the used part is written by each fit, the rest stays zero)."""
    return [np.zeros(trees, np.int64)] + [np.zeros(bound, dt) for dt in
                                          (np.uint32, np.uint32, np.uint16, np.float32, np.uint32)]


# ----------------------------------------------------------------- prepare
def _prepare_grow(case, seed):
    """Resident data (feature-major samples, labels, presort) and the buffers
    of a fit, which a program that grows forests on the device keeps."""
    x, y = _data(case["data"], case["n"], case["f"], case["c"], seed)
    n, f = x.shape
    c, trees = case["c"], case["trees"]
    ib, lb = (2 if n <= 0xFFFF else 4), (1 if c <= 0xFF else 2)
    st = {"n": n, "f": f}
    xd = torch.from_numpy(x).cuda()
    st["x_fm"] = torch.empty((f, n), dtype=torch.float32, device="cuda")
    _lib.call("ct_transpose_rows", xd.data_ptr(), n, f, st["x_fm"].data_ptr(), None, _stream())
    st["labels"] = torch.from_numpy(y.astype(np.uint8 if lb == 1 else np.uint16).view(np.uint8)).cuda()
    st["presort"] = _bytes(f * n * ib)
    b = _workspace("ct_presort_workspace_size", n, f)
    work = _bytes(b)
    _lib.call("ct_presort", st["x_fm"].data_ptr(), n, f, ib, st["presort"].data_ptr(), work.data_ptr(), b, _stream())
    del xd, work
    m = case["max_features"] or int(math.ceil(math.sqrt(f)))
    st["prob"] = _lib.Problem(st["x_fm"].data_ptr(), st["labels"].data_ptr(), st["presort"].data_ptr(), n, f, c, ib, lb,
                              m, case["min_samples_split"], int(case["bootstrap"]), 2000 + seed)
    st["si"] = [_bytes(trees * f * n * ib) for _ in range(2)]
    st["mark"] = _bytes(_lib.mark_bytes(n, trees))
    st["lists"] = _lib.Lists(st["si"][0].data_ptr(), st["si"][1].data_ptr(), st["mark"].data_ptr(), n, trees)
    st["raw"] = [torch.empty(trees * 2 * n, dtype=torch.int32, device="cuda") for _ in range(5)]
    st["n_nodes"] = torch.zeros(trees, dtype=torch.int32, device="cuda")
    st["tb"] = _lib.TreeBuffers(*[r.data_ptr() for r in st["raw"]], st["n_nodes"].data_ptr(), 2 * n)
    st["opts"] = _lib.FitOptions(_lib.CT_FIT_BATCHED, 0, 32, 0)
    st["ws_bytes"] = _workspace("ct_fit_workspace_size", C.byref(st["prob"]), trees, C.byref(st["opts"]))
    st["ws"] = _bytes(st["ws_bytes"])
    st["trees"] = trees
    st["out"] = _node_columns(trees, _node_bound(case))
    st["scratch_bytes"] = int(_lib.load().ct_fetch_trees_scratch(st["out"][1].size, trees))
    st["scratch"] = _bytes(st["scratch_bytes"])
    torch.cuda.synchronize()
    return st


def _queue_shapes(case):
    """(rows, features, classes) of each job: fixed by the case, spread over
    its ranges (the inputs' values come from the seed)."""
    rng = np.random.default_rng(case["jobs"] * 7919 + case["hi"])
    shapes = []
    for _ in range(case["jobs"]):
        n = int(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]))))
        shapes.append((n, int(rng.integers(16, case["f_hi"] + 1)), int(rng.integers(2, 51))))
    return shapes


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grow":
        return {"case": case, **_prepare_grow(case, seed)}
    if kind == "queue":
        jobs = [_blobs(n, f, c, 1000 + seed * 4096 + i) for i, (n, f, c) in enumerate(_queue_shapes(case))]
        shapes = _queue_shapes(case)
        out = _node_columns(case["trees"] * len(jobs), sum(case["trees"] * 2 * n for n, _, _ in shapes))
        return {"case": case, "jobs": jobs, "seed": seed, "out": out}
    x, y = _data(case["data"], case["n"], case["f"], case["c"], seed)
    if kind == "fit":
        if case["pinned"]:
            x, y = torch.from_numpy(x).pin_memory(), torch.from_numpy(y)
        return {"case": case, "x": x, "y": y, "seed": seed, "out": _node_columns(case["trees"], _node_bound(case))}
    # predict: a fitted forest, resident from its first prediction on
    forest = _forest(case, seed).fit(x, y)
    rows = np.ascontiguousarray(x[np.random.default_rng(3000 + seed).integers(0, x.shape[0], case["rows"])])
    rows = rows + np.random.default_rng(4000 + seed).normal(0.0, 0.1, rows.shape).astype(np.float32)
    st = {"case": case, "forest": forest, "rows": rows}
    if case["resident"]:
        st["nodes"], st["offs"], st["compact"] = forest._device_forest()
        st["x"] = torch.from_numpy(rows).cuda()
        st["votes"] = torch.empty((rows.shape[0], forest.n_labels), dtype=torch.int32, device="cuda")
        st["pred"] = torch.empty(rows.shape[0], dtype=torch.int32, device="cuda")
    else:
        forest.predict(rows[:1])
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------------- run
def _store_trees(trees, out):
    names = ("left_children", "right_children", "feature_idx_array", "feature_threshold_array", "values_array")
    out[0][:] = [t.n_nodes for t in trees]
    total = int(out[0].sum())
    for name, col in zip(names, out[1:]):
        np.concatenate([getattr(t, name) for t in trees], out=col[:total])
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "grow":
        _lib.call("ct_fit", C.byref(state["prob"]), C.byref(state["lists"]), 0, state["trees"], C.byref(state["opts"]),
                  C.byref(state["tb"]), state["ws"].data_ptr(), state["ws_bytes"], _stream())
        counts = state["n_nodes"].cpu().numpy().astype(np.uint32)
        out = state["out"]
        out[0][:] = counts
        if int(out[0].sum()) > out[1].size:
            raise RuntimeError("more nodes than the case leaves room for")
        _lib.call("ct_fetch_trees", C.byref(state["tb"]), state["trees"], counts.ctypes.data,
                  state["scratch"].data_ptr(), state["scratch_bytes"], *[c.ctypes.data for c in out[1:]], _stream())
        return out
    if kind == "fit":
        forest = _forest(case, state["seed"]).fit(state["x"], state["y"])
        return _store_trees(forest._trees, state["out"])
    if kind == "queue":
        forests = fit_forests(state["jobs"], n_estimators=case["trees"],
                              seeds=[2000 + state["seed"] + i for i in range(len(state["jobs"]))])
        return _store_trees([t for f in forests for t in f._trees], state["out"])
    forest = state["forest"]
    if case["resident"]:
        nodes = state["nodes"]
        _lib.call("ct_predict_compact" if state["compact"] else "ct_predict", nodes.data_ptr(),
                  nodes.numel() // (8 if state["compact"] else 16), state["offs"].data_ptr(), len(forest._trees),
                  state["x"].data_ptr(), state["x"].shape[0], forest.n_features, forest.n_labels,
                  state["votes"].data_ptr(), state["pred"].data_ptr(), _stream())
        return [state["pred"], state["votes"]]
    return forest.predict_proba(state["rows"]) if case["proba"] else forest.predict(state["rows"])


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: samples and labels read once, nodes (or labels) written once.
    Operations: one comparison per row, tree and level of a balanced tree, and
    per sampled column in a fit."""
    if case["kind"] == "queue":
        total = {"bytes": 0, "flops": 0}
        for n, f, c in _queue_shapes(case):
            w = work({"kind": "fit", "n": n, "f": f, "c": c, "trees": case["trees"], "max_features": 0,
                      "min_samples_split": 1})
            total = {k: total[k] + w[k] for k in total}
        return total
    depth = max(1.0, math.log2(case["n"]))
    if case["kind"] == "predict":
        rows, trees = case["rows"], case["trees"]
        # a node is 8 bytes; a walk needs one node per level at most, and no
        # more nodes are read than the forest holds (one leaf per 8 rows or so)
        nodes = min(rows * trees * depth, trees * case["n"] / 4)
        return {"bytes": int(rows * case["f"] * 4 + nodes * 8 + rows * (8 * case["c"] if case["proba"] else 4 * case["c"] + 4)),
                "flops": int(rows * trees * depth)}
    m = case["max_features"] or int(math.ceil(math.sqrt(case["f"])))
    nodes = case["trees"] * case["n"] / 4 / case["min_samples_split"]
    return {"bytes": int(case["n"] * (4 * case["f"] + 1) + nodes * 18),
            "flops": int(case["n"] * case["trees"] * m * depth)}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """Predictions by walking the fitted trees in plain torch, fractions in 64
    bits.  Fits return trees (whole numbers and values of the input), which
    have no further value to be compared with."""
    if case["kind"] != "predict":
        return None
    state = prepare(case, seed)
    forest = state["forest"]
    x = torch.from_numpy(state["rows"]).cuda().double()
    votes = torch.zeros((x.shape[0], forest.n_labels), dtype=torch.float64, device="cuda")
    row = torch.arange(x.shape[0], device="cuda")
    for t in forest._trees:
        left = torch.from_numpy(t.left_children.astype(np.int64)).cuda()
        feat = torch.from_numpy(t.feature_idx_array.astype(np.int64)).cuda()
        thr = torch.from_numpy(t.feature_threshold_array.astype(np.float64)).cuda()
        val = torch.from_numpy(t.values_array.astype(np.int64)).cuda()
        pos = torch.zeros_like(row)
        while True:
            inner = left[pos] != 0
            if not bool(inner.any()):
                break
            nxt = left[pos] + (x[row, feat[pos]] >= thr[pos]).long()
            pos = torch.where(inner, nxt, pos)
        votes[row, val[pos]] += 1.0
    ids = votes.argmax(dim=1).cpu().numpy()
    if case["resident"]:
        return [torch.from_numpy(ids.astype(np.int32)).cuda(), votes.int()]
    if case["proba"]:
        return (votes / len(forest._trees)).cpu().numpy()
    return forest.compt_table[ids]
