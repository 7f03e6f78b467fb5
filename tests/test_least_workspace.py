"""Where the workspace of row-list growth is not to be had, fits, the autotuner
and the queue take the least workspace instead of giving up (CPU: the device's
memory is a count, and the fit itself is replaced)."""
import ctypes as C

import numpy as np
import pytest
import torch

from cudatree_b200 import _lib, forest_queue, random_forest
from cudatree_b200.random_forest import RandomForestClassifier

GB = 10**9
WORKSPACE = {"ct_fit": 7, "ct_autotune": 6}  # position of the workspace's bytes


class Device:
    """A device that holds `room` bytes; what is allocated is counted, not held."""

    def __init__(self, monkeypatch, room):
        self.room, self.used, self.given = room, 0, []
        self.dev = torch.device("cpu")
        self.empty, self.call = torch.empty, _lib.call
        monkeypatch.setattr(random_forest, "_device", lambda: self.dev)
        monkeypatch.setattr(random_forest, "_stream", lambda: None)
        monkeypatch.setattr(random_forest, "_dev_bytes", lambda n, dev: self.take(n))
        monkeypatch.setattr(random_forest, "free_bytes", lambda dev: self.room)
        monkeypatch.setattr(torch.cuda, "get_device_properties", lambda *a: type("P", (), {"total_memory": self.room}))
        monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "counted")
        monkeypatch.setattr(_lib, "call", self._call)

    def take(self, nbytes):
        if self.used + nbytes > self.room:
            raise torch.OutOfMemoryError("counted device is full")
        self.used += nbytes
        return self.empty(16, dtype=torch.uint8)

    def _call(self, name, *args):
        if name in WORKSPACE:
            self.given.append(int(args[WORKSPACE[name]]))
        else:
            self.call(name, *args)


def _forest(monkeypatch, n, f, trees):
    forest = RandomForestClassifier(trees, max_features=2, seed=1)
    forest.n_samples, forest.n_features, forest.n_labels = n, f, 2
    forest.index_bytes, forest._m, forest._seed = random_forest.best_index_bytes(n), 2, 1
    forest.dtype_labels = np.dtype(np.uint8)
    forest.bfs_threshold = 5000
    forest._x_fm = forest._labels = forest._presort = torch.empty(1)
    monkeypatch.setattr(forest, "_fetch_trees", lambda tb, nn, kk, dev: [None] * kk)
    return forest


def _sizes(forest, trees):
    prob, opts = forest._problem(), forest._fit_options(_lib.CT_FIT_BATCHED, 0)
    return [_lib.size_of(f"ct_fit_{w}workspace_size", C.byref(prob), trees, C.byref(opts)) for w in ("", "least_")]


# room for one tree's index lists and the least workspace, and for more with the larger one
@pytest.mark.parametrize("spare,larger", [(0, False), (200 * GB, True)])
def test_one_tree_of_a_table_that_fills_the_device(monkeypatch, spare, larger):
    n, f = 900_000, 4000
    forest = _forest(monkeypatch, n, f, 1)
    full, least = _sizes(forest, 1)
    assert full > least + 60 * GB
    lists = 2 * 4 * n * f + _lib.mark_bytes(n, 1)
    dev = Device(monkeypatch, lists + least + GB // 10 + spare)
    assert len(forest._fit_trees(0, 1, "batched", 0)) == 1
    assert dev.given == [full if larger else least]


def test_autotuner(monkeypatch):
    n, f = 900_000, 2000
    forest = _forest(monkeypatch, n, f, 1)
    _, least = _sizes(forest, 1)
    dev = Device(monkeypatch, 2 * 4 * n * f + _lib.mark_bytes(n, 1) + least + GB)
    monkeypatch.setattr(random_forest.tune_cache, "put", lambda *a: None)
    forest._run_autotune("batched", 1)
    assert least <= dev.given[0] <= least + GB


@pytest.mark.parametrize("room_for_all", [True, False])
def test_queue(monkeypatch, room_for_all):
    jobs = [forest_queue._host_job(np.zeros((3000, 200), np.float32), np.arange(3000) % 3, 1, None) for _ in range(4)]
    plans = {k: forest_queue._GroupPlan(jobs[2 * k:2 * k + 2], {}, False) for k in range(2)}
    before = {k: (p.size, p.ws_bytes) for k, p in plans.items()}
    want = sum((p.size + 255) & ~255 for p in plans.values())
    empty = torch.empty

    def counted(n, **kw):
        if n > (want if room_for_all else want - 1):
            raise torch.OutOfMemoryError("counted device is full")
        return empty(n, **kw)

    monkeypatch.setattr(torch, "empty", counted)
    arena, offs = forest_queue._wave_memory(plans, torch.device("cpu"))
    assert offs[0] == 0 and offs[1] >= plans[0].size and arena.numel() >= offs[1] + plans[1].size
    for k, p in plans.items():
        least = _lib.size_of("ct_fit_queue_least_workspace_size", p.arr, 2, C.byref(p.opts))
        assert least < before[k][1]
        assert p.ws_bytes == (before[k][1] if room_for_all else least)
        assert p.size >= p.work + p.ws_bytes
