"""The memory figure behind group and batch sizes does not move with the caching
allocator: what a call's buffers leave in the cache still counts (CPU, with
the allocator's figures replaced)."""
import pytest
import torch

from cudatree_b200 import forest_queue, random_forest

GB = 1 << 30


def _device_with(monkeypatch, free, reserved, allocated):
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (free, 180 * GB))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda *a: reserved)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda *a: allocated)


@pytest.mark.parametrize("cached", [0, 7 * GB, 81 * GB])
def test_cached_memory_counts_as_free(monkeypatch, cached):
    held = 3 * GB  # tensors of the caller, in use
    _device_with(monkeypatch, 170 * GB - cached, held + cached, held)
    assert random_forest.free_bytes(torch.device("cuda", 0)) == 170 * GB
    assert forest_queue.free_bytes is random_forest.free_bytes


def test_trees_in_flight_do_not_change_with_the_cache(monkeypatch):
    """A forest of more than half of the device: a repeated fit is cut as the first was."""
    forest = random_forest.RandomForestClassifier(100, max_features=10, seed=1)
    forest.n_samples, forest.n_features, forest.n_labels = 2_000_000, 100, 2
    forest.index_bytes, forest._m, forest._seed = 4, 10, 1
    forest.dtype_labels = torch.empty(0, dtype=torch.uint8).numpy().dtype
    forest._x_fm = forest._labels = forest._presort = torch.empty(1)
    monkeypatch.setattr(random_forest, "_device", lambda: torch.device("cuda", 0))
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda *a: type("P", (), {"total_memory": 180 * GB}))
    got = []
    for cached in (0, 100 * GB):
        _device_with(monkeypatch, 170 * GB - cached, cached, 0)
        got.append(forest.trees_in_flight("batched"))
    assert got[0] == got[1] and 1 < got[0] < 100
