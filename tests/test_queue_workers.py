"""Worker threads of the forest queue (CPU): who gets which, how many are kept,
and that a call leaves no thread behind that still uses its buffers."""
import threading
import time

import pytest

from cudatree_b200 import forest_queue as Q


@pytest.fixture(autouse=True)
def no_idle_workers():
    Q._IDLE.clear()
    yield
    for idle in Q._IDLE.values():
        for w in idle:
            w.close()
    Q._IDLE.clear()


def test_a_caller_alone_gets_the_same_workers():
    a = Q._take_workers(0, 3)
    Q._give_back(0, a)
    assert Q._take_workers(0, 3) == a
    Q._give_back(0, a[::-1])
    assert Q._take_workers(0, 2) == a[:2]
    Q._give_back(0, a[:2])


def test_callers_and_devices_share_no_worker():
    a, b, c = Q._take_workers(0, 4), Q._take_workers(0, 4), Q._take_workers(1, 4)
    assert len({id(w) for w in a + b + c}) == 12
    Q._give_back(0, a)
    Q._give_back(1, c)
    assert all(w not in a for w in Q._take_workers(1, 4))
    Q._give_back(0, b)


def test_kept_workers_are_bounded():
    Q._give_back(0, Q._take_workers(0, Q.IDLE_WORKERS + 5))
    assert len(Q._IDLE[0]) == Q.IDLE_WORKERS


def test_two_callers_run_side_by_side():
    """Each caller's group waits for the other's: with shared threads they would time out."""
    met = threading.Barrier(2, timeout=20)

    def caller():
        w = Q._take_workers(0, 1)
        try:
            Q._run_all(w, lambda worker, item: met.wait(), [0])
        finally:
            Q._give_back(0, w)

    other = threading.Thread(target=caller)
    other.start()
    caller()
    other.join()
    assert not met.broken


@pytest.mark.parametrize("what", ["interrupt", "group fails"])
def test_run_all_returns_when_every_thread_has_ended(monkeypatch, what):
    ended = []

    def group(worker, item):
        if item == 0 and what == "group fails":
            raise ValueError("group 0")
        time.sleep(0.3)
        ended.append(item)

    if what == "interrupt":
        wait, calls = Q.wait, []

        def interrupted(work):
            calls.append(1)
            if len(calls) == 1:
                raise KeyboardInterrupt
            return wait(work)

        monkeypatch.setattr(Q, "wait", interrupted)
    w = Q._take_workers(0, 3)
    with pytest.raises(KeyboardInterrupt if what == "interrupt" else ValueError):
        Q._run_all(w, group, [0, 1, 2])
    assert sorted(ended) == ([0, 1, 2] if what == "interrupt" else [1, 2])
    Q._give_back(0, w)
