"""When a large result gets a page-locked buffer, on the CPU with the locking
counted: never for results that are kept or larger than the pool keeps idle,
once for results that are dropped, whatever else lies idle."""
import gc
import threading

import numpy as np
import pytest

from turbogp_b200 import engine

MB = 1 << 20


@pytest.fixture
def pool(monkeypatch):
    p = engine._PinnedPool()
    p.locked, p.unlocked = [], []

    def register(size):
        p.locked.append(size)
        return np.empty(size, dtype=np.uint8)
    monkeypatch.setattr(p, "_register", register, raising=False)
    monkeypatch.setattr(p, "_unregister", lambda buf: p.unlocked.append(buf.nbytes), raising=False)
    monkeypatch.setattr(engine, "_PINNED", p)
    return p


def array(nbytes):
    return engine._result_array(nbytes // 4, np.uint32)


def test_kept_results_lock_nothing(pool):
    kept = [array(12 * MB) for _ in range(20)]
    assert pool.locked == [] and len({a.ctypes.data for a in kept}) == 20


def test_dropped_results_lock_once(pool):
    for _ in range(20):
        array(12 * MB)
    assert pool.locked == [12 * MB] and pool.unlocked == []
    keep = [array(12 * MB) for _ in range(20)]   # the one buffer, then ordinary arrays
    assert pool.locked == [12 * MB]
    del keep
    assert pool._bytes == pool._idle_bytes == 12 * MB


def test_a_window_of_kept_results_ends_on_locked_buffers(pool):
    window = []
    for _ in range(40):
        window.append(array(8 * MB))
        del window[:-4]
    assert pool.locked == [8 * MB] * 5 and pool.unlocked == []


@pytest.mark.parametrize("nbytes", [256 * MB + 4, 400 * MB])
def test_results_above_the_idle_bound_are_ordinary(pool, nbytes):
    for _ in range(4):
        array(nbytes)
    assert pool.locked == [] and pool._bytes == 0 and not pool._dropped


def test_small_idle_buffers_make_room(pool):
    held = [pool.take(16 * MB) for _ in range(16)]
    del held
    assert pool._idle_bytes == pool.KEEP
    for _ in range(6):
        array(48 * MB)
    assert pool.locked[16:] == [48 * MB]         # locked once although the bound was reached
    assert pool.unlocked == [16 * MB] * 3 and pool._idle_bytes <= pool.KEEP


def test_idle_buffers_make_room_below_the_limit(pool):
    held = [pool.take(192 * MB) for _ in range(5)]
    held.pop()
    assert pool._bytes == 960 * MB and pool._idle_bytes == 192 * MB
    assert pool.take(128 * MB) is not None       # 1,088 MB with the idle one
    assert pool.unlocked == [192 * MB]


@pytest.mark.parametrize("nbytes", [MB, MB + 1, 3 * MB, 5 * MB + 17, 130 * MB, 256 * MB - 1, 256 * MB])
def test_buffers_waste_at_most_a_quarter(pool, nbytes):
    size = pool._size(nbytes)
    assert nbytes <= size <= nbytes * 1.25 and pool._size(size) == size


def test_release_gives_the_idle_buffers_back(pool):
    held = pool.take(4 * MB)
    for _ in range(3):
        array(12 * MB)
    pool.take(2 * MB)
    assert pool._idle_bytes == 14 * MB
    pool.release()
    assert sorted(pool.unlocked) == [2 * MB, 12 * MB] and pool._idle_bytes == 0 and pool._bytes == 4 * MB
    del held
    assert pool._bytes == pool._idle_bytes == 4 * MB      # on loan meanwhile: idle now


@pytest.mark.gpu
def test_a_closed_context_keeps_no_idle_buffer():
    with engine.Context(0) as ctx:
        t = ctx.register({"k": np.zeros(4_000_000, dtype=np.int32)}, {"k": "int"})
        for _ in range(4):
            assert t.filter(engine.col("k") < 1).count == 4_000_000
        assert engine._PINNED._idle_bytes >= 16_000_000
    assert engine._PINNED._idle_bytes == 0


def test_arrays_dropped_by_a_collection_at_any_point(pool):
    """Arrays in reference cycles come back while take() runs, on every thread:
    no buffer is lost, none is handed out twice."""
    class Node:
        def __init__(self, a):
            self.a, self.me = a, self

    stop, bad = threading.Event(), []

    def work(seed):
        rng = np.random.default_rng(seed)
        while not stop.is_set():
            a = pool.take(int(rng.integers(1, 9)) * MB)
            if a is None:
                gc.collect()
                continue
            a[:8] = seed
            Node(a)
            if not (a[:8] == seed).all():
                bad.append(seed)
    old = gc.get_threshold()
    gc.set_threshold(5)
    try:
        ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
        [t.start() for t in ts]
        stop.wait(3)
        stop.set()
        [t.join() for t in ts]
    finally:
        gc.set_threshold(*old)
    gc.collect()
    idle = [b for free in pool._idle.values() for b in free]
    assert not bad and not pool._returned
    assert pool._bytes == pool._idle_bytes == sum(b.nbytes for b in idle) <= pool.KEEP
    assert sorted(pool.locked) == sorted(pool.unlocked + [b.nbytes for b in idle])
