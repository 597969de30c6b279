"""The page-locked buffers behind large result arrays, on the CPU: lifetime
through views, bounds, and threads (locking itself is replaced)."""
import threading

import numpy as np
import pytest

from turbogp_b200 import engine


@pytest.fixture
def pool(monkeypatch):
    p = engine._PinnedPool()
    monkeypatch.setattr(p, "_register", lambda size: np.empty(size, dtype=np.uint8), raising=False)
    p.unlocked = []
    monkeypatch.setattr(p, "_unregister", lambda buf: p.unlocked.append(buf.nbytes), raising=False)
    return p


def test_a_buffer_serves_again_once_every_view_is_gone(pool):
    a = pool.take(3 << 20)
    addr, view = a.ctypes.data, a[100:200].view(np.uint32)
    del a
    assert pool.take(3 << 20).ctypes.data != addr   # the view still holds it
    del view
    seen = {pool.take(3 << 20).ctypes.data for _ in range(2)}
    assert addr in {pool.take(1 + (2 << 20)).ctypes.data for _ in range(2)} | seen


def test_bounds(pool):
    held = [pool.take(256 << 20) for _ in range(5)]
    assert [x is None for x in held] == [False] * 4 + [True]      # LIMIT
    del held
    assert pool._idle_bytes == pool.KEEP and pool._bytes == pool.KEEP
    assert pool.unlocked == [256 << 20] * 3


def test_threads_share_it(pool):
    def work():
        for i in range(200):
            x = pool.take((1 << 20) + i)
            x[:8] = i % 251
            assert (x[:8] == i % 251).all()
    ts = [threading.Thread(target=work) for _ in range(8)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert pool._bytes == pool._idle_bytes <= 8 * (2 << 20)


@pytest.mark.parametrize("n", [0, 1, 100])
def test_result_words(n):
    def call(alloc):
        if n:
            np.ctypeslib.as_array((engine.C.c_uint32 * n).from_address(alloc(None, n)))[:] = np.arange(n)
    assert np.array_equal(engine._result_words(call), np.arange(n, dtype=np.uint32))
