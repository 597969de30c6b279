"""Large result arrays when page-locking fails: an ordinary array serves, and the
pool's account is as before."""
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from turbogp_b200 import engine


@pytest.mark.parametrize("error", [ImportError, MemoryError, OSError, None])
def test_a_failed_lock_gives_an_ordinary_array(monkeypatch, error):
    def register(size):
        if error:
            raise error("no page-locked memory")
        return None
    pool = engine._PinnedPool()
    monkeypatch.setattr(pool, "_register", register, raising=False)
    monkeypatch.setattr(engine, "_PINNED", pool)
    for _ in range(3):
        assert pool.take(3 << 20) is None
        a = engine._result_array(1 << 20, np.uint32)
        assert a.shape == (1 << 20,) and a.dtype == np.uint32 and a.flags.writeable
    assert pool._bytes == pool._idle_bytes == 0


@pytest.mark.parametrize("error", [MemoryError, KeyboardInterrupt])
def test_an_error_while_the_result_is_allocated_is_raised_as_itself(monkeypatch, error):
    def no_array(n, dtype):
        raise error("no room")

    def call(alloc):
        if alloc(None, 5) is None:
            raise engine.A.TgpError(engine.A.OOM, "row-id buffer allocation failed")
    monkeypatch.setattr(engine, "_result_array", no_array)
    with pytest.raises(error, match="no room"):
        engine._result_words(call)


PROGRAM = """
import sys
sys.modules["torch"] = None      # not installed
import numpy as np
from turbogp_b200.engine import Context, col
with Context(0) as ctx:
    n = 9_000_001
    h = {"k": (np.arange(n) % 5).astype(np.int32)}
    t = ctx.register(h, {"k": "int"})
    for _ in range(4):
        r = t.filter(col("k") < 4)
        assert np.array_equal(r.rowids, np.flatnonzero(h["k"] < 4).astype(np.uint32))
        assert np.array_equal(np.unpackbits(r.bitmap, bitorder="little")[:n], h["k"] < 4)
    j = ctx.register({"k": np.array([2], dtype=np.int32)}, {"k": "int"}).join_build("k")
    p, b = j.probe_pairs(t, "k")
    assert np.array_equal(p, np.flatnonzero(h["k"] == 2)) and not b.any()
print("ok")
"""


@pytest.mark.gpu
def test_large_results_need_no_torch():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True)
    assert r.stdout.strip() == "ok", r.stderr[-2000:]
