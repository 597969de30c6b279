"""A filter whose row-id scratch cannot be had fails as out of memory with its
bitmap complete: no copy into the caller's memory is under way once it has
returned. The device memory is taken by another allocation, in a process of its
own."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes as C
import numpy as np
import torch
from turbogp_b200 import _capi as A
from turbogp_b200.engine import Context, col
n = 64_000_003
k = (np.arange(n, dtype=np.int64) * 2_654_435_761 % 1000).astype(np.int32)
with Context(0) as ctx:
    t = ctx.register({"k": k}, {"k": "int"})
    assert len(t.filter(col("k") < 1).rowids) == (k < 1).sum()      # scratch and kernels are there
    nodes, m = t.lower_pred(col("k") < 900)
    bitmap = np.zeros((n + 7) // 8, dtype=np.uint8)
    assert ctx.lib.tgp_host_lock(bitmap.ctypes.data, bitmap.nbytes) == A.OK
    ids = np.empty(n, dtype=np.uint32)
    alloc = A.AllocFn(lambda user, count: ids.ctypes.data)
    count = C.c_uint64()
    call = lambda: ctx.lib.tgp_filter_alloc(ctx.h, t.id, nodes, m, bitmap.ctypes.data, alloc, None, C.byref(count))
    taken, step = [], 1 << 36
    while step >= 16 << 20:                                          # 230 MB of row ids no longer fit
        try:
            taken.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            step >>= 1
    assert call() == A.OOM
    want = np.packbits(k < 900, bitorder="little")
    assert np.array_equal(bitmap, want) and count.value == (k < 900).sum()
    del taken
    torch.cuda.empty_cache()
    bitmap[:] = 0
    assert call() == A.OK
    assert np.array_equal(bitmap, want) and np.array_equal(ids[:count.value], np.flatnonzero(k < 900))
    assert ctx.lib.tgp_host_unlock(bitmap.ctypes.data) == A.OK
print("ok")
"""


def test_no_copy_outlives_the_call():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True)
    assert r.stdout.strip() == "ok", r.stderr[-2000:]
