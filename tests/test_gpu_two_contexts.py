"""Two contexts on two threads launch the same kernel with different amounts of
shared memory at the same time: the streaming joins, limb tables, hash groups and
Q1. Every call succeeds with the result it has alone."""
import threading
import time

import numpy as np
import pytest

from turbogp_b200 import datagen, workloads
from turbogp_b200.engine import Context, build_col, col, count_star, sum_

pytestmark = pytest.mark.gpu
CT = {**datagen.LINEITEM_COLTYPES, "fk": "int"}


def raw(pq):
    r = pq.run(decode=False)
    n = int(pq.res.ngroups)
    return r.rows_selected, n, pq.keys[:n * pq.nk].tobytes(), pq._vals_np[:n * pq.na].tobytes()


def join(c, big):
    """A payload of 160,000 bytes, or of 40."""
    n, nb = (1_700_000, 160_000) if big else (30_000, 40)
    dim, fact = datagen.dimension(nb, seed=1), datagen.lineitem(n, seed=2)
    fact["fk"] = np.random.default_rng(3).integers(1, nb + 1, n).astype(np.int32)
    f, d = c.register(fact, CT), c.register(dim, datagen.DIMENSION_COLTYPES)
    return f.prepare([sum_(col("price_cents") * (100 - col("discount_pct"))), count_star()], (build_col("segment"),), None,
                     join=d.join_build("key"), probe_key="fk")


def limbs(c, big):
    """2,526 groups, or 50."""
    t = c.register(datagen.lineitem(1_200_000 if big else 30_000, seed=4), datagen.LINEITEM_COLTYPES)
    p, q = col("price_cents"), col("discount_pct")
    return t.prepare([sum_(p), sum_(q), count_star()], ("ship_day",) if big else ("quantity", "tax_pct"), None)


def sparse(c, big):
    """Hash slots with a shared table, or with values too large for one."""
    n, rng = 200_000, np.random.default_rng(5)
    ids = rng.integers(0, 2**60, 500)
    v = rng.integers(0, 100 if big else 2**26, n).astype(np.int32)
    t = c.register({"id": ids[rng.integers(0, 500, n)], "v": v}, {"id": "int", "v": "int"})
    return t.prepare([sum_(col("v")), count_star()], ("id",), None)


def flags(c, big):
    """The Q1 shape over 6 groups, or over 2."""
    h = datagen.lineitem(50_000, seed=6)
    if not big:
        h["flag_a"] = np.zeros_like(h["flag_a"])
    q = workloads.filtered_group_agg()
    return c.register(h, datagen.LINEITEM_COLTYPES).prepare(q.aggs, q.group_by, q.where)


@pytest.mark.parametrize("make", [join, limbs, sparse, flags])
def test_same_kernel_at_two_sizes(ctx, make):
    with Context(0) as second:
        queries = [make(ctx, True), make(second, False)]
        want = [raw(pq) for pq in queries]
        end, bad = time.monotonic() + 4.0, []

        def work(i):
            try:
                while time.monotonic() < end and not bad:
                    if raw(queries[i]) != want[i]:
                        bad.append((i, "another result"))
            except Exception as e:
                bad.append((i, str(e)))
        ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
        [t.start() for t in ts]
        [t.join() for t in ts]
        assert not bad
