"""The streaming join probe against the oracle and against the scan engine:
payload bytes and match bits in shared memory, key ranges at and past both
limits, keys outside the build range, no match at all, leaves (one to four,
negated) and a predicate it does not take, ragged row counts, several
build-side keys, alone and in a batch."""
import numpy as np
import pytest

import oracle
from turbogp_b200 import datagen
from turbogp_b200.engine import build_col, col, count_star, sum_

pytestmark = pytest.mark.gpu
CT = {**datagen.LINEITEM_COLTYPES, "fk": "int"}


@pytest.mark.parametrize("n,nb,base", [(1, 5, 1), (127, 40, -20), (128, 40, 1), (100_003, 1_000, 1), (3_000_001, 163_840, 1),
                                       (3_000_001, 163_841, -9), (2_500_003, 1_556_480, 1), (2_500_003, 1_556_481, 1)])
def test_join_shape(ctx, n, nb, base):
    rng = np.random.default_rng(n + nb)
    dim = datagen.dimension(nb, seed=5)
    dim["key"] = (dim["key"] - 1 + base).astype(np.int32)
    fact = datagen.lineitem(n, seed=6)
    fact["price_cents"] -= 4_000_000   # negative products too
    fact["fk"] = rng.integers(base - 3, base + nb + 3, n).astype(np.int32)
    f, d = ctx.register(fact, CT), ctx.register(dim, datagen.DIMENSION_COLTYPES)
    p, disc, q, x = col("price_cents"), col("discount_pct"), col("quantity"), col("tax_pct")
    aggs = [sum_(p * (100 - disc)), count_star()]
    wheres = [None, q < 30, ~(q < 10) & (x >= 2) & (disc != 4) & (col("ship_day") < datagen.DAY0 + 2000)]
    if n < 200_000:
        wheres.append((q < 5) | (x > 6))
    day = datagen.DAY0 + datagen.NDAYS // 2
    for bw in (col("order_day") < day, col("order_day") < 0, None):
        j = d.join_build("key", bw)
        for keys in ((build_col("segment"),), ()):
            outs = [f.aggregate(aggs, keys, w, join=j, probe_key="fk") for w in wheres]
            pqs = [f.prepare(aggs, keys, w, join=j, probe_key="fk") for w in wheres]
            ctx.batch_config(shared_scans=False)
            batched = ctx.submit(pqs).wait()
            ctx.batch_config()
            for w, g, b in zip(wheres, outs, batched):
                o = oracle.aggregate(fact, CT, aggs, keys, w, build=(dim, datagen.DIMENSION_COLTYPES, "key", bw),
                                     probe_key="fk") if n < 200_000 else pqs[0].table.aggregate(
                    aggs + [sum_(q)], keys, w, join=j, probe_key="fk")   # another value program: the scan engine
                for r in (g, b):
                    assert r.rows_selected == o.rows_selected and r.keys == o.keys
                    assert [[(v.value, v.count) for v in row] for row in r.values] == \
                           [[(v.value, v.count) for v in row[:2]] for row in o.values]
        j.drop()
    f.drop()
    d.drop()
