"""The streaming limb tables against the oracle, alone and as merged scans of a
batch: key types and counts, leaves, every value form, row counts around a
chunk, tables and rows past the kernel's conditions (the scan engine runs)."""
import numpy as np
import pytest

import oracle
from turbogp_b200 import datagen, workloads
from turbogp_b200.engine import avg, build_col, col, count_col, count_star, max_, min_, sum_

pytestmark = pytest.mark.gpu
CT = {**datagen.LINEITEM_COLTYPES, "fk": "int"}


def same(a, b):
    assert a.rows_selected == b.rows_selected and a.keys == b.keys
    assert [[(v.value, v.count) for v in r] for r in a.values] == [[(v.value, v.count) for v in r] for r in b.values]


@pytest.mark.parametrize("n", [1, 127, 128, 129, 60_003, 700_001])
def test_value_forms(ctx, n):
    h = datagen.lineitem(n, seed=n)
    h["neg"] = np.random.default_rng(n).integers(-2**31, 2**31, n).astype(np.int32)
    h["wide"] = np.random.default_rng(n + 1).integers(-2**34, 2**34, n)
    t = ctx.register(h, datagen.LINEITEM_COLTYPES)
    p, q, x, w = col("price_cents"), col("quantity"), col("neg"), col("wide")
    d0 = datagen.DAY0
    shapes = [[count_star()], [sum_(p), min_(p), max_(p), avg(q)], [min_(x), max_(3 - x), sum_(x), count_col(col("tax_pct"))],
              [sum_(w), sum_(w - 5), sum_(-p)], [sum_(p), sum_(q), sum_(w), sum_(x)], [min_(w), sum_(p)],
              [sum_(p * (100 - col("discount_pct"))), max_(q)]]
    shapes.append(workloads.filtered_group_agg().aggs)
    wheres = [None, q < 30, ~(q < 10) & (col("tax_pct") >= 2) & (col("discount_pct") != 4) & (col("ship_day") < d0 + 2000),
              (col("flag_a") == 1) & (q < 40)]
    for keys in (("ship_day",), ("quantity", "flag_a"), ("flag_b", "discount_pct", "quantity"),
                 ("flag_a", "flag_b", "tax_pct", "discount_pct")):
        for aggs in shapes if n < 100_000 else shapes[1:4]:
            for where in wheres if n < 100_000 else wheres[1:3]:
                if len(keys) == 4 and where is wheres[2]:
                    continue   # more than the eight columns a query may read
                same(t.aggregate(aggs, keys, where), oracle.aggregate(h, datagen.LINEITEM_COLTYPES, aggs, keys, where))
    t.drop()


@pytest.mark.parametrize("n,nb", [(129, 30), (40_001, 700), (400_003, 170_000)])
def test_merged_scans(ctx, n, nb):
    """Batches of same-shape requests (bucket keys, rows no request accepts,
    the join's count scan) against the same requests alone."""
    dim, fact = datagen.dimension(nb, seed=4), datagen.fact_fk(n, nb, 0.8, seed=5)
    fact["fk"][::97] = nb + 5
    f, d = ctx.register(fact, CT), ctx.register(dim, datagen.DIMENSION_COLTYPES)
    j = d.join_build("key", col("order_day") < datagen.DAY0 + datagen.NDAYS // 2)
    rng = np.random.default_rng(n)
    tj = workloads.join_group_agg()
    specs = []
    for i in range(14):
        lo, disc = int(rng.integers(0, 2000)), int(rng.integers(0, 9))
        s = workloads.selective_scan_sum(datagen.DAY0 + lo, int(rng.integers(1, 400)), disc, disc + 2, int(rng.integers(2, 50)))
        specs.append((s.aggs, s.group_by, s.where, None, None))
        q = workloads.filtered_group_agg(datagen.DAY0 + int(rng.integers(0, 2600)))
        specs.append((q.aggs, q.group_by, q.where, None, None))
        specs.append((tj.aggs, tj.group_by, col("quantity") < int(rng.integers(1, 52)), j, "fk"))
    pqs = [f.prepare(a, g, w, join=jj, probe_key=k) for a, g, w, jj, k in specs]
    for got, (a, g, w, jj, k) in zip(ctx.submit(pqs).wait(), specs):
        build = (dim, datagen.DIMENSION_COLTYPES, "key", col("order_day") < datagen.DAY0 + datagen.NDAYS // 2) if jj else None
        same(got, oracle.aggregate(fact, CT, a, g, w, build=build, probe_key=k))
    j.drop()
    f.drop()
    d.drop()
