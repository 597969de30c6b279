"""The autotuner reports what its candidates launched: the CTA size and stages of
the scan engine, as the size rule for scalar scans sets them, and the streaming
kernels' own (no stages)."""
import pytest

from turbogp_b200 import datagen, workloads
from turbogp_b200.engine import col, count_star, max_, sum_

pytestmark = pytest.mark.gpu
CT = {**datagen.LINEITEM_COLTYPES, "fk": "int"}


def candidates(ctx, pq):
    return [c for c in ctx.autotune(pq, reps=1)["candidates"] if c["status"] == 0]


@pytest.mark.parametrize("rows,threads", [(500_000, 512), (3_000_000, 256)])
def test_scalar_scan(ctx, rows, threads):
    t = ctx.register(datagen.lineitem(rows, seed=1), datagen.LINEITEM_COLTYPES)
    q = workloads.selective_scan_sum()
    cands = candidates(ctx, t.prepare(q.aggs, q.group_by, q.where))
    rule = cands[0]
    assert rule["threads"] == threads and rule["stages"] == (5 if threads == 512 else 2)   # 40 KB a stage
    for c in cands[1:]:
        if c["variant"]["threads"] and c["mode"] == rule["mode"]:
            assert c["threads"] == c["variant"]["threads"] and c["stages"] >= 1
    t.drop()


def test_streaming_kernels(ctx):
    fact, dim = datagen.fact_fk(400_000, 1_000, 0.8, seed=2), datagen.dimension(1_000, seed=3)
    f, d = ctx.register(fact, CT), ctx.register(dim, datagen.DIMENSION_COLTYPES)
    j = d.join_build("key")
    p = col("price_cents")
    tj, q1 = workloads.join_group_agg(), workloads.filtered_group_agg()
    for pq, threads in ((f.prepare(tj.aggs, tj.group_by, None, join=j, probe_key="fk"), 1024),
                        (f.prepare([sum_(p), max_(p), count_star()], ("ship_day",)), 1024),
                        (f.prepare(q1.aggs, q1.group_by, q1.where), 512)):
        assert (candidates(ctx, pq)[0]["threads"], candidates(ctx, pq)[0]["stages"]) == (threads, 0)
    j.drop()
    f.drop()
    d.drop()
