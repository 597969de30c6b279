"""Grouped aggregates over the ranges where their route changes: direct
accumulators formatted on the device, one key in one-word slots below the
direct-accumulator limit, each against the oracle (exact integers)."""
import numpy as np
import pytest

import oracle
from turbogp_b200 import datagen, workloads
from turbogp_b200.engine import Context, avg, col, count_col, count_star, max_, min_, sum_

pytestmark = pytest.mark.gpu

CT = datagen.LINEITEM_COLTYPES


def same(a, b):
    assert a.rows_selected == b.rows_selected
    assert a.keys == b.keys
    for ga, gb in zip(a.values, b.values):
        for x, y in zip(ga, gb):
            assert (x.value, x.count) == (y.value, y.count)
            assert x.as_f64 == y.as_f64 or abs(x.as_f64 - y.as_f64) <= 1e-12 * abs(y.as_f64)


def keyed(n, groups, kmin, dtype, seed):
    rng = np.random.default_rng(seed)
    key = rng.integers(0, groups, n)
    key[: min(n, groups // 2)] = np.arange(min(n, groups // 2))   # most keys occur
    return {"key": (key + kmin).astype(dtype), "v": rng.integers(-900, 1001, n, dtype=np.int32),
            "u": rng.integers(0, 256, n, dtype=np.uint8), "w": rng.integers(-2**33, 2**33, n, dtype=np.int64),
            "big": rng.integers(-2**61, 2**61, n, dtype=np.int64)}


@pytest.mark.parametrize("n,groups,kmin,dtype", [
    (1, 1, 5, np.int32), (4_097, 4_000, -2_000, np.int32), (50_021, 20_011, -7, np.int64),
    (300_007, 400_003, 2**40, np.int64), (100_000, 65_536, 2**31 - 65_536, np.int32),
    (40_000, 3_000_001, 0, np.int32)])
def test_one_key_below_the_direct_limit(ctx, n, groups, kmin, dtype):
    """COUNT(*) with one, none or two values, every value width, with and
    without WHERE: one-word slots where they fit, direct accumulators else."""
    h = keyed(n, groups, kmin, dtype, 3 + n)
    t = ctx.register(h)
    shapes = [[count_star()], [count_star(), sum_(col("v"))], [avg(col("u")), count_star()],
              [count_col(col("u")), count_star()], [sum_(7 - col("v"))],
              [sum_(col("w")), count_star()], [sum_(col("v")), sum_(col("u"))], [min_(col("v")), max_(col("w"))],
              [sum_(col("big") * col("v")), count_star()]]
    for aggs in shapes:
        for where in (None, col("u") < 100, col("v") > 5_000):
            same(t.aggregate(aggs, ("key",), where), oracle.aggregate(h, None, aggs, ("key",), where))
    t.drop()


@pytest.mark.parametrize("n", [0, 1, 2_049, 200_003])
def test_many_direct_groups_of_several_keys(ctx, n):
    """Two and three keys over thousands of direct groups: key tuples, extremes
    and sums formatted on the device; an output buffer that is too small."""
    h = datagen.lineitem(n, seed=5 + n)
    t = ctx.register(h, CT)
    p, q = col("price_cents"), col("quantity")
    aggs = [count_star(), sum_(p), min_(p), max_(q), avg(q)]
    for keys in (("ship_day",), ("flag_a", "ship_day"), ("ship_day", "flag_b", "discount_pct")):
        for where in (None, q < 20):
            same(t.aggregate(aggs, keys, where, group_cap=1), oracle.aggregate(h, CT, aggs, keys, where))
    t.drop()


@pytest.mark.parametrize("n,groups", [(1, 1), (2_047, 300), (2_048, 1_200), (150_001, 2_500), (150_001, 9_001)])
def test_limb_tables_of_sums_and_extremes(ctx, n, groups):
    """One shared table word per extreme and per small sum, two per wide sum:
    negative values, ranges of and past 2^32, joins through a payload, the
    same query forced onto the other placements and captured."""
    h = keyed(n, groups, -17, np.int32, 11 + n)
    h["edge"] = np.where(np.arange(n) % 2 == 0, -2**31, 2**31 - 1).astype(np.int64)   # a range of 2^32 - 1
    t = ctx.register(h)
    v, u, w = col("v"), col("u"), col("w")
    shapes = [[count_star(), min_(v), max_(v)], [min_(100 - v), max_(v * u), sum_(u), count_col(v)],
              [sum_(w), min_(col("edge")), max_(col("edge"))], [min_(w), sum_(v)], [avg(v * u), max_(u), sum_(w * 2)]]
    try:
        for placement in (0, 4, 2, 3):
            ctx.set_default_variant(placement=placement)
            for aggs in shapes:
                for where in (None, (u >= 30) & (v < 500), v > 5_000):
                    same(t.aggregate(aggs, ("key",), where), oracle.aggregate(h, None, aggs, ("key",), where))
    finally:
        ctx.set_default_variant(placement=0)
    pq = t.prepare(shapes[1], ("key",), u < 200, group_cap=16_384)
    if groups < 9_000:
        pq.capture()
    same(pq.run(), oracle.aggregate(h, None, shapes[1], ("key",), u < 200))
    pq.drop_graph()
    same(ctx.submit([pq, t.prepare(shapes[4], ("key",), None, group_cap=16_384)]).wait()[1],
         oracle.aggregate(h, None, shapes[4], ("key",), None))
    t.drop()


def test_autotuner_times_launches_whose_results_are_handed_over():
    """A result handed over by the kernel is read before the launch has
    ended: the tuner waits for the launch before it reads its time."""
    host = datagen.lineitem(400_000, seed=77)
    with Context(0) as ctx:
        t = ctx.register(host, datagen.LINEITEM_COLTYPES)
        for tpl in (workloads.filtered_group_agg(), workloads.selective_scan_sum()):
            rep = ctx.autotune(t.prepare(tpl.aggs, tpl.group_by, tpl.where), reps=3)
            ran = [c for c in rep["candidates"] if c["status"] == 0 and c["same_result"]]
            assert ran and all(c["ms"] > 0 for c in ran)
        t.drop()
