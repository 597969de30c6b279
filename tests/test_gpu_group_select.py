"""ORDER BY aggregate LIMIT n by selection, and group tables sized from a key
sketch, against the oracle's groups sorted whole: ties at the cut, every
ordering kind and direction, limits at and past the selection's, all groups
equal, few groups, sparse and direct keys, tables past the sketch's size."""
import numpy as np
import pytest

import oracle
from turbogp_b200 import _capi as A
from turbogp_b200.engine import avg, col, count_col, count_star, max_, min_, sum_

pytestmark = pytest.mark.gpu


def order_of(o, i, desc):
    """The oracle's groups in the wanted order (ties in key order)."""
    rows = list(zip(o.keys, o.values))
    value = (lambda r: r[1][i].as_f64) if o.is_avg[i] else (lambda r: r[1][i].value)
    return sorted(rows, key=lambda r: (-value(r) if desc else value(r), r[0]))


def check(t, h, aggs, keys, where, limits=(1, 3, 1000, 1024, 1025, 4000)):
    o = oracle.aggregate(h, None, aggs, keys, where)
    o.is_avg = [a.func == A.AGG_AVG for a in aggs]
    for i in range(len(aggs)):
        for desc in (True, False):
            want = order_of(o, i, desc)
            for limit in limits:
                g = t.aggregate_topn(aggs, keys, where, i, desc, limit)
                assert g.keys == [k for k, _ in want[:limit]], (i, desc, limit)
                assert [[(v.value, v.count) for v in r] for r in g.values] == \
                       [[(v.value, v.count) for v in r] for _, r in want[:limit]]


def table(n, groups, kind, seed):
    rng = np.random.default_rng(seed)
    ids = {"sparse": rng.integers(0, 1 << 62, groups), "dense": np.arange(groups) * 3 - 50,
           "pairs": rng.integers(0, 1 << 30, groups)}[kind]
    pick = np.minimum(rng.zipf(1.3, n) - 1, groups - 1) if groups > 1 else np.zeros(n, dtype=np.int64)
    pick[: min(n, groups)] = np.arange(min(n, groups))
    return {"id": ids[pick].astype(np.int64), "sub": rng.integers(0, 5, n, dtype=np.uint8),
            "v": rng.integers(-1000, 1001, n, dtype=np.int32), "w": rng.integers(-2**40, 2**40, n, dtype=np.int64)}


@pytest.mark.parametrize("n,groups,kind", [(0, 1, "sparse"), (1, 1, "sparse"), (40_003, 31, "sparse"),
                                           (60_001, 30_000, "sparse"), (50_000, 6_000, "dense"), (30_000, 3_000, "pairs")])
def test_top_n_by_selection(ctx, n, groups, kind):
    h = table(n, groups, kind, 3 + n)
    t = ctx.register(h)
    keys = ("id", "sub") if kind == "pairs" else ("id",)
    for where in (None, col("v") >= 0):
        check(t, h, [count_star(), sum_(col("v")), min_(col("w")), avg(col("v")), max_(col("v"))], keys, where)
    t.drop()


def test_every_ordering_value_equal(ctx):
    """All ties: the keys alone decide, through several narrowings."""
    rng = np.random.default_rng(9)
    h = {"id": rng.permutation(rng.integers(0, 1 << 61, 50_000)), "v": np.full(50_000, 7, dtype=np.int32)}
    t = ctx.register(h)
    check(t, h, [count_star(), sum_(col("v")), count_col(col("v"))], ("id",), None, limits=(1, 10, 1024))
    t.drop()


@pytest.mark.parametrize("distinct", [40, 70_000, 1_500_000])
def test_group_tables_sized_from_a_sketch(ctx, distinct):
    """More rows than a table of every row's slot may take without the sketch:
    full results and top-N against numpy (exact)."""
    n = 1_600_003
    rng = np.random.default_rng(distinct)
    ids = np.unique(rng.integers(-2**61, 2**61, distinct))
    pick = rng.integers(0, ids.size, n)
    pick[: ids.size] = np.arange(ids.size)
    h = {"id": ids[pick], "v": rng.integers(0, 1000, n, dtype=np.int32), "u": rng.integers(0, 3, n, dtype=np.uint8)}
    t = ctx.register(h)
    q = t.prepare([count_star(), sum_(col("v"))], ("id",), col("u") < 2, group_cap=n)
    k, lo, _, cnt = q.run().arrays()
    m = h["u"] < 2
    wc = np.bincount(pick[m], minlength=ids.size)
    ws = np.bincount(pick[m], weights=h["v"][m], minlength=ids.size).astype(np.int64)
    some = wc > 0
    assert np.array_equal(k[:, 0], ids[some]) and np.array_equal(cnt[:, 0], wc[some].astype(np.uint64))
    assert np.array_equal(lo[:, 1].view(np.int64), ws[some])
    g = t.aggregate_topn([count_star(), sum_(col("v"))], ("id",), col("u") < 2, 1, True, 20)
    best = np.argsort(-ws[some], kind="stable")[:20]
    assert [x[0] for x in g.keys] == ids[some][best].tolist()
    t.drop()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 70_001])
def test_sparse_key_streaming_forms(ctx, n):
    """The streaming kernel of one sparse key: key and value types, no value,
    COUNT(col), affine arguments, one to four leaves and negated ones, values
    too wide for the shared table, leaves it does not take (u8, OR)."""
    rng = np.random.default_rng(n)
    ids = rng.integers(-2**62, 2**62, max(1, n // 3))
    pick = rng.integers(0, ids.size, n)
    h = {"id": ids[pick], "i32": (ids[pick] >> 32).astype(np.int32), "v": rng.integers(-1000, 1001, n, dtype=np.int32),
         "u": rng.integers(0, 256, n, dtype=np.uint8), "w": rng.integers(-2**38, 2**38, n, dtype=np.int64),
         "a": rng.integers(0, 50, n, dtype=np.int32), "b": rng.integers(0, 50, n, dtype=np.int32)}
    t = ctx.register(h)
    a, b, v, u = col("a"), col("b"), col("v"), col("u")
    for key in ("id", "i32"):
        for aggs in ([count_star()], [sum_(v), count_star()], [avg(7 - v)], [count_col(u)], [sum_(col("w"))]):
            for where in (None, a < 30, ~(a < 10) & (b >= 5) & (v > -900) & (a != 33), (u < 200) & (a < 40),
                          (a < 5) | (b < 5)):
                g, o = t.aggregate(aggs, (key,), where), oracle.aggregate(h, None, aggs, (key,), where)
                assert g.rows_selected == o.rows_selected and g.keys == o.keys
                assert [[(x.value, x.count) for x in r] for r in g.values] == \
                       [[(x.value, x.count) for x in r] for r in o.values]
    t.drop()
