"""Results handed over by the kernel: blocks of a few words up to the largest
that is handed over, from every kernel that does it, in turn on one context and
on two contexts at once. Each result is compared whole with the first one, and
that one with the oracle: a word that arrived late or was left from another
query shows."""
import threading

import numpy as np
import pytest

import oracle
from turbogp_b200 import datagen, workloads
from turbogp_b200.engine import Context, col, count_star, max_, min_, sum_

pytestmark = pytest.mark.gpu
ROUNDS = 150


def prepared(c, h, dim):
    f, d = c.register(h, {**datagen.LINEITEM_COLTYPES, "fk": "int"}), c.register(dim, datagen.DIMENSION_COLTYPES)
    j = d.join_build("key")
    build = (dim, datagen.DIMENSION_COLTYPES, "key", None)
    scan, q1, tj = workloads.selective_scan_sum(), workloads.filtered_group_agg(), workloads.join_group_agg()
    p, q = col("price_cents"), col("quantity")
    forms = [(scan.aggs, scan.group_by, scan.where, None), (q1.aggs, q1.group_by, q1.where, None),
             ([sum_(p), min_(p), max_(p), count_star()], ("ship_day",), q < 40, None),
             ([count_star()], ("quantity",), None, None), (tj.aggs, tj.group_by, None, j)]
    return [(f.prepare(a, k, w, join=jj, probe_key="fk" if jj else None), (a, k, w, build if jj else None))
            for a, k, w, jj in forms]


def raw(pq):
    r = pq.run(decode=False)
    n = int(pq.res.ngroups)
    return r.rows_selected, n, pq.keys[:n * pq.nk].tobytes(), pq._vals_np[:n * pq.na].tobytes()


def test_every_word_arrives(ctx):
    h, dim = datagen.fact_fk(200_003, 900, 0.8, seed=3), datagen.dimension(900, seed=4)
    with Context(0) as second:
        sets = [prepared(ctx, h, dim), prepared(second, h, dim)]
        first = []
        for pq, (a, k, w, build) in sets[0]:
            o = oracle.aggregate(h, {**datagen.LINEITEM_COLTYPES, "fk": "int"}, a, k, w, build=build,
                                 probe_key="fk" if build else None)
            g = pq.run()
            assert g.rows_selected == o.rows_selected and g.keys == o.keys
            assert [[(v.value, v.count) for v in r] for r in g.values] == [[(v.value, v.count) for v in r] for r in o.values]
            first.append(raw(pq))
        bad = []

        def work(queries, seed):
            for i in np.random.default_rng(seed).integers(0, len(queries), ROUNDS * len(queries)):
                if raw(queries[i][0]) != first[i]:
                    bad.append(int(i))
        ts = [threading.Thread(target=work, args=(s, k)) for k, s in enumerate(sets)]
        [t.start() for t in ts]
        [t.join() for t in ts]
        assert not bad
