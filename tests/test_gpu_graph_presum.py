"""A captured GROUP BY of many groups keeps the shared pre-aggregation only where
its 32-bit partials hold a CTA's rows, as the same query does when it is executed:
values at which they do and at which they do not."""
import numpy as np
import pytest

import oracle
from turbogp_b200.engine import avg, col, count_star, sum_

pytestmark = pytest.mark.gpu
CT = {"a": "int", "b": "int", "v": "int"}


@pytest.mark.parametrize("top", [100, 2**31 // 2048 - 1, 2**31 // 2048, 2**31 - 1])
@pytest.mark.parametrize("n", [1_397, 2_048, 400_000])
def test_captured_global_groups(ctx, n, top):
    rng = np.random.default_rng(n)
    h = {"a": rng.integers(0, 900, n).astype(np.int32), "b": rng.integers(0, 1_500, n).astype(np.int32),
         "v": (top - rng.integers(0, 3, n)).astype(np.int32)}
    h["a"][: n - 5], h["b"][: n - 5] = 7, 9        # one group with nearly every row, 1.3M possible ones
    h["a"][0], h["b"][0] = 899, 1_499
    t = ctx.register(h, CT)
    for aggs in ([sum_(col("v")), count_star()], [avg(col("v") + 70), sum_(-col("v"))]):
        o = oracle.aggregate(h, CT, aggs, ("a", "b"), None)
        want = o.keys, [[(v.value, v.count) for v in r] for r in o.values]
        for pq in (t.prepare(aggs, ("a", "b")), t.prepare(aggs, ("a", "b")).capture()):
            g = pq.run()
            assert (g.keys, [[(v.value, v.count) for v in r] for r in g.values]) == want
            if pq.graph:
                pq.drop_graph()
    t.drop()
