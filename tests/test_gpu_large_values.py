"""Sums of values near 2^62, of which an int64 partial holds one to twelve: every
accumulator placement, value program and launch form against the oracle, at row
counts of whole tiles (a thread's rows of a tile are added together) and around."""
import numpy as np
import pytest

import oracle
from turbogp_b200.engine import Context, col, count_col, count_star, sum_

pytestmark = pytest.mark.gpu
CT = {"big": "int", "x": "int", "k": "int", "k2": "int"}
DEFAULT = dict(threads=0, max_stages=8, placement=0, presum=1, dense=1, shapes=1, payload=1)


def values(r):
    return r.rows_selected, r.keys, [[(v.value, v.count) for v in row] for row in r.values]


@pytest.mark.parametrize("knobs", [{}, {"dense": 0}, {"threads": 256}, {"placement": 2}, {"placement": 4}])
@pytest.mark.parametrize("top", [2**59 + 2**57, 2**60 - 1, 2**60 + 2**59, 2**61, 2**62 - 1])
def test_sums_are_exact(top, knobs):
    with Context(0) as ctx:
        ctx.set_default_variant(**{**DEFAULT, **knobs})
        for n in (100, 2048, 10_241, 700_000):
            rng = np.random.default_rng(n)
            h = {"big": top - rng.integers(0, 5, n), "x": rng.integers(-9, 9, n).astype(np.int32),
                 "k": rng.integers(0, 5, n).astype(np.uint8), "k2": rng.integers(0, 900, n).astype(np.int32)}
            t = ctx.register(h, CT)
            for big in (col("big"), -col("big")):
                for aggs in ([sum_(big)], [sum_(3 - col("x")), sum_(big), count_col(col("x"))],
                             [sum_(big), count_star()]):
                    for keys in ((), ("k",), ("k2",)):
                        for where in (None, col("x") < 5):
                            want = values(oracle.aggregate(h, CT, aggs, keys, where))
                            pq = t.prepare(aggs, keys, where)
                            assert values(pq.run()) == want
                            assert values(ctx.submit([pq]).wait()[0]) == want
                            captured = t.prepare(aggs, keys, where).capture()
                            assert values(captured.run()) == want
                            captured.drop_graph()
            t.drop()
