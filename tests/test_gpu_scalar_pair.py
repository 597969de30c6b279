"""Scalar aggregates over many tiles run as two CTAs of 256 threads per SM: the
row counts on both sides of that line, ragged last tiles, stage sizes from one
narrow column (eight stages) to five columns, one and two sums; every result
equals the one of a variant that names its threads (the single-CTA launch) and
the oracle's, whole numbers bit for bit."""
import pytest

import oracle
from turbogp_b200 import datagen
from turbogp_b200.engine import Context, col, count_star, sum_

pytestmark = pytest.mark.gpu

CT = datagen.LINEITEM_COLTYPES
LINE = 4 * 2 * 148 * 2048   # rows of four tiles per CTA, two CTAs per SM

QUERIES = [
    ([sum_(col("quantity"))], None),
    ([sum_(col("price_cents") * col("discount_pct")), count_star()],
     (col("ship_day") >= 9000) & (col("discount_pct") < 7) & (col("quantity") < 24)),
    ([sum_(col("price_cents")), sum_(col("quantity") * col("tax_pct"))], col("discount_pct") > 6),
]


@pytest.fixture(scope="module")
def ctx():
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("rows", [LINE - 2048, LINE - 2047, LINE + 1, 2 * LINE + 1777])
def test_scalar_pair(ctx, rows):
    host = datagen.lineitem(rows, seed=rows % 1000)
    t = ctx.register(host, CT)
    try:
        for aggs, where in QUERIES:
            out = t.aggregate(aggs, where=where)
            exp = oracle.aggregate(host, CT, aggs, (), where)
            ctx.set_default_variant(threads=512)
            try:
                one = t.aggregate(aggs, where=where)
            finally:
                ctx.set_default_variant(threads=0)
            for got in (out, one):
                assert got.rows_selected == exp.rows_selected
                for ra, rb in zip(got.values, exp.values):
                    assert [(x.value, x.count) for x in ra] == [(y.value, y.count) for y in rb]
    finally:
        t.drop()
