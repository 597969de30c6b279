"""int32 probe keys against build keys of 64 bits: a probe row matches a build
row of equal value, never one 2^32 away. Build ranges past int32 on either side
and across its ends beside the two ranges that just fit, payload bytes and match
bits, one fixed value program, another one, and both as merged scans of a batch."""
import numpy as np
import pytest

import oracle
from turbogp_b200 import datagen
from turbogp_b200.engine import build_col, col, count_star, max_, sum_

pytestmark = pytest.mark.gpu
CT = {**datagen.LINEITEM_COLTYPES, "fk": "int"}
NB = {"bytes": 1_000, "bits": 200_000}
LOWEST = {"past 2^32": lambda nb: 2**32 + 1, "across 2^31": lambda nb: 2**31 - nb // 2,
          "ends at 2^31 - 1": lambda nb: 2**31 - nb, "starts at -2^31": lambda nb: -2**31,
          "across -2^31": lambda nb: -2**31 - nb // 2, "below -2^32": lambda nb: -2**32 - 5}


def same(a, b):
    assert a.rows_selected == b.rows_selected and a.keys == b.keys
    assert [[(v.value, v.count) for v in r] for r in a.values] == [[(v.value, v.count) for v in r] for r in b.values]


@pytest.mark.parametrize("form", NB)
@pytest.mark.parametrize("where_lies", LOWEST)
def test_keys_are_compared_in_64_bits(ctx, form, where_lies):
    nb, n = NB[form], 300_003
    base = LOWEST[where_lies](nb)
    rng = np.random.default_rng(nb)
    dim = datagen.dimension(nb, seed=5)
    dim["key"] = dim["key"].astype(np.int64) - 1 + base
    fact = datagen.lineitem(n, seed=6)
    # Half the probe keys are the build keys' low 32 bits, the others small.
    low = (rng.integers(base, base + nb, n) & 0xffffffff).astype(np.uint32).astype(np.int32)
    fact["fk"] = np.where(rng.random(n) < 0.5, low, rng.integers(-nb, nb, n)).astype(np.int32)
    f, d = ctx.register(fact, CT), ctx.register(dim, {**datagen.DIMENSION_COLTYPES, "key": "int"})
    j = d.join_build("key")
    build = (dim, {**datagen.DIMENSION_COLTYPES, "key": "int"}, "key", None)
    p, q, disc = col("price_cents"), col("quantity"), col("discount_pct")
    fixed, other = [sum_(p * (100 - disc)), count_star()], [sum_(q), max_(disc), count_star()]
    specs = [(fixed, (build_col("segment"),), None), (other, (build_col("segment"), col("quantity")), disc < 9)]
    # Same-shape requests that differ in a bound: merged scans over bucket keys.
    specs += [(fixed, (build_col("segment"),), q < b) for b in (3, 11, 20, 31, 44)]
    want = [oracle.aggregate(fact, CT, a, k, w, build=build, probe_key="fk") for a, k, w in specs]
    pqs = [f.prepare(a, k, w, join=j, probe_key="fk") for a, k, w in specs]
    for got in ([pq.run() for pq in pqs], ctx.submit(pqs).wait()):
        for g, o in zip(got, want):
            same(g, o)
    j.drop()
    f.drop()
    d.drop()
