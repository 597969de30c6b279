"""One-word sums of the limb tables at the bound of their 32 bits: one table per
CTA (10,000 groups of COUNT(*) and one SUM), one key with nearly every row, and
values for which the sum of one CTA's rows lies just below 2^31 or just above it,
by the tiles of the scan engine (odd numbers per SM) and by the chunks of the
streaming kernel, at ragged ends too."""
import numpy as np
import pytest

import oracle
from turbogp_b200.engine import col, count_star, sum_

pytestmark = pytest.mark.gpu
TILE = 2048


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("tiles,ragged", [(5, 0), (5, -127), (5, 128), (6, 0), (7, 0), (7, 1), (13, 0)])
def test_dominant_key(ctx, tiles, ragged, sign):
    n = tiles * ctx.sm_count * TILE + ragged
    rng = np.random.default_rng(tiles)
    h = {"k": np.full(n, 4_321, dtype=np.int32)}
    h["k"][:10_000] = np.arange(10_000)        # every group, one key with the other rows
    rows = {tiles * TILE, (tiles + 1) // 2 * 2 * TILE, (tiles + 2) // 2 * 2 * TILE}
    for r in sorted(rows):
        top = (2**31 - 1) // r                 # r rows of it stay within 32 bits, one tile more does not
        h["v"] = (sign * (top - rng.integers(0, 3, n))).astype(np.int32)
        t = ctx.register(h, {"k": "int", "v": "int"})
        for where in (None, col("k") > 17):
            a = t.aggregate([count_star(), sum_(col("v"))], ("k",), where)
            o = oracle.aggregate(h, {"k": "int", "v": "int"}, [count_star(), sum_(col("v"))], ("k",), where)
            assert a.rows_selected == o.rows_selected and a.keys == o.keys
            assert [[(x.value, x.count) for x in r_] for r_ in a.values] == [[(x.value, x.count) for x in r_] for r_ in o.values]
        t.drop()
