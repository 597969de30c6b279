"""Join pairs written in place: every table form (unique keys, repeated keys,
runs of one key past the in-place limit, wide key ranges), key dtypes, WHERE
or none, chunk edges and more pairs than probe rows, against the oracle."""
import numpy as np
import pytest

import oracle
from turbogp_b200.engine import col

pytestmark = pytest.mark.gpu


def sides(n, nb, repeat, dtype, spread, seed):
    rng = np.random.default_rng(seed)
    keys = (rng.permutation(nb) // repeat).astype(np.int64) * spread
    build = {"k": keys.astype(dtype), "b": rng.integers(0, 100, nb, dtype=np.int32)}
    probe = {"k": (rng.integers(-3, nb // repeat + 3, n) * spread).astype(dtype),
             "v": rng.integers(0, 100, n, dtype=np.int32), "u": rng.integers(0, 4, n, dtype=np.uint8)}
    return probe, build


@pytest.mark.parametrize("n,nb,repeat,dtype,spread", [
    (0, 10, 1, np.int32, 1), (1, 1, 1, np.int32, 1), (127, 50, 1, np.int32, 1), (128, 50, 2, np.int64, 1),
    (129, 0, 1, np.int32, 1), (4_099, 3_000, 1, np.int64, 2**33), (50_001, 4_000, 3, np.int32, 7),
    (3_001, 640, 64, np.int32, 1), (3_001, 1_300, 65, np.int32, 1), (20_003, 200, 2, np.uint8, 1),
    (9_000, 900, 4, np.int64, 2**34)])
def test_pairs_in_order(ctx, n, nb, repeat, dtype, spread):
    probe, build = sides(n, nb, repeat, dtype, spread, 5 + n)
    tp, tb = ctx.register(probe), ctx.register(build)
    for bw in (None, col("b") < 60):
        j = tb.join_build("k", bw)
        for where in (None, (col("v") < 40) | (col("u") == 1), col("v") > 500):
            pr, br = j.probe_pairs(tp, "k", where)
            opr, obr = oracle.join_pairs(probe, None, "k", where, build, None, "k", bw)
            assert np.array_equal(pr, opr) and np.array_equal(br, obr)
        j.drop()
    tp.drop()
    tb.drop()
