"""Performance cases of the engine's hot path: what a program that queries
resident tables has it do, through the Python engine API.

Every case is one pass of one of these paths, on seeded tables with the
benchmark workloads' distributions (``turbogp_b200.datagen``), generated on
the GPU and registered in place:

* ``scan``    — WHERE over four int32 columns, scalar SUM of a product + COUNT.
* ``q1``      — WHERE + GROUP BY two flag columns, six aggregates (TPC-H Q1 shape).
* ``group``   — GROUP BY one dictionary-sized column with SUM / MIN / MAX / COUNT.
* ``key``     — GROUP BY one key of up to millions of values (Zipf), all groups read back.
* ``topn``    — WHERE + GROUP BY a sparse 62-bit id, ORDER BY an aggregate LIMIT n.
* ``filter``  — WHERE into a selection bitmap and ascending row ids.
* ``join``    — hash-join build, probe and grouped aggregate.
* ``pairs``   — hash-join build and probe into (probe row, build row) pairs.
* ``batch``   — queries of uneven sizes and templates submitted together.
* ``serving`` — same-shape requests of three templates submitted together.

Results are the engine's raw result arrays (128-bit sums as two limbs, row
counts, f64 views).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from turbogp_b200 import datagen, workloads
from turbogp_b200.datagen import DAY0, NDAYS
from turbogp_b200.engine import Context, avg, col, count_star, max_, min_, sum_

FACT_COLTYPES = {**datagen.LINEITEM_COLTYPES, "fk": "int"}
_VALUE = np.dtype([("lo", "<i8"), ("hi", "<i8"), ("count", "<i8"), ("as_f64", "<f8")])


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # One small lookup: planning, launch and readback are the whole cost.
        {"name": "scan_small", "kind": "scan", "rows": 10_007, "days": 365, "disc_lo": 5, "disc_hi": 7, "qty_lt": 24},
        # The bandwidth-bound selective scan (TPC-H Q6 shape) at its full size.
        {"name": "scan_large", "kind": "scan", "rows": 60_000_000, "days": 365, "disc_lo": 5, "disc_hi": 7,
         "qty_lt": 24},
        # The plain filtered grouped aggregate (TPC-H Q1 shape) at its full size.
        {"name": "q1", "kind": "q1", "rows": 6_000_000, "ship_max": DAY0 + NDAYS - 91},
        # A report per day: 2,526 groups, extremes beside sums, no fixed shape.
        {"name": "group_day", "kind": "group", "rows": 20_000_003, "by": "ship_day", "extremes": True, "qty_lt": 46},
        # Counts and totals per customer, half a million of them, all read back.
        {"name": "group_key", "kind": "key", "rows": 40_000_000, "nkeys": 500_000, "wide": True},
        # Counts and totals per rarely repeating key (the high-cardinality table), all read back.
        {"name": "group_highcard", "kind": "key", "rows": 50_000_000, "nkeys": 5_000_000, "wide": True},
        # The ten busiest of a million sparse ids (ClickBench shape).
        {"name": "top_ids", "kind": "topn", "rows": 20_000_000, "nkeys": 1_000_000, "value_ge": 100, "limit": 10},
        # A WHERE with OR over integer, date and float columns, rows handed on.
        {"name": "filter_rows", "kind": "filter", "rows": 20_000_017, "days": 365, "ratio_gt": 0.9, "qty_lt": 5},
        # Star join: filtered dimension, 60M-row fact table, grouped total.
        {"name": "join_group", "kind": "join", "rows": 60_000_000, "dim": 1_500_000, "order_day_lt": DAY0 + NDAYS // 2},
        # A join whose rows go on to another operator; some keys repeat.
        {"name": "join_pairs", "kind": "pairs", "rows": 8_000_000, "dim": 400_000, "repeat": 2, "qty_lt": 26},
        # A night's worth of mixed dashboard queries, each over its own range of rows.
        {"name": "batch_uneven", "kind": "batch", "rows": 60_000_000, "dim": 1_500_000, "queries": 64},
        # What a request loop submits under load: the three light templates, random literals.
        {"name": "serving_batch", "kind": "serving", "rows": 60_000_000, "dim": 1_500_000, "each": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "q1", "group", "key", "topn", "filter", "join", "pairs", "batch", "serving"])
    if kind == "scan":
        lo = rng.randrange(0, 8)
        return {"kind": kind, "rows": _log(rng, 1_000, 60_000_000), "days": rng.randrange(20, 1500), "disc_lo": lo,
                "disc_hi": lo + rng.randrange(0, 4), "qty_lt": rng.randrange(3, 50)}
    if kind == "q1":
        return {"kind": kind, "rows": _log(rng, 10_000, 30_000_000), "ship_max": DAY0 + rng.randrange(200, NDAYS)}
    if kind == "group":
        return {"kind": kind, "rows": _log(rng, 200_000, 40_000_000),
                "by": rng.choice(["ship_day", "quantity", "flag_a"]), "extremes": rng.random() < 0.5,
                "qty_lt": rng.randrange(20, 51)}
    if kind == "key":
        rows = _log(rng, 100_000, 50_000_000)
        return {"kind": kind, "rows": rows, "nkeys": _log(rng, 5_000, min(5_000_000, rows // 2)),
                "wide": rng.random() < 0.5}
    if kind == "topn":
        rows = _log(rng, 100_000, 30_000_000)
        return {"kind": kind, "rows": rows, "nkeys": _log(rng, 1_000, rows // 4), "value_ge": rng.randrange(0, 800),
                "limit": rng.randrange(5, 100)}
    if kind == "filter":
        return {"kind": kind, "rows": _log(rng, 10_000, 40_000_000), "days": rng.randrange(20, 1000),
                "ratio_gt": round(rng.uniform(0.3, 0.99), 3), "qty_lt": rng.randrange(2, 25)}
    if kind == "join":
        rows = _log(rng, 100_000, 60_000_000)
        return {"kind": kind, "rows": rows, "dim": _log(rng, 2_000, min(1_500_000, rows // 8)),
                "order_day_lt": DAY0 + rng.randrange(800, NDAYS)}
    if kind == "pairs":
        rows = _log(rng, 50_000, 12_000_000)
        return {"kind": kind, "rows": rows, "dim": _log(rng, 1_000, min(1_000_000, rows // 4)),
                "repeat": rng.choice([1, 1, 2, 3]), "qty_lt": rng.randrange(3, 51)}
    if kind == "batch":
        return {"kind": kind, "rows": _log(rng, 2_000_000, 60_000_000), "dim": _log(rng, 50_000, 1_500_000),
                "queries": rng.randrange(8, 64)}
    return {"kind": kind, "rows": _log(rng, 500_000, 60_000_000), "dim": _log(rng, 20_000, 1_500_000),
            "each": rng.randrange(1, 17)}


# ---------------------------------------------------------------------------
# Inputs, generated on the GPU from (case, seed)
# ---------------------------------------------------------------------------
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _ints(lo, hi, n, dtype, gen):
    return torch.randint(lo, hi, (n,), dtype=dtype, device="cuda", generator=gen)


def _lineitem(n, seed):
    g = _gen(seed, 1)
    return {
        "quantity": _ints(1, 51, n, torch.int32, g),
        "price_cents": _ints(90_000, 10_500_001, n, torch.int64, g),
        "discount_pct": _ints(0, 11, n, torch.int32, g),
        "tax_pct": _ints(0, 9, n, torch.int32, g),
        "ship_day": _ints(DAY0, DAY0 + NDAYS, n, torch.int32, g),
        "flag_a": _ints(0, 3, n, torch.uint8, g),
        "flag_b": _ints(0, 2, n, torch.uint8, g),
    }


def _zipf(n, nkeys, s, gen):
    """n ranks 1..nkeys with P(r) proportional to r^-s."""
    cdf = torch.cumsum(torch.arange(1, nkeys + 1, dtype=torch.float64, device="cuda") ** -s, 0)
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) * cdf[-1]
    return torch.searchsorted(cdf, u, right=True).clamp_(max=nkeys - 1) + 1


def _fact(n, nkeys, seed):
    t = _lineitem(n, seed)
    t["fk"] = _zipf(n, nkeys, 0.8, _gen(seed, 2)).to(torch.int32)
    return t


def _shuffled(columns, seed):
    """The same rows in an order of the seed's own: row counts of a result
    do not depend on the seed."""
    n = next(iter(columns.values())).numel()
    order = torch.randperm(n, device="cuda", generator=_gen(seed, 8))
    return {k: v[order] for k, v in columns.items()}


def _dimension(n, seed, repeat=1):
    """Keys 1..n/repeat in random order, each `repeat` times."""
    g = _gen(seed, 3)
    key = torch.randperm(n, device="cuda", generator=g) % max(1, n // repeat) + 1
    return {"key": key.to(torch.int32), "order_day": _ints(DAY0, DAY0 + NDAYS, n, torch.int32, g),
            "segment": _ints(0, 25, n, torch.uint8, g)}


def _columns(case, seed):
    """The case's tables: {"t": the scanned table, "d": the dimension}."""
    kind, n = case["kind"], case["rows"]
    if kind in ("scan", "q1", "group"):
        return {"t": _lineitem(n, seed)}
    if kind == "filter":
        t = {k: v for k, v in _lineitem(n, 0).items() if k in ("quantity", "price_cents", "ship_day")}
        t["ratio"] = torch.rand(n, dtype=torch.float64, device="cuda", generator=_gen(0, 4))
        return {"t": _shuffled(t, seed)}
    if kind == "key":
        rank = _zipf(n, case["nkeys"], 1.1, _gen(0, 5))
        return {"t": {**_shuffled({"key": rank if case["wide"] else rank.to(torch.int32)}, seed),
                      "value": _ints(0, 1001, n, torch.int32, _gen(seed, 6))}}
    if kind == "topn":
        ids = _ints(0, 1 << 62, case["nkeys"], torch.int64, _gen(seed, 7))
        return {"t": {"id": ids[_zipf(n, case["nkeys"], 1.1, _gen(seed, 5)) - 1],
                      "value": _ints(0, 1001, n, torch.int32, _gen(seed, 6))}}
    if kind == "pairs":
        t = _fact(n, max(1, case["dim"] // case["repeat"]), 0)
        return {"t": _shuffled({k: t[k] for k in ("quantity", "price_cents", "fk")}, seed),
                "d": _shuffled(_dimension(case["dim"], 0, case["repeat"]), seed)}
    return {"t": _fact(n, case["dim"], seed), "d": _dimension(case["dim"], seed)}


def _scan(day_lo, days, disc_lo, disc_hi, qty_lt):
    return {"kind": "scan", "day_lo": day_lo, "days": days, "disc_lo": disc_lo, "disc_hi": disc_hi, "qty_lt": qty_lt}


def _requests(case, seed):
    """The queries of a batch: (rows, template and literals) each; the seed
    draws the literals."""
    rng, sizes = random.Random(int(seed) * 7919 + 13), random.Random(case["rows"])
    out = []
    if case["kind"] == "batch":
        for i in range(case["queries"]):
            n = case["rows"] if i == 0 else min(case["rows"], _log(sizes, 10_000, case["rows"]))
            k = i % 3
            if k == 0:
                p = _scan(DAY0 + rng.randrange(0, 2000), rng.randrange(30, 526), rng.randrange(0, 6),
                          rng.randrange(5, 11), rng.randrange(2, 51))
            elif k == 1:
                p = {"kind": "q1", "ship_max": DAY0 + rng.randrange(300, NDAYS)}
            else:
                p = {"kind": "join", "qty_lt": rng.randrange(12, 51)}
            out.append((n, p))
        return out
    for _ in range(case["each"]):
        lo = rng.randrange(0, 6)
        out.append((case["rows"], _scan(DAY0 + rng.randrange(0, 2100), rng.randrange(30, 425), lo,
                                        lo + rng.randrange(1, 5), rng.randrange(5, 50))))
        out.append((case["rows"], {"kind": "q1", "ship_max": DAY0 + rng.randrange(300, NDAYS)}))
        out.append((case["rows"], {"kind": "join", "qty_lt": rng.randrange(5, 51)}))
    return out


def _median_day():
    return DAY0 + NDAYS // 2


# ---------------------------------------------------------------------------
# The programs
# ---------------------------------------------------------------------------
_CTX = None


def _context():
    """The program's one context."""
    global _CTX
    if _CTX is None:
        _CTX = Context(0)
    return _CTX


class _State:
    """What a program holds between calls: its resident tables and prepared
    queries, released with it."""

    def __init__(self, case):
        self.case = case
        self.ctx = _context()
        self.tables, self.joins, self.queries = [], [], []

    def register(self, columns, coltypes=None):
        t = self.ctx.register_device(columns, coltypes)
        self.tables.append(t)
        return t

    def __del__(self):
        for j in self.joins:
            j.drop()
        for t in self.tables:
            t.drop()


def _where_scan(p):
    return ((col("ship_day") >= p["day_lo"]) & (col("ship_day") < p["day_lo"] + p["days"]) &
            col("discount_pct").between(p["disc_lo"], p["disc_hi"]) & (col("quantity") < p["qty_lt"]))


def _where_filter(case):
    return (((col("ship_day") >= DAY0 + 400) & (col("ship_day") < DAY0 + 400 + case["days"]) &
             (col("ratio") > case["ratio_gt"])) | (col("quantity") < case["qty_lt"]))


def _template(p, join=None):
    """(aggregates, group keys, WHERE, join, probe key) of one request."""
    if p["kind"] == "scan":
        return ([sum_(col("price_cents") * col("discount_pct")), count_star()], (), _where_scan(p), None, None)
    if p["kind"] == "q1":
        t = workloads.filtered_group_agg(p["ship_max"])
        return t.aggs, t.group_by, t.where, None, None
    t = workloads.join_group_agg()
    where = col("quantity") < p["qty_lt"] if "qty_lt" in p else None
    return t.aggs, t.group_by, where, join, "fk"


def _group_aggs(case):
    p, q = col("price_cents"), col("quantity")
    if case["extremes"]:
        return [count_star(), sum_(p), min_(p), max_(p), avg(q)]
    return [count_star(), sum_(p), sum_(p * (100 - col("discount_pct"))), avg(q)]


def prepare(case, seed):
    s = _State(case)
    cols = _columns(case, seed)
    torch.cuda.synchronize()
    kind = case["kind"]
    if kind == "scan":
        t = s.register(cols["t"], datagen.LINEITEM_COLTYPES)
        s.queries.append(t.prepare(*_template({**case, "day_lo": DAY0 + 730})[:3]))
    elif kind == "q1":
        t = s.register(cols["t"], datagen.LINEITEM_COLTYPES)
        s.queries.append(t.prepare(*_template(case)[:3]))
    elif kind == "group":
        t = s.register(cols["t"], datagen.LINEITEM_COLTYPES)
        s.queries.append(t.prepare(_group_aggs(case), (case["by"],), col("quantity") < case["qty_lt"],
                                   group_cap=4096))
    elif kind == "key":
        t = s.register(cols["t"])
        s.queries.append(t.prepare([count_star(), sum_(col("value"))], ("key",), None,
                                   group_cap=min(case["nkeys"], case["rows"])))
    elif kind == "topn":
        s.register(cols["t"])
    elif kind == "filter":
        s.register(cols["t"], {"ship_day": "date", "ratio": "float"})
    elif kind in ("join", "pairs"):
        s.register(cols["t"], FACT_COLTYPES)
        s.register(cols["d"], datagen.DIMENSION_COLTYPES)
    else:
        d = s.register(cols["d"], datagen.DIMENSION_COLTYPES)
        j = d.join_build("key", col("order_day") < _median_day())
        s.joins.append(j)
        views = {}
        for n, p in _requests(case, seed):
            if n not in views:
                views[n] = s.register({k: v[:n] for k, v in cols["t"].items()}, FACT_COLTYPES)
            aggs, keys, where, join, probe = _template(p, j)
            s.queries.append(views[n].prepare(aggs, keys, where, join=join, probe_key=probe, group_cap=64))
    return s


def _raw(q, result):
    """A prepared query's raw results: keys, and the aggregates' records."""
    n = int(result.ngroups)
    return q.keys[:n * q.nk].view(np.int64), np.frombuffer(q.vals, dtype=_VALUE, count=n * q.na)


def _outputs(keys, vals):
    return {"keys": keys, "lo": vals["lo"], "hi": vals["hi"], "count": vals["count"], "as_f64": vals["as_f64"]}


def run(s):
    case = s.case
    kind = case["kind"]
    if kind in ("scan", "q1", "group", "key"):
        q = s.queries[0]
        q.run(decode=False)
        return _outputs(*_raw(q, q.res))
    if kind == "topn":
        out = s.tables[0].aggregate_topn([count_star(), sum_(col("value"))], ("id",),
                                         col("value") >= case["value_ge"], 0, True, case["limit"])
        return {"keys": np.array(out.keys, dtype=np.int64).reshape(-1),
                "sum": np.array([[v.value, v.count] for r in out.values for v in r], dtype=np.int64),
                "as_f64": np.array([v.as_f64 for r in out.values for v in r])}
    if kind == "filter":
        f = s.tables[0].filter(_where_filter(case))
        return {"count": f.count, "bitmap": f.bitmap, "rowids": f.rowids}
    if kind == "join":
        fact, dim = s.tables
        j = dim.join_build("key", col("order_day") < case["order_day_lt"])
        aggs, keys, where, join, probe = _template({"kind": "join"}, j)
        q = fact.prepare(aggs, keys, where, join=join, probe_key=probe, group_cap=64)
        q.run(decode=False)
        out = _outputs(*_raw(q, q.res))
        j.drop()
        return out
    if kind == "pairs":
        fact, dim = s.tables
        j = dim.join_build("key", col("order_day") < _median_day())
        probe, build = j.probe_pairs(fact, "fk", col("quantity") < case["qty_lt"])
        j.drop()
        return {"probe": probe, "build": build}
    batch = s.ctx.submit(s.queries, decode=False)
    batch.wait()
    parts = [_raw(q, it.result) for q, it in zip(s.queries, batch.items)]
    return _outputs(np.concatenate([k for k, _ in parts]), np.concatenate([v for _, v in parts]))


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
_SCAN_ROW, _Q1_ROW, _JOIN_ROW = 20, 26, 16   # bytes of the columns a template reads per row


def work(case):
    """Bytes of the referenced columns read once and of the results written
    once; operations: a compare per predicate leaf and an operation per
    aggregate step, per row."""
    kind, n = case["kind"], case["rows"]
    if kind == "scan":
        return {"bytes": n * _SCAN_ROW + 64, "flops": n * 6}
    if kind == "q1":
        return {"bytes": n * _Q1_ROW + 6 * (16 + 6 * 32), "flops": n * 11}
    if kind == "group":
        groups = {"ship_day": NDAYS, "quantity": min(50, case["qty_lt"] - 1), "flag_a": 3}[case["by"]]
        width = {"ship_day": 4, "quantity": 0, "flag_a": 1}[case["by"]]
        return {"bytes": n * (4 + 8 + width + (0 if case["extremes"] else 4)) + groups * (8 + 5 * 32), "flops": n * 7}
    if kind == "key":
        groups = _expected_distinct(n, case["nkeys"], 1.1)
        return {"bytes": n * (12 if case["wide"] else 8) + groups * (8 + 2 * 32), "flops": n * 2}
    if kind == "topn":
        return {"bytes": n * 12 + case["limit"] * (8 + 2 * 32), "flops": n * 3}
    if kind == "filter":
        q = (case["qty_lt"] - 1) / 50
        hit = q + (1 - q) * case["days"] / NDAYS * (1 - case["ratio_gt"])
        return {"bytes": n * (4 + 8 + 4) + n / 8 + n * hit * 4, "flops": n * 5}
    if kind == "join":
        return {"bytes": n * _JOIN_ROW + case["dim"] * 9 + 25 * (8 + 2 * 32), "flops": n * 5}
    if kind == "pairs":
        hits = n * (case["qty_lt"] - 1) / 50 * 0.5 * case["repeat"]
        return {"bytes": n * 8 + case["dim"] * 8 + hits * 8, "flops": n * 3}
    per = {"scan": (_SCAN_ROW, 6), "q1": (_Q1_ROW, 11), "join": (_JOIN_ROW + 4, 6)}
    if kind == "serving":
        # One read of the table's eight columns serves every request.
        return {"bytes": n * 30 + 3 * case["each"] * 512, "flops": n * 23 * case["each"]}
    rows = [(m, p["kind"]) for m, p in _requests(case, 0)]
    return {"bytes": sum(m * per[k][0] for m, k in rows), "flops": sum(m * per[k][1] for m, k in rows)}


def _expected_distinct(n, nkeys, s):
    w = np.arange(1, nkeys + 1, dtype=np.float64) ** -s
    return int(np.sum(-np.expm1(-n * w / w.sum())))


# ---------------------------------------------------------------------------
# The exact results, in 64-bit integers and floats, with plain torch
# ---------------------------------------------------------------------------
def _leaves_scan(t, p):
    d, day, q = t["discount_pct"], t["ship_day"], t["quantity"]
    return ((day >= p["day_lo"]) & (day < p["day_lo"] + p["days"]) & (d >= p["disc_lo"]) & (d <= p["disc_hi"]) &
            (q < p["qty_lt"]))


def _records(count, columns):
    """Records of one query's groups: `columns` holds, per aggregate, int64
    values (None: the row count) and whether it is an average."""
    n = len(count)
    v = np.zeros((n, len(columns)), dtype=_VALUE)
    for a, (x, mean) in enumerate(columns):
        x = count if x is None else x
        v["lo"][:, a] = x
        v["hi"][:, a] = x >> 63
        v["count"][:, a] = count
        v["as_f64"][:, a] = x.astype(np.float64) / count if mean else x.astype(np.float64)
    return v.reshape(-1)


def _host(x):
    return x.cpu().numpy()


def _by_mask(group, ngroups, args):
    """Row count and int64 sums of few groups, one masked sum each."""
    counts, sums = [], [[] for _ in args]
    for g in range(ngroups):
        m = group == g
        counts.append(int(m.sum()))
        for a, x in enumerate(args):
            sums[a].append(int((x * m).sum()))
    return np.array(counts, dtype=np.int64), [np.array(s, dtype=np.int64) for s in sums]


def _exact_template(p, t, d=None):
    """(keys, records) of one request over the columns `t`."""
    price = t["price_cents"]
    if p["kind"] == "scan":
        m = _leaves_scan(t, p)
        n = int(m.sum())
        s = int((price * t["discount_pct"] * m).sum())
        rec = np.zeros(2, dtype=_VALUE)
        rec["lo"], rec["hi"], rec["count"], rec["as_f64"] = [s, n], [s >> 63, 0], n, [float(s), float(n)]
        return np.zeros(0, dtype=np.int64), rec
    disc = price * (100 - t["discount_pct"].long())
    if p["kind"] == "q1":
        group = torch.where(t["ship_day"] <= p["ship_max"], t["flag_a"].to(torch.int32) * 2 + t["flag_b"], -1)
        count, sums = _by_mask(group, 6, [t["quantity"].long(), price, disc, disc * (100 + t["tax_pct"].long())])
        some = count > 0
        ids = np.flatnonzero(some)
        sums = [s[some] for s in sums]
        rec = _records(count[some], [(None, False), *((s, False) for s in sums), (sums[0], True)])
        return np.stack([ids // 2, ids % 2], 1).reshape(-1).astype(np.int64), rec
    seg = torch.full((int(d["key"].max()) + 1,), -1, dtype=torch.int32, device="cuda")
    hit = d["order_day"] < p.get("order_day_lt", _median_day())
    seg[d["key"][hit].long()] = d["segment"][hit].to(torch.int32)
    # A key past the dimension's last (fk reaches it, its build row may not) matches nothing.
    fk = t["fk"].long().clamp(max=seg.numel() - 1)
    group = torch.where(t["fk"] < seg.numel(), seg[fk], -1)
    if "qty_lt" in p:
        group = torch.where(t["quantity"] < p["qty_lt"], group, -1)
    count, sums = _by_mask(group, 25, [disc])
    some = count > 0
    return np.flatnonzero(some).astype(np.int64), _records(count[some], [(sums[0][some], False), (None, False)])


def _by_index(index, n, args, extremes=None):
    """Row count, int64 sums and extremes of many groups."""
    count = torch.bincount(index, minlength=n)
    sums = [torch.zeros(n, dtype=torch.int64, device="cuda").index_add_(0, index, x.long()) for x in args]
    ends = []
    if extremes is not None:
        for how in ("amin", "amax"):
            z = torch.zeros(n, dtype=torch.int64, device="cuda")
            ends.append(z.scatter_reduce_(0, index, extremes, how, include_self=False))
    some = count > 0
    return _host(torch.nonzero(some).reshape(-1)), _host(count[some]), [_host(x[some]) for x in sums + ends]


def exact(case, seed):
    cols = _columns(case, seed)
    t, kind = cols["t"], case["kind"]
    if kind == "scan":
        return _outputs(*_exact_template({**case, "day_lo": DAY0 + 730}, t))
    if kind in ("q1", "join"):
        return _outputs(*_exact_template(case, t, cols.get("d")))
    if kind == "group":
        m = t["quantity"] < case["qty_lt"]
        by, price, qty = t[case["by"]][m].long(), t["price_cents"][m], t["quantity"][m]
        lo = int(t[case["by"]].min())
        if case["extremes"]:
            ids, count, (s, q, mn, mx) = _by_index(by - lo, 4096, [price, qty], price)
            rec = _records(count, [(None, False), (s, False), (mn, False), (mx, False), (q, True)])
        else:
            ids, count, (s, ds, q) = _by_index(by - lo, 4096, [price, price * (100 - t["discount_pct"][m].long()), qty])
            rec = _records(count, [(None, False), (s, False), (ds, False), (q, True)])
        return _outputs(ids + lo, rec)
    if kind == "key":
        ids, count, (s,) = _by_index(t["key"].long(), case["nkeys"] + 1, [t["value"]])
        return _outputs(ids, _records(count, [(None, False), (s, False)]))
    if kind == "topn":
        m = t["value"] >= case["value_ge"]
        ids, inv = torch.unique(t["id"][m], return_inverse=True)
        _, count, (s,) = _by_index(inv, ids.numel(), [t["value"][m]])
        top = np.argsort(-count, kind="stable")[:case["limit"]]
        count, s = count[top], s[top]
        return {"keys": _host(ids)[top], "sum": np.stack([count, count, s, count], 1).reshape(-1, 2),
                "as_f64": np.stack([count, s], 1).reshape(-1).astype(np.float64)}
    if kind == "filter":
        day = t["ship_day"]
        m = (((day >= DAY0 + 400) & (day < DAY0 + 400 + case["days"]) & (t["ratio"] > case["ratio_gt"])) |
             (t["quantity"] < case["qty_lt"]))
        m = _host(m)
        rows = np.flatnonzero(m)
        return {"count": len(rows), "bitmap": np.packbits(m, bitorder="little"), "rowids": rows.astype(np.uint32)}
    if kind == "pairs":
        d = cols["d"]
        rows = torch.nonzero(d["order_day"] < _median_day()).reshape(-1)
        key, order = torch.sort(d["key"][rows], stable=True)
        probe = torch.nonzero(t["quantity"] < case["qty_lt"]).reshape(-1)
        fk = t["fk"][probe].contiguous()
        first = torch.searchsorted(key, fk)
        many = torch.searchsorted(key, fk, right=True) - first
        pr = torch.repeat_interleave(probe, many)
        nth = torch.arange(pr.numel(), device="cuda") - torch.repeat_interleave(torch.cumsum(many, 0) - many, many)
        br = rows[order][torch.repeat_interleave(first, many) + nth]
        return {"probe": _host(pr).astype(np.uint32), "build": _host(br).astype(np.uint32)}
    parts = [_exact_template(p, {k: v[:n] for k, v in t.items()}, cols["d"]) for n, p in _requests(case, seed)]
    return _outputs(np.concatenate([k for k, _ in parts]), np.concatenate([v for _, v in parts]))
