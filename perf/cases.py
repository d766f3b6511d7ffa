"""The work a user of the library has it do, as cases that can be timed.

One case is a dict of plain values: a ``kind`` (which public entry points it
goes through), sizes, and the options of that kind.  ``listed()`` names twelve
of them, from a 10,007-row star-join to the 600M-row one; ``draw`` gives more
of the same ranges.  Inputs are synthetic, made on the GPU from the seed alone
with the sizes and distributions of ``workloads.py`` and ``bench.py``.

Sums and row ids are whole numbers, the same bit for bit on every run (groups
come back unordered, so the group cases put them in key order, as a report
does); only the double aggregation has a floating result, and ``exact`` gives
its value in plain torch.  The number of rows that pass a filter, match or
form a group is fixed by the case, which rows they are by the seed, so that
outputs have the same shape for every seed; where that number is the seed's
(the column-wise list), the caller's whole buffers and the count come back.
"""
import math

import numpy as np
import torch

from memory_database_b200 import batch, olapcore, operators, q5
from memory_database_b200.olapcore import AGG_M1, AGG_M1_PLUS_M2, AGG_M1_TIMES_M2

DATE_ROWS = 2556
SCALE_DIMS = "3000000,200000,1400000,2556"
SMALL_DIMS = "30000,2000,200000,2556"


def listed():
    return [
        # The star-join at scale: 600M fact rows, SUM(m1) and SUM(m1*m2) by
        # 4096 groups, with the plan the autotuner keeps for the query shape.
        {"name": "star_scale", "kind": "star", "rows": 599_999_993, "dims": SCALE_DIMS, "sele": "0.5,0.2,0.1,1.0",
         "groups": "8,8,8,8", "sums": 2, "zipf": 0.0, "tuned": True},
        # An ordinary report over a 6M-row fact table: 35,000 groups, no tuning.
        {"name": "star_small", "kind": "star", "rows": 6_000_000, "dims": SMALL_DIMS, "sele": "0.2,0.2,0.2,0.2",
         "groups": "5,25,40,7", "sums": 1, "zipf": 0.0, "tuned": False},
        # The smallest call: a few thousand rows, where launches count.
        {"name": "star_tiny", "kind": "star", "rows": 10_007, "dims": "1000,200,2000,2556", "sele": "0.2,0.5,0.5,1.0",
         "groups": "5,1,25,7", "sums": 1, "zipf": 0.0, "tuned": False},
        # The column-wise model: the list of surviving rows, then their sums.
        {"name": "star_columnwise", "kind": "columnwise", "rows": 120_000_001, "dims": SCALE_DIMS,
         "sele": "0.5,0.2,0.5,1.0", "groups": "8,8,8,8", "form": "dv"},
        # A fact table that stays in (pinned) host memory.
        {"name": "star_host", "kind": "host", "rows": 12_000_000, "dims": SMALL_DIMS, "sele": "0.5,0.2,0.1,1.0",
         "groups": "8,8,8,8"},
        # A dashboard's 64 queries in one pass over a shared fact table.
        {"name": "star_batch", "kind": "batch", "rows": 240_000_007, "dims": SCALE_DIMS, "groups": "25,25,40,7",
         "queries": 64},
        # The five-table chain at the serving sizes.
        {"name": "q5_chain", "kind": "q5", "lines": 60_000_000, "queries": 1},
        # A filter and the late materialisation of four columns.
        {"name": "select_gather", "kind": "select", "rows": 268_435_399, "share": 0.1, "columns": 4},
        # A hash join: build on 2^24 unique keys, SUM over the probe side.
        {"name": "join_large", "kind": "join", "build": 1 << 24, "probe": (1 << 27) + 5, "match": 0.5, "zipf": 0.0,
         "pairs": False},
        # Many groups: 2^20 keys, SUM and COUNT.
        {"name": "group_many", "kind": "group", "rows": (1 << 27) + 3, "groups": 1 << 20, "values": 1, "zipf": 0.0},
        # A whole small query: join a dimension, fetch the measure, few groups.
        {"name": "join_group", "kind": "join_group", "dim": 200_000, "rows": 20_000_003, "groups": 1000},
        # The aggregation module's expression over doubles.
        {"name": "aggregate", "kind": "aggregate", "rows": (1 << 27) + 1, "type": "f64"},
    ]


# ---- more cases of the same ranges ------------------------------------------

def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _star_shape(rng, sf):
    """Dimension sizes and filters of a star schema at scale factor sf."""
    dims = (max(100, int(30_000 * sf)), max(50, int(2_000 * sf)),
            max(200, int(200_000 * min(sf, 1 + math.log2(max(sf, 1))))), DATE_ROWS)
    sele = [rng.choice((0.04, 0.1, 0.2, 0.5, 0.85, 1.0)) for _ in range(4)]
    groups = [rng.choice((1, 5, 7, 8, 25)) for _ in range(4)]
    return {"dims": ",".join(map(str, dims)), "sele": ",".join(map(str, sele)), "groups": ",".join(map(str, groups))}


def draw(rng):
    kind = rng.choice(("star", "star", "columnwise", "host", "batch", "q5", "select", "join", "group", "join_group",
                       "aggregate"))
    if kind == "star":
        rows = _log(rng, 10_000, 500_000_000)
        return {"kind": kind, "rows": rows, **_star_shape(rng, rows / 6e6), "sums": rng.choice((1, 2)),
                "zipf": rng.choice((0.0, 0.0, 0.8)), "tuned": rows > 50_000_000 and rng.random() < 0.5}
    if kind == "columnwise":
        rows = _log(rng, 50_000, 200_000_000)
        shape = _star_shape(rng, rows / 6e6)
        shape["groups"] = ",".join(str(rng.choice((1, 5, 7, 8))) for _ in range(4))  # int16 group ids
        return {"kind": kind, "rows": rows, **shape, "form": rng.choice(("dv", "sv"))}
    if kind == "host":
        rows = _log(rng, 100_000, 16_000_000)
        return {"kind": kind, "rows": rows, **_star_shape(rng, rows / 6e6)}
    if kind == "batch":
        rows = _log(rng, 1_000_000, 240_000_000)
        return {"kind": kind, "rows": rows, "dims": _star_shape(rng, rows / 6e6)["dims"], "groups": "25,25,40,7",
                "queries": rng.randint(4, 64)}
    if kind == "q5":
        return {"kind": kind, "lines": _log(rng, 60_000, 120_000_000), "queries": rng.choice((1, 1, 64))}
    if kind == "select":
        return {"kind": kind, "rows": _log(rng, 10_000, 268_435_456), "share": 10 ** rng.uniform(-3, -0.3),
                "columns": rng.randint(1, 4)}
    if kind == "join":
        build = _log(rng, 1_000, 1 << 24)
        return {"kind": kind, "build": build, "probe": min(1 << 27, _log(rng, 2 * build, 32 * build)),
                "match": rng.choice((0.1, 0.5, 1.0)), "zipf": rng.choice((0.0, 0.0, 1.0)), "pairs": rng.random() < 0.5}
    if kind == "group":
        rows = _log(rng, 10_000, 1 << 28)
        return {"kind": kind, "rows": rows, "groups": _log(rng, 16, max(32, min(1 << 22, rows // 8))),
                "values": rng.choice((1, 2)), "zipf": rng.choice((0.0, 0.0, 1.0))}
    if kind == "join_group":
        dim = _log(rng, 2_000, 3_000_000)
        return {"kind": kind, "dim": dim, "rows": _log(rng, 10 * dim, 100_000_000), "groups": _log(rng, 5, min(2_000, dim // 10))}
    return {"kind": kind, "rows": _log(rng, 100_000, 200_000_000), "type": rng.choice(("f64", "fixed"))}


# ---- inputs --------------------------------------------------------------------

def _nums(text, to=int):
    return tuple(to(x) for x in text.split(","))


def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _ints(g, n, lo, hi):
    """n int32 values uniform in [lo, hi]."""
    return torch.randint(lo, hi + 1, (n,), generator=g, device="cuda", dtype=torch.int32)


def _keys(g, n, domain, zipf):
    """n int32 keys in [0, domain): uniform, or Zipf(zipf) by the inverse of its continuous distribution."""
    if not zipf:
        return _ints(g, n, 0, domain - 1)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    for b in range(0, n, 1 << 26):
        u = torch.rand(min(1 << 26, n - b), generator=g, device="cuda", dtype=torch.float64)
        if zipf == 1.0:
            x = (u * math.log(domain + 1.0)).exp_()
        else:
            x = u.mul_((domain + 1.0) ** (1 - zipf) - 1).add_(1).pow_(1 / (1 - zipf))
        out[b: b + x.numel()] = x.sub_(1).clamp_(0, domain - 1)
    return out


def _star_inputs(case, seed):
    """Dimension vectors (a group code, or DIM_NULL where the filter drops the row), fact columns and plan."""
    g = _gen(seed)
    dims, sele, groups = _nums(case["dims"]), _nums(case["sele"], float), _nums(case["groups"])
    s = {"dims": dims, "vec": [], "fk": []}
    for n, p, k in zip(dims, sele, groups):
        code = torch.randint(0, k, (n,), generator=g, device="cuda", dtype=torch.int8)
        live = torch.rand(n, generator=g, device="cuda") < p
        s["vec"].append(torch.where(live, code, olapcore.DIM_NULL).to(torch.int8))
    for n in dims:
        s["fk"].append(_keys(g, case["rows"], n, case.get("zipf", 0.0)))
    s["m1"], s["m2"] = _ints(g, case["rows"], 1, 10_000), _ints(g, case["rows"], 1, 10_000)
    s["orders"], s["factor"], s["nd"], s["groups"] = olapcore.plan_olapcore(sele, (1, 1, 1, 1), groups)
    return s


def _star_args(s):
    o = s["orders"]
    return [s["vec"][t] for t in o], [s["fk"][t] for t in o], s["factor"], s["m1"], s["m2"], s["groups"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "star":
        s = _star_inputs(case, seed)
        s["aggs"] = (AGG_M1, AGG_M1_TIMES_M2) if case["sums"] == 2 else (AGG_M1_PLUS_M2,)
        s["ctx"] = olapcore.default_context()
        if case["tuned"]:
            s["ctx"] = olapcore.Context(0)
            olapcore.autotune(*_star_args(s), aggs=s["aggs"], ctx=s["ctx"])
        return s
    if kind == "columnwise":
        s = _star_inputs(case, seed)
        n = case["rows"]
        s["gid"] = torch.zeros(n, dtype=torch.int16, device="cuda")
        s["oid"] = torch.zeros(n if case["form"] == "dv" else 1, dtype=torch.int64, device="cuda")
        s["sums"] = torch.empty(s["groups"], dtype=torch.int64, device="cuda")
        s["form"], s["rows"] = case["form"], n
        return s
    if kind == "host":
        s = _star_inputs(case, seed)

        def pinned(x):
            h = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
            h.copy_(x)
            return h.numpy()
        for k in ("vec", "fk"):
            s[k] = [pinned(x) for x in s[k]]
        s["m1"], s["m2"] = pinned(s["m1"]), pinned(s["m2"])
        return s
    if kind == "batch":
        g = _gen(seed)
        dims, groups, n = _nums(case["dims"]), _nums(case["groups"]), case["rows"]
        d = batch.DimTables(dims, groups)
        for size, k in zip(dims, groups):
            d.filt.append(_ints(g, size, 0, batch.FILTER_DOMAIN - 1))
            d.grp.append(_ints(g, size, 0, k - 1))
        s = {"fk": [_ints(g, n, 0, size - 1) for size in dims], "m1": _ints(g, n, 1, 10_000),
             "m2": _ints(g, n, 1, 10_000)}
        # the panels keep their group columns; their filters and fact ranges are the seed's
        s["queries"] = batch.random_queries(np.random.default_rng(case["queries"]), case["queries"], n, groups)
        for q, new in zip(s["queries"], batch.random_queries(np.random.default_rng(seed), case["queries"], n, groups)):
            q.lo, q.hi, q.row_begin, q.row_end = new.lo, new.hi, new.row_begin, new.row_end
        s["engine"] = batch.BatchEngine(olapcore.default_context(), d, max_queries=64)
        s["engine"].autotune(s["queries"], s["fk"], s["m1"], s["m2"])
        return s
    if kind == "q5":
        g = _gen(seed)
        lines = case["lines"]
        supp, cust, orders = max(10, lines // 600), max(100, lines // 40), max(100, lines // 4)
        cols = {
            "r_regionkey": torch.arange(5, dtype=torch.int32, device="cuda"),
            "n_regionkey": torch.arange(25, dtype=torch.int32, device="cuda") % 5,
            "s_nationkey": _ints(g, supp, 0, 24), "c_nationkey": _ints(g, cust, 0, 24),
            "o_custkey": _ints(g, orders, 1, cust), "o_orderdate": _ints(g, orders, 0, q5.DAYS - 1),
            "l_orderkey": _ints(g, lines, 0, orders - 1), "l_suppkey": _ints(g, lines, 1, supp),
            "l_price": _ints(g, lines, 90_000, 10_500_000), "l_discount": _ints(g, lines, 0, 10),
        }
        return {"data": q5.Q5Data(cols), "queries": q5.random_q5_queries(np.random.default_rng(seed), case["queries"]),
                "ctx": olapcore.default_context()}
    if kind == "select":
        g = _gen(seed)
        n, top, below = case["rows"], 1 << 20, max(1, int(case["share"] * (1 << 20)))
        perm = torch.randperm(n, generator=g, device="cuda", dtype=torch.int32)
        col = torch.where(perm < int(n * case["share"]), perm % below, below + perm % (top - below))
        return {"col": col, "below": below, "cols": [_ints(g, case["rows"], -1000, 1000) for _ in range(case["columns"])]}
    if kind == "join":
        g = _gen(seed)
        nb = case["build"]
        keys = torch.randperm(nb, generator=g, device="cuda", dtype=torch.int32).add_(1)  # unique, 1 .. nb
        probe = keys[_keys(g, case["probe"], nb, case["zipf"]).long()]
        hits = int(case["probe"] * case["match"])
        miss = torch.randperm(case["probe"], generator=g, device="cuda", dtype=torch.int32) >= hits
        probe = torch.where(miss, probe + (nb + 7), probe)  # past the build keys: matches nothing
        return {"keys": keys, "pay": _ints(g, nb, -1000, 1000), "probe": probe, "pairs": case["pairs"]}
    if kind == "group":
        g = _gen(seed)
        n, k = case["rows"], case["groups"]
        keys = _keys(g, n, k, case["zipf"])
        keys[:: n // k][:k] = torch.arange(k, dtype=torch.int32, device="cuda")  # every group has a row
        return {"keys": keys, "groups": k, "vals": [_ints(g, case["rows"], -1000, 1000) for _ in range(case["values"])]}
    if kind == "join_group":
        g = _gen(seed)
        return {"dk": torch.randperm(case["dim"], generator=g, device="cuda", dtype=torch.int32).add_(1),
                "cat": torch.randperm(case["dim"], generator=g, device="cuda", dtype=torch.int32) % case["groups"],
                "groups": case["groups"],
                "fk": _ints(g, case["rows"], 1, case["dim"]), "m": _ints(g, case["rows"], 1, 10_000)}
    return {"cols": _lineitem(case, seed), "type": case["type"]}


def _lineitem(case, seed):
    """Tax, quantity and extended price of line items: doubles, or whole percents, pieces and cents."""
    g = _gen(seed)
    tax, qty, price = (_ints(g, case["rows"], lo, hi) for lo, hi in ((0, 8), (1, 50), (90_000, 10_500_000)))
    if case["type"] == "fixed":
        return tax, qty, price
    return tax.double() / 100, qty.double(), price.double() / 100


# ---- one pass --------------------------------------------------------------------

def _by_key(keys, sums, counts):
    order = torch.argsort(keys)
    return keys[order], sums[order], counts[order]


def run(state):
    s = state
    if "aggs" in s:
        return olapcore.starjoin_groupsum(*_star_args(s), aggs=s["aggs"], ctx=s["ctx"])
    if "oid" in s:
        n, dv = s["rows"], s["form"] == "dv"
        if dv:
            k = olapcore.join_cwm_dv(s["vec"], s["fk"], s["orders"], s["nd"], s["oid"], s["gid"], s["factor"], n)
            total = olapcore.agg_cwm_dv(s["oid"], s["gid"], k, s["m1"], s["m2"], n, s["groups"], group_vector=s["sums"])
            return k, s["oid"], s["gid"], s["sums"], total
        olapcore.join_cwm_sv(s["vec"], s["fk"], s["orders"], s["nd"], s["gid"], s["factor"], n)
        total = olapcore.agg_cwm_sv(s["gid"], n, s["m1"], s["m2"], s["groups"], group_vector=s["sums"])
        return s["gid"], s["sums"], total
    if "vec" in s:  # host arrays
        return olapcore.starjoin_groupsum(*_star_args(s))
    if "engine" in s:
        return s["engine"].run(s["queries"], s["fk"], s["m1"], s["m2"])[:2]
    if "data" in s:
        if len(s["queries"]) == 1:
            return q5.q5(s["ctx"], s["data"], *s["queries"][0])
        return q5.q5_batch(s["ctx"], s["data"], s["queries"])
    if "below" in s:
        rows = operators.select_rowids(s["col"], s["below"], operators.CMP_LT)
        return rows, operators.gather(rows, s["cols"])
    if "probe" in s:
        table = operators.HashTable(s["keys"].numel()).build(s["keys"], s["pay"])
        return table.probe_pairs(s["probe"]) if s["pairs"] else table.probe(s["probe"])
    if "vals" in s:
        return _by_key(*operators.group_hash(s["keys"], *s["vals"], max_groups=s["groups"]))
    if "dk" in s:
        rows, cat = operators.HashTable(s["dk"].numel()).build(s["dk"], s["cat"]).probe_pairs(s["fk"])
        (m,) = operators.gather(rows, [s["m"]])
        return _by_key(*operators.group_hash(cat, m, max_groups=s["groups"]))
    tax, qty, price = s["cols"]
    if s["type"] == "f64":
        return operators.aggalgo_f64(tax.numel(), tax, qty, price)
    return operators.aggalgo_fixed(price, qty, tax)


# ---- what a pass cannot do without -------------------------------------------------

def work(case):
    """Bytes: each input read once, each output written once.  Operations: a
    probe, compare or add for each value that takes part."""
    kind = case["kind"]
    if kind in ("star", "columnwise", "host"):
        n, groups = case["rows"], math.prod(_nums(case["groups"]))
        passing = n * math.prod(_nums(case["sele"], float))
        vec = sum(_nums(case["dims"]))
        if kind != "columnwise":
            return {"bytes": 24 * n + vec + 8 * groups * case.get("sums", 1), "flops": 5 * n}
        # the key columns; the list written and read back with its measures, or the vector and the measures
        more = passing * (2 * 10 + 8) if case["form"] == "dv" else 2 * 2 * n + 8 * n
        return {"bytes": 16 * n + vec + more + 8 * groups, "flops": 5 * n}
    if kind == "batch":
        return {"bytes": 24 * case["rows"] + 8 * sum(_nums(case["dims"])), "flops": 5 * case["rows"]}
    if kind == "q5":
        n = case["lines"]
        return {"bytes": 16 * n + 8 * (n // 4) + 4 * (n // 40) + 4 * (n // 600), "flops": 3 * n}
    if kind == "select":
        k = case["rows"] * case["share"]
        return {"bytes": 4 * case["rows"] + 4 * k + 8 * k * case["columns"], "flops": case["rows"]}
    if kind == "join":
        pairs = 8 * case["probe"] * case["match"] if case["pairs"] else 16
        return {"bytes": 8 * case["build"] + 4 * case["probe"] + pairs, "flops": case["build"] + case["probe"]}
    if kind == "group":
        return {"bytes": 4 * case["rows"] * (1 + case["values"]) + 20 * case["groups"], "flops": 2 * case["rows"]}
    if kind == "join_group":
        return {"bytes": 8 * case["dim"] + 8 * case["rows"] + 20 * case["groups"], "flops": 3 * case["rows"]}
    return {"bytes": (24 if case["type"] == "f64" else 12) * case["rows"], "flops": 4 * case["rows"]}


def exact(case, seed):
    """The double aggregation in plain torch; every other output is whole numbers, compared bit for bit."""
    if case["kind"] != "aggregate" or case["type"] != "f64":
        return None
    tax, qty, price = _lineitem(case, seed)
    net = price * qty
    return float((net * tax + net).sum().item())
