"""Performance cases: the work a user has this framework do, through its
public entry points (``Engine.execute``, ``Engine.batch``,
``Engine.load_table`` and the C ABI's ``sdb_sort_rows``).

A case is a dict of plain values.  Its ``kind`` is one of

* ``query``  one plan executed on resident tables.  ``mode`` says how:
  ``prepared`` (an engine with a plan cache that has seen the plan: a
  dashboard's repeated query), ``adhoc`` (a default engine, the plan parsed
  and planned on every call), ``operators`` (fusion off: one kernel per
  operator, the path of a program that binds the operator kernels one by
  one).  ``order_by`` has the engine order the result rows on the device.
* ``batch``  many star-join plans with their own constants, prepared once and
  run together, each over its own fact partition (``shared`` = False) or all
  over one fact table, star joins, date joins and filter-sums mixed
  (``shared`` = True).
* ``load``   fact columns in pinned host memory registered and queried: the
  end-to-end step of a program whose data lives on the host.
* ``sort``   ORDER BY of row ids by one to three key columns.

Fact sizes run from 100 thousand rows (a test database, SF 1/60) to 120
million (SF 20, the benchmark's size); dimensions scale with them.  Columns
come from the repository's seeded generator with the benchmark's value ranges.
Another seed gives other prices, revenues and costs and starts the fact rows'
keys and filter columns at another row, so that a plan, whose constants belong
to the case, keeps the number of its result rows.
"""
from __future__ import annotations

import ctypes
import json
import math
import random

import numpy as np
import torch

from sycldb_gb300 import capi, plans, ssb, workloads
from sycldb_gb300.engine import Engine


# ------------------------------------------------------------------ plans
def _profit_by(left_key, region, nation_filter):
    """SSB flights 4.2 and 4.3: four joins, three group-by keys.  4.2 groups
    profit by (year, supplier nation, part category) for one region of
    customers and suppliers and two manufacturers; 4.3 by (year, supplier
    city, part brand) for one supplier nation and one part category.  Both
    keep two years."""
    b = plans.PlanBuilder()
    f = b.scan("lineorder")
    c = b.scan("customer")
    c = b.filter(plans.expr("==", plans.col(5), plans.lit(region)))
    j1 = b.join(f, c, 2, 17, "semi")          # 17 + 8 = 25 columns
    s = b.scan("supplier")
    if nation_filter is None:
        s = b.filter(plans.expr("==", plans.col(5), plans.lit(region)))
    else:
        s = b.filter(plans.expr("==", plans.col(4), plans.lit(nation_filter)))
    j2 = b.join(j1, s, 4, 25)                 # supplier -> 25..31
    p = b.scan("part")
    if nation_filter is None:
        p = b.filter(plans.search_points(2, 0, 1))
    else:
        p = b.filter(plans.expr("==", plans.col(3), plans.lit(left_key)))
    j3 = b.join(j2, p, 3, 32)                 # part -> 32..40
    d = b.scan("ddate")
    d = b.filter(plans.search(4, 1997, 1998))
    b.join(j3, d, 5, 41)                      # ddate -> 41..57
    s_key, p_key = (4, 3) if nation_filter is None else (3, 4)
    b.project([plans.col(41 + 4), plans.col(25 + s_key), plans.col(32 + p_key),
               plans.expr("-", plans.col(12), plans.col(13))])
    b.aggregate([0, 1, 2], 3)
    b.sort([0, 1, 2])
    return b.plan()


def _select_rows(discount, quantity):
    """Rows of a fact filter returned to the host (no aggregate)."""
    b = plans.PlanBuilder()
    b.scan("lineorder")
    b.filter(plans.AND(plans.expr("==", plans.col(11), plans.lit(discount)),
                       plans.expr("<", plans.col(8), plans.lit(quantity))))
    b.project([plans.col(5), plans.col(9)])
    return b.plan()


def _filter_group(discount_lo):
    """A group-by of the fact table alone: revenue by quantity for a range of
    discounts."""
    b = plans.PlanBuilder()
    b.scan("lineorder")
    b.filter(plans.search(11, discount_lo, discount_lo + 2))
    b.project([plans.col(8), plans.col(12)])
    b.aggregate([0], 1)
    b.sort([0])
    return b.plan()


# plan name -> (fact columns, {dimension: columns read}, plan from a random.Random)
QUERIES = {
    # SSB flight 1 as the reference plans it: filters on the fact table, SUM
    "filter_sum": ((5, 8, 9, 11), {},
                   lambda r: plans.plan_filter_sum(r.randint(1992, 1998), 1, 3, 25)),
    # one join and a group by year
    "date_join": ((5, 9, 11), {"ddate": 2},
                  lambda r: plans.plan_date_join(r.randint(1992, 1997), 4, 6)),
    # SSB flight 2
    "star": ((3, 4, 5, 12), {"supplier": 2, "part": 3, "ddate": 2},
             lambda r: plans.plan_star(r.randint(0, 4), r.randint(0, 24))),
    # SSB flight 3.1 (nations) and 3.3 (two cities on each side)
    "flight3": ((2, 4, 5, 12), {"customer": 3, "supplier": 3, "ddate": 2},
                lambda r: plans.plan_customer_supplier_date(r.randint(0, 4))),
    "flight3_city": ((2, 4, 5, 12), {"customer": 2, "supplier": 2, "ddate": 2},
                     lambda r: plans.plan_customer_supplier_date(0, 1992, 1997, sorted(r.sample(range(250), 2)))),
    # SSB flights 4.1, 4.2 and 4.3
    "flight41": ((2, 3, 4, 5, 12, 13), {"customer": 3, "supplier": 2, "part": 2, "ddate": 2},
                 lambda r: plans.plan_profit(r.randint(0, 4))),
    "flight42": ((2, 3, 4, 5, 12, 13), {"customer": 2, "supplier": 3, "part": 3, "ddate": 2},
                 lambda r: _profit_by(0, r.randint(0, 4), None)),
    "flight43": ((2, 3, 4, 5, 12, 13), {"customer": 2, "supplier": 3, "part": 3, "ddate": 2},
                 lambda r: _profit_by(r.randint(0, 24), r.randint(0, 4), r.randint(0, 24))),
    "select_rows": ((5, 8, 9, 11), {}, lambda r: _select_rows(r.randint(0, 10), 3)),
    "filter_group": ((8, 11, 12), {}, lambda r: _filter_group(r.randint(0, 8))),
}

# sort key sets: (type, low, high, descending); int32 keys compare signed,
# uint64 unsigned
SORT_KEYS = {
    "value_sum": ((0, -2**31, 2**31 - 1, False), (1, 0, 2**62, True)),
    "year_revenue": ((0, 1992, 1998, False), (1, 0, 2**40, True)),
    "brand": ((0, 0, 999, False),),
    "nations_year_sum": ((0, 0, 24, False), (0, 0, 24, False), (1, 0, 2**44, True)),
}


def listed():
    return [
        # the smallest call: an ad-hoc star join over a test-sized database
        {"name": "star_600k_adhoc", "kind": "query", "query": "star", "rows": 600_000, "mode": "adhoc", "order_by": False},
        # SF1 dashboard queries, repeated: filter-project-sum and the date join
        {"name": "filter_sum_sf1", "kind": "query", "query": "filter_sum", "rows": 6_000_000, "mode": "prepared",
         "order_by": False},
        {"name": "date_join_sf1", "kind": "query", "query": "date_join", "rows": 6_000_000, "mode": "prepared",
         "order_by": False},
        # the benchmark's headline: the SF20 star join, repeated
        {"name": "star_sf20", "kind": "query", "query": "star", "rows": 120_000_000, "mode": "prepared",
         "order_by": False},
        # SSB flight 3 at SF20: three joins, three group-by keys
        {"name": "flight3_sf20", "kind": "query", "query": "flight3", "rows": 120_000_000, "mode": "prepared",
         "order_by": False},
        # SSB flight 3.3 asked once, its rows ordered: a sparse group-by over a large key space, a ragged fact size
        {"name": "flight33_ordered", "kind": "query", "query": "flight3_city", "rows": 29_999_987, "mode": "adhoc",
         "order_by": True},
        # SSB flight 4.2 at SF10: four joins over six fact columns
        {"name": "flight42_sf10", "kind": "query", "query": "flight42", "rows": 60_000_000, "mode": "prepared",
         "order_by": False},
        # the operator kernels one by one
        {"name": "star_operators", "kind": "query", "query": "star", "rows": 30_000_000, "mode": "operators",
         "order_by": False},
        # a filter whose rows come back to the host
        {"name": "select_rows_sf5", "kind": "query", "query": "select_rows", "rows": 30_000_000, "mode": "adhoc",
         "order_by": False},
        # the batched configuration: 64 star joins over uneven partitions, 636 M fact rows
        {"name": "batch_64", "kind": "batch", "plans": 64, "median_rows": 7_000_000, "shared": False},
        # host data: four fact columns from pinned memory, then the star join on them
        {"name": "load_star_sf2", "kind": "load", "rows": 12_000_000},
        # ORDER BY by a value and a 64-bit sum
        {"name": "order_by_16m", "kind": "sort", "rows": 1 << 24, "keys": "value_sum"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query"] * 6 + ["batch", "batch", "load", "sort"])
    if kind == "query":
        mode = rng.choice(["prepared", "adhoc", "adhoc", "operators"])
        most = 30_000_000 if mode == "operators" else 120_000_000
        return {"kind": kind, "query": rng.choice(sorted(QUERIES)), "rows": _log_int(rng, 100_000, most), "mode": mode,
                "order_by": mode == "adhoc" and rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "plans": _log_int(rng, 2, 64), "median_rows": _log_int(rng, 200_000, 7_000_000),
                "shared": rng.random() < 0.5}
    if kind == "load":
        return {"kind": kind, "rows": _log_int(rng, 100_000, 12_000_000)}
    return {"kind": kind, "rows": _log_int(rng, 1_000, 1 << 24), "keys": rng.choice(sorted(SORT_KEYS))}


# ------------------------------------------------------------------ states
def _sf(rows):
    return max(rows / 6e6, 0.02)


MEASURES = (9, 12, 13)  # extendedprice, revenue, supplycost


def _fact(rows, cols, sf, seed, salt=0):
    """Device fact columns: the measures of ``seed``, the other columns of the
    repository's seed starting at a row of ``seed``'s choice (the same rows in
    another place)."""
    fact = ssb.gen_lineorder_device(rows, [c for c in cols if c not in MEASURES], sf, salt=salt)
    shift = random.Random(seed).randrange(rows)
    fact = {c: torch.roll(t, shift) for c, t in fact.items()}
    fact.update(ssb.gen_lineorder_device(rows, [c for c in cols if c in MEASURES], sf, seed=seed, salt=salt))
    torch.cuda.synchronize()
    return {c: fact[c] for c in cols}


def _load_dims(eng, dims, names):
    for t in sorted(names):
        eng.load_table(t, dims[t])


def _batch_parts(case):
    """Fact rows of each plan of a batch and its star-join constants: the
    lognormal partitions of the batched workload."""
    med = case["median_rows"]
    return workloads.batch_workload(case["plans"], lo=max(med // 7, 1000), hi=med * 7, median=med,
                                    dim_sf=_sf(med * 17))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "query":
        cols, dims, plan = QUERIES[case["query"]]
        sf = _sf(case["rows"])
        eng = Engine(fuse=case["mode"] != "operators", plan_cache=8 if case["mode"] == "prepared" else 0,
                     order_by=case["order_by"])
        eng.load_table("lineorder", _fact(case["rows"], cols, sf, seed))
        if dims:
            _load_dims(eng, ssb.gen_dims(sf), dims)
        text = json.dumps(plan(random.Random(case["rows"])))
        if case["mode"] == "prepared":  # a repeated query: the engine has prepared it on its second execution
            eng.execute(text)
            eng.execute(text)
        return {"kind": kind, "engine": eng, "plan": text}
    if kind == "batch":
        wl = _batch_parts(case)
        eng = Engine()
        _load_dims(eng, ssb.gen_dims(wl.dim_sf), ("supplier", "part", "ddate"))
        if case["shared"]:
            eng.load_table("lineorder", _fact(case["median_rows"], (3, 4, 5, 8, 9, 11, 12), wl.dim_sf, seed))
            texts = [json.dumps(q.plan) for q in workloads.poisson_stream(1000.0, case["plans"])]
        else:
            for p, n in enumerate(wl.rows):
                eng.load_table(wl.table(p), _fact(n, workloads.STAR_COLS, wl.dim_sf, seed, salt=p + 1))
            texts = [json.dumps(p) for p in wl.plans()]
        return {"kind": kind, "engine": eng, "batch": eng.batch(texts)}
    if kind == "load":
        cols, dims, plan = QUERIES["star"]
        sf = _sf(case["rows"])
        dev = _fact(case["rows"], cols, sf, seed)
        host = {c: t.cpu().pin_memory() for c, t in dev.items()}
        eng = Engine(plan_cache=8)
        _load_dims(eng, ssb.gen_dims(sf), dims)
        st = {"kind": kind, "engine": eng, "pinned": host, "columns": {c: t.numpy() for c, t in host.items()},
              "plan": json.dumps(plan(random.Random(case["rows"])))}
        run(st)
        run(st)
        return st
    n = case["rows"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    keys = []
    for typ, lo, hi, _desc in SORT_KEYS[case["keys"]]:
        keys.append(torch.randint(lo, hi + 1, (n,), dtype=torch.int64, device="cuda", generator=g))
        if typ == 0:
            keys[-1] = keys[-1].to(torch.int32)
    spec = SORT_KEYS[case["keys"]]
    need = capi.lib().sdb_sort_scratch_bytes(n)
    scratch = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
    return {"kind": kind, "keys": keys, "n": n, "perm": torch.empty(n, dtype=torch.int32, device="cuda"),
            "scratch": scratch, "scratch_ptr": (scratch.data_ptr() + 255) // 256 * 256, "need": need,
            "ptrs": (ctypes.c_void_p * len(keys))(*[k.data_ptr() for k in keys]),
            "types": (ctypes.c_int * len(keys))(*[s[0] for s in spec]),
            "desc": (ctypes.c_int * len(keys))(*[1 if s[3] else 0 for s in spec])}


def run(state):
    kind = state["kind"]
    if kind == "query":
        return state["engine"].execute(state["plan"]).columns
    if kind == "batch":
        # every plan's rows, column by column (star plans give three columns,
        # date joins two, filter-sums one), and how many rows each plan has
        res = state["batch"].run()
        return {"rows": np.array([r.nrows for r in res]),
                "columns": [np.concatenate([r.columns[-1 - c].view(np.int64) if c == 0 else r.columns[-1 - c]
                                            for r in res if len(r.columns) > c])
                            for c in range(max(len(r.columns) for r in res))]}
    if kind == "load":
        state["engine"].load_table("lineorder", state["columns"])
        return state["engine"].execute(state["plan"]).columns
    capi.check(capi.lib().sdb_sort_rows(state["ptrs"], state["types"], state["desc"], len(state["ptrs"]), state["n"],
                                        state["perm"].data_ptr(), state["scratch_ptr"], state["need"],
                                        torch.cuda.current_stream().cuda_stream or None))
    return state["perm"]


# ------------------------------------------------------------------ what a pass cannot do without
def _dim_bytes(dims, sf):
    return sum(4 * k * ssb.dim_rows(t, sf) for t, k in dims.items())


def work(case):
    """Every referenced column read once, every result written once (group-by
    results are a few kilobytes and left out)."""
    kind = case["kind"]
    if kind in ("query", "load"):
        cols, dims, _ = QUERIES["star" if kind == "load" else case["query"]]
        b = 4 * len(cols) * case["rows"] + _dim_bytes(dims, _sf(case["rows"]))
        if kind == "query" and case["query"] == "select_rows":
            b += int(case["rows"] / 11 * 2 / 50) * 8
        return {"bytes": b, "flops": 0}
    if kind == "batch":
        wl = _batch_parts(case)
        if not case["shared"]:
            return {"bytes": wl.algorithmic_bytes(), "flops": 0}
        # one shared table: its seven columns once, each plan's dimensions
        return {"bytes": 28 * case["median_rows"] + _dim_bytes(QUERIES["star"][1], wl.dim_sf), "flops": 0}
    key_bytes = sum(8 if s[0] else 4 for s in SORT_KEYS[case["keys"]])
    return {"bytes": (key_bytes + 4) * case["rows"], "flops": 0}
