"""Ordered compaction at the edges of its tiles: the one-launch form
(sdb_compact_gather, _occ), row ids over several tiles (sdb_compact_row_ids),
and the executor's results above the one-launch limits."""
import ctypes

import numpy as np
import pytest

from sycldb_gb300 import capi, plans
from sycldb_gb300.engine import Engine
from tests import datasets
from tests.gpu_util import dev, host, stream, zeros

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 2047, 2048, 2049, 4097, 65535, 65536])
@pytest.mark.parametrize("share", [0.0, 0.01, 0.6, 1.0])
@pytest.mark.parametrize("occ,pad", [(False, 0), (False, 1), (True, 0), (True, 4)])
def test_one_launch_compaction(n, share, occ, pad):
    rng = np.random.default_rng(n)
    fl = (rng.random(n) < share) * rng.integers(1, 200, n)
    _, f = dev(fl.astype(np.uint32 if occ else np.uint8), pad)
    cols = [rng.integers(-2**31, 2**31 - 1, n, dtype=np.int64).astype(np.int32),
            rng.integers(0, 2**63, n).astype(np.uint64)]
    outs = [zeros(n, c.dtype) for c in cols]
    cb, cnt = zeros(1, np.uint32)
    src = (ctypes.c_void_p * 2)(*[dev(c)[1] for c in cols])
    dst = (ctypes.c_void_p * 2)(*[p for _, p in outs])
    wide = (ctypes.c_int * 2)(0, 1)
    entry = capi.lib().sdb_compact_gather_occ if occ else capi.lib().sdb_compact_gather
    capi.check(entry(f, n, 2, src, wide, dst, cnt, stream()))
    ids = np.flatnonzero(fl)
    assert int(host(cb, cnt, 1, np.uint32)[0]) == ids.size
    for (b, p), c in zip(outs, cols):
        assert np.array_equal(host(b, p, ids.size, c.dtype), c[ids])


@pytest.mark.parametrize("n", [4095, 4096, 4097, 16_385, 1 << 22, (1 << 22) + 1, 5_000_001, (1 << 26) + 17])
def test_row_ids_over_tiles(n):
    import torch

    L = capi.lib()
    g = torch.Generator(device="cuda").manual_seed(n)
    f = (torch.randint(0, 100, (n,), device="cuda", generator=g) < 7).to(torch.uint8)
    f[-1] = 1
    ids = torch.zeros(n, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    sb = L.sdb_compact_scratch_bytes(n)
    scratch = torch.empty(sb, dtype=torch.uint8, device="cuda")
    capi.check(L.sdb_compact_row_ids(f.data_ptr(), n, ids.data_ptr(), cnt.data_ptr(), scratch.data_ptr(), sb, stream()))
    want = torch.nonzero(f).flatten().to(torch.int32)
    assert int(cnt[0]) == want.numel()
    assert torch.equal(ids[:want.numel()], want)


@pytest.mark.parametrize("mode", ["plain", "prepared", "ordered"])
@pytest.mark.parametrize("seg", [0, 1 << 17])
def test_results_above_the_one_launch_limits(mode, seg):
    """A filter's rows over more than 65536 rows (one and several segments)
    and a group-by over more than 65536 slots."""
    ds = datasets.dataset(0.05)
    b = plans.PlanBuilder()
    b.scan("lineorder")
    b.filter(plans.expr("<", plans.col(8), plans.lit(20)))
    b.project([plans.col(5), plans.col(9)])
    b.sort([1])
    rows = b.plan()
    city = plans.plan_customer_supplier_date(0, 1992, 1997, (3, 17))
    with Engine(arena_bytes=1 << 30, segment_rows=seg, plan_cache=4 if mode == "prepared" else 0,
                order_by=mode == "ordered") as eng:
        for name, cols in ds.items():
            eng.load_table(name, cols)
        for plan in (rows, city):
            want = datasets.oracle_run(ds, plan, seg or (1 << 28))
            for _ in range(3 if mode == "prepared" else 1):
                got = eng.execute(plan)
                assert got.canonical() == want
            if mode == "ordered" and plan is rows:
                assert np.all(np.diff(got.columns[1].astype(np.int64)) >= 0)


@pytest.mark.parametrize("qty,seg", [(2, 0), (8, 0), (9, 0), (30, 0), (8, 1 << 17)])
def test_ordered_results_around_the_counted_sort_limit(qty, seg):
    """ORDER BY (descending price, then date) of a filter's rows: below, at
    about and above 4096 of them, and of a group-by; the same rows as without."""
    ds = datasets.dataset(0.05)
    b = plans.PlanBuilder()
    b.scan("lineorder")
    b.filter(plans.AND(plans.expr("<", plans.col(8), plans.lit(qty)), plans.search(11, 4, 5)))
    b.project([plans.col(5), plans.col(9)])
    b.rels.append({"id": len(b.rels), "relOp": "SORT",
                   "collation": [{"field": 1, "direction": "DESCENDING"}, {"field": 0, "direction": "ASCENDING"}]})
    rows, star = b.plan(), plans.plan_star(1, 3)
    with Engine(arena_bytes=1 << 30, segment_rows=seg, order_by=True) as eng, \
            Engine(arena_bytes=1 << 30, segment_rows=seg) as plain:
        for name, cols in ds.items():
            eng.load_table(name, cols)
            plain.load_table(name, cols)
        for _ in range(2):
            got, base = eng.execute(rows), plain.execute(rows)
            date, price = base.columns
            at = np.lexsort((date, -price.astype(np.int64)))  # stable: ties keep row order
            assert np.array_equal(got.columns[0], date[at]) and np.array_equal(got.columns[1], price[at])
            g, p = eng.execute(star), plain.execute(star)
            at = np.lexsort((p.columns[1], p.columns[0]))
            for x, y in zip(g.columns, p.columns):
                assert np.array_equal(x, y[at])


@pytest.mark.parametrize("seg", [0, 4096])
@pytest.mark.parametrize("join_tables", [0, 2])
def test_builds_in_one_launch_and_unfiltered_results(seg, join_tables):
    """Ad-hoc plans whose tables are built together: one to four of them, build
    sides of one and of several segments (a table's segments stay in order),
    direct and open-addressing tables; and results of every row, without
    flags."""
    ds = datasets.dataset(0.2)
    b = plans.PlanBuilder()
    b.scan("part")
    b.project([plans.col(4), plans.col(0)])
    every = b.plan()
    b = plans.PlanBuilder()
    b.scan("lineorder")
    b.project([plans.col(12)])
    b.aggregate([], 0)
    total = b.plan()
    pls = [plans.plan_date_join(1994), plans.plan_star(1, 3), plans.plan_star(2, 7, 1993, 1995, 9),
           plans.plan_customer_supplier_date(2), plans.plan_profit(1), every, total]
    with Engine(arena_bytes=1 << 30, segment_rows=seg, join_tables=join_tables) as eng:
        for name, cols in ds.items():
            eng.load_table(name, cols)
        for plan in pls:
            assert eng.execute(plan).canonical() == datasets.oracle_run(ds, plan, seg or (1 << 28))
