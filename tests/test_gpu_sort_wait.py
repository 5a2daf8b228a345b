"""A wait inside the device sort that runs out: the bounded look-back of a
pass gives up (at once, with a limit of no polls), the sort's order is 0..n-1
and counted as a device error, and an ORDER BY of the engine fails instead of
returning rows out of order.  The next sort is right again."""
import ctypes

import numpy as np
import pytest

from sycldb_gb300 import capi, plans
from sycldb_gb300.engine import Engine
from tests import datasets
from tests.gpu_util import dev, host, stream, zeros

pytestmark = pytest.mark.gpu


def device_errors():
    v = ctypes.c_uint64()
    capi.check(capi.lib().sdb_device_errors(ctypes.byref(v), stream()))
    return v.value


@pytest.mark.parametrize("n", [6145, 50_000])
@pytest.mark.parametrize("wide", [False, True])  # ordered by the head; by every digit
def test_sort_whose_wait_runs_out(n, wide):
    rng = np.random.default_rng(n)
    k = rng.integers(0, 1000, n).astype(np.int32)
    if wide:
        k = np.where(rng.random(n) < 0.9, 5, rng.integers(0, 2**62, n)).astype(np.uint64)
    L = capi.lib()
    ptrs, types, desc = (ctypes.c_void_p * 1)(dev(k)[1]), (ctypes.c_int * 1)(int(wide)), (ctypes.c_int * 1)(0)
    sb = L.sdb_sort_scratch_bytes(n)
    scratch = zeros(sb, np.uint8)[1]
    device_errors()
    pb, perm = zeros(n, np.uint32)
    capi.check(L.sdb_sort_rows_polls(ptrs, types, desc, 1, n, perm, scratch, sb, 0, stream()))
    assert np.array_equal(host(pb, perm, n, np.uint32), np.arange(n, dtype=np.uint32))
    assert device_errors() > 0
    capi.check(L.sdb_sort_rows(ptrs, types, desc, 1, n, perm, scratch, sb, stream()))
    assert np.array_equal(host(pb, perm, n, np.uint32), np.argsort(k, kind="stable").astype(np.uint32))
    assert device_errors() == 0


@pytest.mark.parametrize("segment_rows", [0, 1 << 14])
def test_order_by_whose_wait_runs_out_is_an_error(segment_rows):
    ds = datasets.dataset(0.05)
    b = plans.PlanBuilder()
    b.scan("lineorder")
    b.filter(plans.search(11, 2, 3))
    b.project([plans.col(5), plans.col(9)])
    b.sort([1, 0])
    plan = b.plan()
    with Engine(arena_bytes=1 << 30, segment_rows=segment_rows, order_by=True) as eng:
        for t, cols in ds.items():
            eng.load_table(t, cols)
        want = eng.execute(plan).rows()
        assert len(want) > 6144 and want == sorted(want, key=lambda r: (r[1], r[0]))
        capi.check(capi.lib().sdb_engine_set_sort_polls(eng._h, 0))
        with pytest.raises(capi.SdbError) as e:
            eng.execute(plan)
        assert e.value.status == capi.SDB_ERR_TIMEOUT
        capi.check(capi.lib().sdb_engine_set_sort_polls(eng._h, 1 << 20))
        assert eng.execute(plan).rows() == want
    device_errors()
