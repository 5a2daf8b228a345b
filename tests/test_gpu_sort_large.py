"""ORDER BY past the size at which a 32-bit head of the keys can decide the
order (rows of evenly spread keys share their head more often than the tied
runs are ordered for): every digit is sorted, and heads that hold the whole
keys still are enough."""
import ctypes

import pytest

from sycldb_gb300 import capi
from tests.gpu_util import stream, torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [True, False])
def test_sort_above_two_to_the_26_rows(wide):
    t = torch()
    n = (1 << 26) + 4097
    g = t.Generator(device="cuda").manual_seed(11)
    k0 = t.randint(-2**31, 2**31, (n,), dtype=t.int64, device="cuda", generator=g).to(t.int32)
    keys = [k0]
    if wide:  # a second key that ties of the first need
        k0 //= 4096
        keys.append(t.randint(0, 2**62, (n,), dtype=t.int64, device="cuda", generator=g))
    L = capi.lib()
    m = len(keys)
    need = L.sdb_sort_scratch_bytes(n)
    scratch = t.empty(need + 256, dtype=t.uint8, device="cuda")
    perm = t.empty(n, dtype=t.int32, device="cuda")
    capi.check(L.sdb_sort_rows((ctypes.c_void_p * m)(*[k.data_ptr() for k in keys]), (ctypes.c_int * m)(*range(m)),
                               (ctypes.c_int * m)(*[0] * m), m, n, perm.data_ptr(),
                               (scratch.data_ptr() + 255) // 256 * 256, need, stream()))
    want = t.arange(n, device="cuda")
    for k in reversed(keys):
        want = want[t.sort(k[want], stable=True).indices]
    assert t.equal(perm.long(), want)
    errors = ctypes.c_uint64()
    capi.check(L.sdb_device_errors(ctypes.byref(errors), stream()))
    assert errors.value == 0
