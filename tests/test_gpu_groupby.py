"""The group-by operator at the edges of its forms: P at the last size whose
slots fit shared memory and the first past it, row counts around the first
whose 512-thread blocks fill the GPU, partial last chunks, flags that allow no
16-byte load, and chunks with no, one, a few and all rows flagged.  Sums, occupied slots and their
keys against numpy; everything is whole numbers, so equal."""
import ctypes

import numpy as np
import pytest

from sycldb_gb300 import capi
from tests.gpu_util import dev, host, release, stream, zeros

pytestmark = pytest.mark.gpu

FILL = 152 * 512 * 16  # rows of one 512-thread block per SM


@pytest.mark.parametrize("P", [7, 8192, 8193, 100_000])
@pytest.mark.parametrize("n,pad", [(1, 0), (511, 0), (513, 1), (70_001, 0), (FILL - 512, 0), (FILL, 0), (FILL + 13, 3)])
def test_group_by_forms(P, n, pad):
    rng = np.random.default_rng(n + P)
    width = 7
    key = rng.integers(0, P // width, n).astype(np.int32)
    low = rng.integers(-3, -3 + width, n).astype(np.int32)
    val = rng.integers(-2**31, 2**31, n).astype(np.int32)
    L = capi.lib()
    for density in (0.0005, 0.004, 0.1, 1.0):
        flags = (rng.random(n) < density).astype(np.uint8) * np.uint8(3)
        sb, sums = zeros(P, np.uint64)
        ob, occ = zeros(P, np.uint32)
        kb, k0 = dev(np.full(P, -9, np.int32))
        lb, k1 = dev(np.full(P, -9, np.int32))
        cols = (ctypes.c_void_p * 2)(dev(low)[1], dev(key)[1])
        capi.check(L.sdb_groupby_sum(cols, (ctypes.c_int32 * 2)(-3, 0), (ctypes.c_int32 * 2)(-4 + width, P // width - 1), 2,
                                     dev(val)[1], dev(flags, pad)[1], n, P, (ctypes.c_void_p * 2)(k1, k0), sums, occ,
                                     stream()))
        slot = (low[flags != 0] + 3) + width * key[flags != 0]
        want = np.zeros(P, np.uint64)
        np.add.at(want, slot, val[flags != 0].astype(np.int64).view(np.uint64))
        there = np.bincount(slot, minlength=P)[:P] > 0
        assert np.array_equal(host(sb, sums, P, np.uint64), want)
        assert np.array_equal(host(ob, occ, P, np.uint32) != 0, there)
        assert np.array_equal(host(kb, k0, P, np.int32), np.where(there, np.arange(P) // width, -9))
        assert np.array_equal(host(lb, k1, P, np.int32), np.where(there, np.arange(P) % width - 3, -9))
        release()
