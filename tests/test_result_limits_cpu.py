"""A result segment of more than 2^31 rows is refused by the executor's
compactions (before any launch), as sdb_compact_row_ids refuses it: their
counts are 32-bit words."""
import ctypes

from sycldb_gb300 import capi

# int sdb_copy_rows(uint64_t, int, const void *const *, const int *, void *const *, uint32_t *, cudaStream_t)
COPY = "_Z13sdb_copy_rowsmiPKPKvPKiPKPvPjP11CUstream_st"
# int sdb_compact_gather_large(const void *, bool, uint64_t, int, const void *const *, const int *, void *const *,
#                              uint32_t *, void *, cudaStream_t)
GATHER = "_Z24sdb_compact_gather_largePKvbmiPKS0_PKiPKPvPjS5_P11CUstream_st"


def test_segments_above_two_to_the_31_rows_are_refused():
    L = capi.lib()
    none, wide = (ctypes.c_void_p * 1)(0), (ctypes.c_int * 1)(0)
    copy, gather = getattr(L, COPY), getattr(L, GATHER)
    copy.argtypes = [ctypes.c_uint64, ctypes.c_int] + [ctypes.c_void_p] * 5
    gather.argtypes = [ctypes.c_void_p, ctypes.c_bool, ctypes.c_uint64, ctypes.c_int] + [ctypes.c_void_p] * 6
    for n in ((1 << 31) + 1, 1 << 32, 1 << 40):
        assert copy(n, 1, none, wide, none, None, None) == capi.SDB_ERR_INVALID
        assert gather(None, False, n, 1, none, wide, none, None, None, None) == capi.SDB_ERR_INVALID
    assert capi.lib().sdb_compact_row_ids(0x1000, (1 << 31) + 1, 0x1000, 0x1000, 0x1000, 1 << 40,
                                          None) == capi.SDB_ERR_INVALID
