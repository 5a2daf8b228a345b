"""The late passes (variant 8 of the shapes that have one): chains of each
shape with operands of every kind, against the general pass.  Sums, occupied
slots and their group keys must be equal."""
import ctypes

import numpy as np
import pytest

from sycldb_gb300 import capi
from tests.gpu_util import dev, host, release, stream, zeros

pytestmark = pytest.mark.gpu

SELECT, RANGE, POINTS, SEMI, FULL, BINOP, FILL = range(7)
NONE, AND, OR = 0, 1, 2

# shape: (op kinds, terminal, incoming flags)
SHAPES = {
    "filter_sum": ((RANGE, RANGE, SELECT, BINOP), capi.TERM_SUM, False),
    "filter_sum3": ((RANGE, RANGE, RANGE, BINOP), capi.TERM_SUM, False),
    "date_join": ((RANGE, FULL, BINOP), capi.TERM_GROUPBY, False),
    "star": ((SEMI, FULL, FULL), capi.TERM_GROUPBY, False),
    "flight3": ((FULL, FULL, FULL), capi.TERM_GROUPBY, False),
    "flight4": ((FULL, FULL, BINOP), capi.TERM_GROUPBY, True),
}


def set_col(o, ptr):
    o.kind, o.col = capi.SRC_COL, ptr


def set_reg(o, r):
    o.kind, o.reg = capi.SRC_REG, r


def set_lit(o, v):
    o.kind, o.lit = capi.SRC_LIT, int(v)


def make(rng, shape, n, reg_at=None, hits=0.7):
    """A chain of the shape; op `reg_at` reads register 0 in place of a column."""
    kinds, term, flags = SHAPES[shape]
    d = capi.ChainDesc()
    d.n = n
    lens = (2500, 300, 900)
    cols = [dev(rng.integers(-3, lens[k % 3], n).astype(np.int32))[1] for k in range(3)]
    meas = dev(rng.integers(-2**31, 2**31, n).astype(np.int32))[1]
    if flags:
        d.flags_in = dev((rng.random(n) < hits).astype(np.uint8))[1]
    reg = 0
    for i, kind in enumerate(kinds):
        op = d.ops[i]
        op.kind, op.logic_op = kind, AND
        set_col(op.a, cols[i % 3])
        if kind in (RANGE, SELECT):
            # zero lies outside the range, so what an unwritten register gives
            # shows in the rows that pass
            op.lo, op.hi = 1, int(lens[i % 3] * hits)
            op.cmp_op = 4  # >
            set_lit(op.b, 0)
        elif kind in (SEMI, FULL):
            length = lens[i % 3]
            op.lo, op.hi = 0, length - 1
            live = (rng.random(length) < hits).astype(np.int32)
            live[0] = 0
            if kind == SEMI:
                op.ht = dev(live.astype(np.uint8))[1]
            else:
                op.ht = dev(np.stack([live, rng.integers(0, 20, length).astype(np.int32)], 1).reshape(-1))[1]
                op.out_reg = reg
                reg += 1
        else:
            set_col(op.a, meas)
            set_col(op.b, cols[0])
            op.bin_op = 0
            op.out_reg = reg
            reg += 1
        if i == reg_at:
            set_reg(op.a, 0)
    d.n_ops = len(kinds)
    d.terminal = term
    if kinds[-1] == BINOP:
        set_reg(d.value, reg - 1)
        reg -= 1
    else:
        set_col(d.value, meas)
    if term == capi.TERM_GROUPBY:
        d.n_keys, d.P = reg, 20 ** reg
        for q in range(reg):
            set_reg(d.keys[q], q)
            d.key_min[q], d.key_max[q] = 0, 19
    return d


def run(d, variant):
    """Status, sums, occupied slots and the keys of those."""
    outs = []
    if d.terminal == capi.TERM_SUM:
        b, p = zeros(1, np.uint64)
        d.sum_out = p
        outs.append((b, p, 1, np.uint64))
    else:
        for field, t in (("out_sum", np.uint64), ("occ", np.uint32)):
            b, p = zeros(d.P, t)
            setattr(d, field, p)
            outs.append((b, p, d.P, t))
        for q in range(d.n_keys):
            b, p = dev(np.full(d.P, -77, np.int32))
            d.out_keys[q] = p
            outs.append((b, p, d.P, np.int32))
    st = capi.lib().sdb_fused_chain_variant(ctypes.byref(d), variant, stream())
    return st, [host(*o) for o in outs]


def same(d, variants=(4, 5, 7, 8)):
    st0, want = run(d, 0)
    assert st0 == capi.SDB_OK
    for v in variants:
        st, got = run(d, v)
        assert st == capi.SDB_OK
        for w, g in zip(want, got):
            assert np.array_equal(w, g), v
    return want


@pytest.mark.parametrize("shape,reg_at", [("filter_sum", 0), ("filter_sum", 1), ("filter_sum3", 0), ("date_join", 0),
                                          ("star", 0)])
@pytest.mark.parametrize("n", [2048, 60_013])
def test_dense_op_reads_an_unwritten_register(shape, reg_at, n):
    """An op of the dense level that reads a register nothing has written
    reads zero, as in every other pass (the late passes hold columns there
    alone, and leave such chains to them)."""
    want = same(make(np.random.default_rng(n + reg_at), shape, n, reg_at))
    assert not any(w.any() for w in want[:2])  # no row passes
    release()


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("n", [1, 2047, 60_013])
def test_every_shape_gives_the_sums_and_the_keys(shape, n):
    """Each shape at the edges of its tiles, a few, most and all of the rows
    left: sums, occupied slots and the keys their first writers store."""
    for hits in (0.05, 0.7, 1.0):
        d = make(np.random.default_rng(n), shape, n, hits=hits)
        same(d)
        release()
