"""The sieve pass (csrc/sieve.cuh): random chains of the forms it accepts and
of forms near them, run with the variant that reaches it and with the general
pass; sums, groups and flags must be equal."""
import ctypes

import numpy as np
import pytest

from sycldb_gb300 import capi
from tests.gpu_util import dev, host, release, stream, zeros

pytestmark = pytest.mark.gpu

SELECT, RANGE, POINTS, SEMI, FULL, BINOP, FILL = range(7)
NONE, AND, OR = 0, 1, 2
BIG = (1 << 18) + 5  # entries of a table past the shared-memory bitmap


def set_col(o, ptr):
    o.kind, o.col = capi.SRC_COL, ptr


def set_reg(o, r):
    o.kind, o.reg = capi.SRC_REG, r


def set_lit(o, v):
    o.kind, o.lit = capi.SRC_LIT, int(v)


class Chain:
    """A chain over n rows drawn from `rng`."""

    def __init__(self, rng, n):
        L = capi.lib()
        d = self.d = capi.ChainDesc()
        self.n = d.n = n
        cols = []
        for k in range(6):
            lo, hi = [(0, 99), (-5, 5), (0, 2999), (-40_000, BIG - 40_000), (-2**31, 2**31 - 1), (7, 7)][k]
            a = rng.integers(lo, hi, n, dtype=np.int64, endpoint=True).astype(np.int32)
            pad = 4 if rng.random() < 0.05 else 0  # a column that the ring cannot copy
            cols.append(dev(a, pad)[1])
        pick = lambda: int(rng.integers(0, 6))
        if rng.random() < 0.4:
            d.flags_in = dev((rng.random(n) < 0.6).astype(np.uint8) * rng.integers(1, 4, n).astype(np.uint8),
                             int(rng.integers(0, 2)))[1]
        regs, i = [], 0
        n_ops = int(rng.integers(1, 8))
        term = rng.choice([capi.TERM_SUM, capi.TERM_GROUPBY, capi.TERM_GROUPBY, capi.TERM_FLAGS])

        def operand(o):
            if regs and rng.random() < 0.15:
                set_reg(o, int(rng.choice(regs)))
            else:
                set_col(o, cols[pick()])

        for i in range(n_ops):
            op = d.ops[i]
            op.kind = kind = int(rng.choice([SELECT, SELECT, RANGE, POINTS, SEMI, FULL, BINOP, FILL],
                                            p=[.2, .1, .15, .05, .2, .2, .07, .03]))
            op.logic_op = AND
            if kind in (SELECT, RANGE, POINTS):
                if i == 0 and rng.random() < 0.6:
                    op.logic_op = NONE
                elif rng.random() < (0.3 if i < 2 else 0.03):
                    op.logic_op = OR
                operand(op.a)
                op.cmp_op = int(rng.integers(0, 6))
                lo = int(rng.integers(-10, 80))
                op.lo, op.hi = lo, lo + int(rng.integers(-2, 3000))
                if rng.random() < 0.25:
                    operand(op.b)
                else:
                    set_lit(op.b, rng.choice([0, 1, 50, 7, -2**31, 2**31 - 1]))
            elif kind in (SEMI, FULL):
                c = int(rng.choice([1, 2, 2, 3]))
                set_col(op.a, cols[c])
                if regs and rng.random() < 0.1:
                    set_reg(op.a, int(rng.choice(regs)))
                op.lo = [0, -5, 0, -40_000][c]
                length = [0, 9, 2500, BIG][c]
                op.hi = op.lo + length - 1
                live = (rng.random(length) < 0.5).astype(np.uint8)
                key = np.arange(op.lo, op.lo + length, dtype=np.int32)
                if rng.random() < 0.15:  # open addressing
                    op.ht_log2 = L.sdb_oa_log2_slots(length)
                    words = (2 if kind == FULL else 1) << op.ht_log2
                    op.ht = zeros(words, np.int32)[1]
                    val = dev(rng.integers(0, 20, length).astype(np.int32))[1]
                    if kind == FULL:
                        capi.check(L.sdb_ht_build_kv_oa(dev(key)[1], val, dev(live)[1], length, op.ht, op.ht_log2, op.lo,
                                                        op.hi, 1, stream()))
                    else:
                        capi.check(L.sdb_ht_build_keys_oa(dev(key)[1], dev(live)[1], length, op.ht, op.ht_log2, op.lo,
                                                          op.hi, 1, stream()))
                elif kind == FULL:
                    t = np.stack([live.astype(np.int32), rng.integers(0, 20, length).astype(np.int32)], 1).reshape(-1)
                    op.ht = dev(np.ascontiguousarray(t))[1]
                else:
                    op.ht = dev(live)[1]
            elif kind == BINOP:
                operand(op.a)
                operand(op.b)
                op.bin_op = int(rng.integers(0, 4))
            else:
                set_lit(op.a, rng.integers(0, 20))
            if kind in (FULL, BINOP, FILL):
                reuse = regs and rng.random() < 0.03  # a register written twice
                op.out_reg = int(rng.choice(regs)) if reuse else len(regs)
                if not reuse:
                    regs.append(op.out_reg)
        d.n_ops = n_ops
        d.terminal = int(term)
        operand(d.value)
        if term == capi.TERM_GROUPBY:
            d.n_keys = int(rng.integers(1, 4))
            d.P = 1
            small = [c for c in (0, 1)]
            for q in range(d.n_keys):
                if regs and rng.random() < 0.6:
                    set_reg(d.keys[q], int(rng.choice(regs)))
                    d.key_min[q], d.key_max[q] = 0, 19
                else:
                    c = int(rng.choice(small))
                    set_col(d.keys[q], cols[c])
                    d.key_min[q], d.key_max[q] = ((0, 99), (-5, 5))[c]
                d.P *= d.key_max[q] - d.key_min[q] + 1

    def run(self, variant):
        """(status, outputs) of one pass."""
        d, outs = self.d, []
        if d.terminal == capi.TERM_SUM:
            b, p = zeros(1, np.uint64)
            d.sum_out = p
            outs.append((b, p, 1, np.uint64))
        elif d.terminal == capi.TERM_GROUPBY:
            for field, t in (("out_sum", np.uint64), ("occ", np.uint32)):
                b, p = zeros(d.P, t)
                setattr(d, field, p)
                outs.append((b, p, d.P, t))
            for q in range(d.n_keys):
                d.out_keys[q] = zeros(d.P, np.int32)[1]
        else:
            b, p = zeros(self.n, np.uint8)
            d.flags_out = p
            outs.append((b, p, self.n, np.uint8))
        st = capi.lib().sdb_fused_chain_variant(ctypes.byref(d), variant, stream())
        return st, [host(*o) for o in outs]


@pytest.mark.parametrize("n", [1, 31, 2047, 2048, 2049, 50_021, 700_001])
def test_sieve_equals_the_general_pass(n):
    rng = np.random.default_rng(n)
    for _ in range(60 if n < 100_000 else 25):
        c = Chain(rng, n)
        st0, want = c.run(0)
        st1, got = c.run(5)
        assert st0 == st1 == capi.SDB_OK
        for w, g in zip(want, got):
            assert np.array_equal(w, g), [(c.d.ops[k].kind, c.d.ops[k].logic_op) for k in range(c.d.n_ops)]
        release()


@pytest.mark.parametrize("shape", ["star", "flight3", "full2"])
@pytest.mark.parametrize("variant", [4, 7, 8])
def test_probes_that_share_a_register(shape, variant):
    """Chains of the specialised shapes whose probes write one register: the
    last one's value is the row's, whatever order a pass probes in."""
    rng = np.random.default_rng(5)
    n = 60_013
    c = Chain.__new__(Chain)
    d = c.d = capi.ChainDesc()
    c.n = d.n = n
    kinds = {"star": [SEMI, FULL, FULL], "flight3": [FULL, FULL, FULL], "full2": [FULL, FULL]}[shape]
    for i, kind in enumerate(kinds):
        length = (2500, 300, 900)[i]
        col = dev(rng.integers(0, length, n).astype(np.int32))[1]
        op = d.ops[i]
        op.kind, op.lo, op.hi, op.logic_op = kind, 0, length - 1, AND
        set_col(op.a, col)
        live = rng.random(length) < 0.7
        if kind == SEMI:
            op.ht = dev(live.astype(np.uint8))[1]
        else:
            op.ht = dev(np.stack([live.astype(np.int32), rng.integers(0, 20, length).astype(np.int32)], 1).reshape(-1))[1]
            op.out_reg = 0
    d.n_ops = len(kinds)
    d.terminal = capi.TERM_GROUPBY
    set_col(d.value, dev(rng.integers(-1000, 1000, n).astype(np.int32))[1])
    d.n_keys, d.P = 1, 20
    set_reg(d.keys[0], 0)
    d.key_min[0], d.key_max[0] = 0, 19
    st0, want = c.run(0)
    st1, got = c.run(variant)
    assert st0 == st1 == capi.SDB_OK and all(np.array_equal(w, g) for w, g in zip(want, got))
    release()
