"""Which chains go to the sieve, and what it gives there.  A chain without a
specialised pass goes to it from the size on at which it is the faster one;
a variant asked for by name takes it at any size.  Sums, occupied slots and their
keys must equal the general pass's."""
import ctypes

import numpy as np
import pytest

from sycldb_gb300 import capi
from tests.gpu_util import dev, host, release, stream, zeros
from tests.test_gpu_late import run
from tests.test_gpu_sieve import AND, FULL, NONE, RANGE, SEMI, Chain, set_col

pytestmark = pytest.mark.gpu


def launches():
    return capi.lib().sdb_sieve_launches()


def make(rng, term, tests, probes, n, P=40):
    """`tests` interval tests, then `probes` (kind, entries) probes; a group-by
    of P values of one column."""
    d = capi.ChainDesc()
    d.n = n
    for k in range(tests):
        op = d.ops[k]
        op.kind, op.logic_op, op.lo, op.hi = RANGE, NONE if k == 0 else AND, 0, 59
        set_col(op.a, dev(rng.integers(0, 100, n).astype(np.int32))[1])
    for k, (kind, length) in enumerate(probes):
        op = d.ops[tests + k]
        op.kind, op.logic_op, op.lo, op.hi = kind, AND, 0, length - 1
        set_col(op.a, dev(rng.integers(-2, length, n).astype(np.int32))[1])
        live = rng.random(length) < 0.6
        if kind == SEMI:
            op.ht = dev(live.astype(np.uint8))[1]
        else:
            op.ht = dev(np.stack([live.astype(np.int32), rng.integers(0, 20, length).astype(np.int32)], 1).reshape(-1))[1]
            op.out_reg = k
    d.n_ops = tests + len(probes)
    d.terminal = term
    set_col(d.value, dev(rng.integers(-1000, 1000, n).astype(np.int32))[1])
    if term == capi.TERM_GROUPBY:
        d.n_keys, d.P = 1, P
        set_col(d.keys[0], dev(rng.integers(0, P, n).astype(np.int32))[1])
        d.key_min[0], d.key_max[0] = 0, P - 1
    return d


def results(d, launch):
    if d.terminal == capi.TERM_FLAGS:
        b, p = zeros(d.n, np.uint8)
        d.flags_out = p
        outs = [(b, p, d.n, np.uint8)]
    elif d.terminal == capi.TERM_SUM:
        b, p = zeros(1, np.uint64)
        d.sum_out = p
        outs = [(b, p, 1, np.uint64)]
    else:
        outs = []
        for field, t in (("out_sum", np.uint64), ("occ", np.uint32)):
            b, p = zeros(d.P, t)
            setattr(d, field, p)
            outs.append((b, p, d.P, t))
        b, p = dev(np.full(d.P, -77, np.int32))
        d.out_keys[0] = p
        outs.append((b, p, d.P, np.int32))
    st = launch()
    return st, [host(*o) for o in outs]


SUM, GROUP, FLAGS = capi.TERM_SUM, capi.TERM_GROUPBY, capi.TERM_FLAGS
PROBES = [(SEMI, 900), (FULL, 5000)]


@pytest.mark.parametrize("term,tests,probes,n,P,sieve", [
    (FLAGS, 1, [], (1 << 21) - 1, 0, False), (FLAGS, 1, [], 1 << 21, 0, True), (FLAGS, 1, [(SEMI, 900)], 1 << 21, 0, True),
    (GROUP, 1, [], (1 << 20) - 1, 40, False), (GROUP, 1, [], 1 << 20, 40, True), (GROUP, 0, [(SEMI, 900)], 1 << 20, 40, True),
    (GROUP, 0, [(FULL, 900)], 1 << 22, 40, False),
    (GROUP, 2, [], 1 << 20, 512, True), (GROUP, 2, [], 1 << 20, 513, False), (GROUP, 2, [], 1 << 20, 2048, False),
    (GROUP, 2, [], 1 << 20, 2049, True), (GROUP, 1, PROBES, (1 << 17) - 1, 40, False), (GROUP, 1, PROBES, 1 << 17, 40, True),
    (GROUP, 1, PROBES, (1 << 20) - 1, 1000, False),
    (GROUP, 1, PROBES + PROBES, 1000, 1000, True), (SUM, 1, PROBES + PROBES, 1000, 0, True),
    (SUM, 1, [], 1 << 23, 0, False), (SUM, 0, [(SEMI, 900)], 1 << 23, 0, False),
    (SUM, 1, [(SEMI, 900)], (1 << 23) - 1, 0, False), (SUM, 1, [(SEMI, 900)], 1 << 23, 0, True),
    (SUM, 1, PROBES, (1 << 20) - 1, 0, False), (SUM, 1, PROBES, 1 << 20, 0, True), (SUM, 0, PROBES, 1 << 20, 0, True),
    (SUM, 0, [(FULL, 900)] * 4, 1 << 21, 0, False)])
def test_route_and_results(term, tests, probes, n, P, sieve):
    L = capi.lib()
    d = make(np.random.default_rng(n + P), term, tests, probes, n, P)
    capi.force_chain_variant(-1)
    st0, want = results(d, lambda: L.sdb_fused_chain_variant(ctypes.byref(d), 0, stream()))
    assert L.sdb_chain_specialised(ctypes.byref(d)) == 0
    before = launches()
    st1, got = results(d, lambda: L.sdb_fused_chain(ctypes.byref(d), stream()))
    assert launches() - before == (1 if sieve else 0)
    assert st0 == st1 == capi.SDB_OK
    for w, g in zip(want, got):
        assert np.array_equal(w, g)
    release()


@pytest.mark.parametrize("n", [64 * 900 - 1, 64 * 900, 64 * 8 * 900 - 1, 64 * 8 * 900])
def test_sizes_around_the_first_bitmap(n):
    """The first sizes that pack a bitmap of 900 keys, and of 900 key/value entries."""
    L = capi.lib()
    for probes in ([(SEMI, 900)], [(FULL, 900), (SEMI, 70_000)]):
        d = make(np.random.default_rng(n), GROUP, 1, probes, n)
        st0, want = results(d, lambda: L.sdb_fused_chain_variant(ctypes.byref(d), 0, stream()))
        before = launches()
        st1, got = results(d, lambda: L.sdb_fused_chain_variant(ctypes.byref(d), 5, stream()))
        assert launches() - before == 1
        assert st0 == st1 == capi.SDB_OK and all(np.array_equal(w, g) for w, g in zip(want, got))
        release()


@pytest.mark.parametrize("n", [2049, 50_021])
def test_random_chains_reach_the_sieve_and_give_the_keys(n):
    rng = np.random.default_rng(n + 7)
    reached = {SUM: 0, GROUP: 0, FLAGS: 0}
    keyed = 0
    for _ in range(400):
        if min(reached.values()) >= 10 and keyed >= 20:
            break
        c = Chain(rng, n)
        d = c.d
        pass_ = (lambda v: run(d, v)) if d.terminal == GROUP else c.run
        st0, want = pass_(0)
        before = launches()
        st1, got = pass_(5)
        reached[d.terminal] += launches() - before
        assert st0 == st1 == capi.SDB_OK
        for w, g in zip(want[:2], got[:2]):
            assert np.array_equal(w, g)
        if d.terminal == GROUP:
            occ = want[1] != 0
            lo, hi = list(d.key_min)[:d.n_keys], list(d.key_max)[:d.n_keys]
            inside = all(((k[occ] >= a) & (k[occ] <= b)).all() for o in (want, got) for k, a, b in zip(o[2:], lo, hi))
            if inside:  # keys past their range share slots, whose first writer may differ
                keyed += 1
                for w, g in zip(want[2:], got[2:]):
                    assert np.array_equal(w, g)
        release()
    assert min(reached.values()) >= 10 and keyed >= 20, (reached, keyed)
