"""Failure paths, made on the host (include/kache_b200_testing.h), none of which faults or hangs the GPU:

- a device or page-locked allocation that fails surfaces as KACHE_ENOMEM, from kache_new and from an insert that
  needs staging memory, and the table answers correctly once allocations succeed again;
- an insert whose operation must see a racing inserter's value first (KACHE_ASSIGN) meets a claim that is never
  published: the kernel's bounded wait runs out, the kernel ends, and the call returns KACHE_EINTERNAL; an operation
  that commutes (KACHE_ADD) applies itself without waiting and succeeds."""
import ctypes
import time

import numpy as np
import pytest

import kache
import oracle
import synth
from kache import Batch, Options

pytestmark = pytest.mark.gpu


def test_allocation_failure_is_enomem():
    L = kache.lib()
    o = Options(31, 8, 100_000, 0.8, 16, 0)
    h = ctypes.c_void_p()
    try:
        assert L.kache_b200_testing_fail_allocation(0) == kache.KACHE_OK
        assert L.kache_new(ctypes.byref(o), ctypes.byref(h)) == kache.KACHE_ENOMEM and not h.value
    finally:
        L.kache_b200_testing_fail_allocation(-1)
    assert L.kache_new(ctypes.byref(o), ctypes.byref(h)) == kache.KACHE_OK
    L.kache_free(h)

    # An insert into a fresh set, whose first call allocates its staging memory: every allocation of the call in turn
    # fails, until the call gets through; inserting the keys again then leaves the set the oracle makes.
    g = synth.genome(300_000, seed=71)
    b = Batch(*synth.reads_fixed(g, 20_000, 150, seed=72))
    T = kache.Table(31, 0, 400_000)
    u = T.register()
    codes = []
    for after in range(64):
        L.kache_b200_testing_fail_allocation(after)
        r = ctypes.c_uint64()
        codes.append(L.kache_insert(T.h, u, *b.args(), kache.KEEP, 0, ctypes.byref(r)))
        L.kache_b200_testing_fail_allocation(-1)
        if codes[-1] == kache.KACHE_OK:
            break
    assert codes[0] == kache.KACHE_ENOMEM and codes[-1] == kache.KACHE_OK
    assert set(codes[:-1]) == {kache.KACHE_ENOMEM}
    T.insert(u, b)
    O = oracle.OracleTable(31, 0, 400_000)
    O.insert(O.register(), b)
    assert np.array_equal(T.dump()[0], O.dump()[0])
    f, _, _ = T.lookup(b, values=False, fwd=False)
    fo, _, _ = O.lookup(b)
    assert np.array_equal(f, fo)
    T.close()


def _planted(op, wait_polls=1000):
    """A map with some keys, a k-mer of a new read claimed and left unpublished, then an insert of that read."""
    g = synth.genome(100_000, seed=73)
    T = kache.Table(31, 8, 200_000)
    u = T.register()
    T.insert(u, Batch(*synth.reads_fixed(g, 2000, 150, seed=74)), kache.ADD, 1)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    rng = np.random.default_rng(75)
    read = acgt[rng.integers(0, 4, 60)].tobytes()
    assert kache.lib().kache_b200_testing_plant_claim(T.h, read[10:41], wait_polls) == kache.KACHE_OK
    r = ctypes.c_uint64()
    t0 = time.perf_counter()
    code = kache.lib().kache_insert(T.h, u, *Batch.of([read]).args(), op, 5, ctypes.byref(r))
    return code, time.perf_counter() - t0, T


def test_unpublished_claim_ends_the_wait_with_einternal():
    code, seconds, T = _planted(kache.ASSIGN)
    assert code == kache.KACHE_EINTERNAL
    assert seconds < 30     # The kernel ended on its own bound.
    T.close()


def test_commuting_insert_does_not_wait():
    code, _, T = _planted(kache.ADD)
    assert code == kache.KACHE_OK
    T.close()


def test_plant_rejects_present_and_invalid_kmers():
    g = synth.genome(50_000, seed=76)
    b = Batch(*synth.reads_fixed(g, 500, 150, seed=77))
    T = kache.Table(31, 8, 100_000)
    T.insert(T.register(), b, kache.ADD, 1)
    L = kache.lib()
    present = bytes(b.bases[int(b.off[0]):int(b.off[0]) + 31])
    if b"N" not in present:
        assert L.kache_b200_testing_plant_claim(T.h, present, 10) == kache.KACHE_EINVAL
    assert L.kache_b200_testing_plant_claim(T.h, b"ACGTN" * 7, 10) == kache.KACHE_EINVAL
    assert L.kache_b200_testing_plant_claim(None, b"A" * 31, 10) == kache.KACHE_EINVAL
    T.close()


def test_failed_first_upsert_leaves_no_keys_behind():
    """A table emptied after it had grown; its next upsert, of keys that share a minimizer, fills the overflow table,
    whose growth fails; the one after, which takes the empty table to a larger capacity again, makes the table the
    oracle makes of it alone."""
    L = kache.lib()
    g = synth.genome(300_000, seed=78)
    first, last = (Batch(*synth.stretches(x, 500)) for x in (g[:150_000], g[150_000:]))
    shared = Batch(*synth.one_minimizer(1000, 79))
    T = kache.Table(31, 8, 1000, capi=False)
    u = T.register()
    T.upsert(u, first, kache.ADD, 1, 1)
    T.clear()
    r = ctypes.c_uint64()
    try:
        L.kache_b200_testing_fail_allocation(0)
        assert L.kache_b200_upsert(T.h, u, *shared.args(), kache.ADD, 1, 1, ctypes.byref(r)) == kache.KACHE_ENOMEM
    finally:
        L.kache_b200_testing_fail_allocation(-1)
    assert T.stats().overflow_keys > 1000       # It was the overflow table's growth that failed.
    inserted = T.upsert(u, last, kache.ADD, 1, 1)
    O = oracle.OracleTable(31, 8, 1000)
    assert inserted == O.upsert(O.register(), last, kache.ADD, 1, 1)
    kg, vg = T.dump()
    ko, vo = O.dump()
    assert T.size() == O.size() and np.array_equal(kg, ko) and np.array_equal(vg, vo)
    T.close()


def test_rebuild_that_failed_midway_takes_the_smaller_table_next():
    """A rebuild at four times the buckets (one doubling ahead) fails at its overflow table, its other arrays made. With
    memory then left for the overflow table of twice the buckets but not of four times, the call made again rebuilds at
    twice, and the table is the oracle's."""
    L = kache.lib()
    g = synth.genome(90_060, seed=80)
    first, more = (Batch(*synth.stretches(x, 500)) for x in (g[:42_600], g[42_600:]))
    T = kache.Table(31, 8, 40_000, 0.8, True, capi=False)       # 2,048 buckets.
    u = T.register()
    T.upsert(u, first, kache.ADD, 1, 1)
    T.lookup(more)      # The batch's staging is allocated.
    r = ctypes.c_uint64()

    def upsert():
        return L.kache_b200_upsert(T.h, u, *more.args(), kache.ADD, 1, 1, ctypes.byref(r))

    try:
        L.kache_b200_testing_fail_allocation(3)
        assert upsert() == kache.KACHE_ENOMEM
        L.kache_b200_testing_fail_allocation(-1)
        L.kache_b200_testing_device_memory(400_000)     # 8,192 slots of 32 bytes, but not 16,384.
        assert upsert() == kache.KACHE_OK
    finally:
        L.kache_b200_testing_fail_allocation(-1)
        L.kache_b200_testing_device_memory(-1)
    O = oracle.OracleTable(31, 8, 40_000, 0.8, True)
    uo = O.register()
    O.upsert(uo, first, kache.ADD, 1, 1)
    assert r.value == O.upsert(uo, more, kache.ADD, 1, 1)
    assert T.capacity() == O.capacity()
    kg, vg = T.dump()
    ko, vo = O.dump()
    assert T.size() == O.size() and np.array_equal(kg, ko) and np.array_equal(vg, vo)
    T.close()
