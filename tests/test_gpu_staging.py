"""Device batches of thousands of sequences with long ones among them: every call against the oracle, at each size by which
their segments are listed differently, once and again; and the time that their staging takes."""
import numpy as np
import pytest

import kache
import oracle
from kache import Batch

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _batch(lens, seed):
    rng = np.random.default_rng(seed)
    off = np.zeros(len(lens) + 1, np.uint64)
    off[1:] = np.cumsum(lens)
    bases = ACGT[rng.integers(0, 4, int(off[-1]))]
    bases[rng.integers(0, len(bases), len(bases) // 5000)] = ord("N")
    return Batch(np.concatenate([bases, np.zeros(16, np.uint8)]), off)


def _on_gpu(b):
    import torch
    return torch.from_numpy(b.bases).cuda(), torch.from_numpy(b.off.view(np.int64)).cuda()


# A thread lists up to 32 segments of 512 positions; a block's sequences (1,024) may have 16,384; the list has room for
# n / 8 + 1,024 more than the sequences.
@pytest.mark.parametrize("n,at,longs", [
    (4097, 4095, [30 + 32 * 512, 31 + 32 * 512]),               # The last segment that a thread lists, the first of a warp.
    (5000, 1023, [600_000]),                                    # Listed by a warp.
    (5000, 0, [1_400_000]),                                       # More than the list has room for.
    (150_000, 77, [30 + 512 * 15_361]),                         # 16,384 segments of one block with its 1,023 others,
    (150_000, 77, [31 + 512 * 15_361]),                         # and one more.
])
def test_long_sequences_among_many(n, at, longs):
    import torch
    lens = np.full(n, 33)
    lens[::7], lens[::11] = 0, 31
    if n > 100_000:
        lens[:1024] = 40        # Each of one segment, so that the long one's make up the block's.
    lens[at:at + len(longs)] = longs[:n - at]
    b = _batch(lens, n)
    bases, off = _on_gpu(b)
    T, O = kache.Table(31, 4, 1000), oracle.OracleTable(31, 4, 1000)
    u, uo = T.register(), O.register()
    P = int(b.positions(31).sum())
    cut = n // 3
    first = int(b.slice(0, cut).positions(31).sum())
    f, v, c = (torch.zeros(m, dtype=t, device="cuda") for m, t in ((P, torch.uint8), (P, torch.int32), (n, torch.int64)))
    torch.cuda.synchronize()
    p, q, s = bases.data_ptr(), off.data_ptr(), off.data_ptr() + 8 * cut
    for _ in range(2):
        assert T.upsert_dev(u, p, q, n, kache.ADD, 1, 1) == O.upsert(uo, b, kache.ADD, 1, 1)
        assert sum(T.run_dev_batches(kache.RUN_UPSERT, [(p, q, cut), (p, s, n - cut)], kache.ADD, 1, 1, u)) == O.upsert(uo, b, kache.ADD, 1, 1)
        assert T.update_dev(p, q, n, kache.ADD, 3) == O.update(b, kache.ADD, 3)
        fo, vo, _ = O.lookup(b)
        co = O.count(b)
        hits = [int((fo[:first] == 1).sum()), int((fo[first:] == 1).sum())]
        for merged in (False, True):
            f.fill_(7), v.fill_(7), c.fill_(7)
            torch.cuda.synchronize()
            if merged:
                assert T.run_dev_batches(kache.RUN_LOOKUP, [(p, q, cut, f.data_ptr(), v.data_ptr()), (p, s, n - cut, f.data_ptr() + first, v.data_ptr() + 4 * first)]) == hits
                assert T.run_dev_batches(kache.RUN_COUNT, [(p, q, cut, c.data_ptr()), (p, s, n - cut, c.data_ptr() + 8 * cut)]) == hits
            else:
                T.lookup_dev(p, q, n, f.data_ptr(), v.data_ptr())
                T.count_dev(p, q, n, c.data_ptr())
            assert np.array_equal(f.cpu().numpy(), fo) and np.array_equal(v.cpu().numpy().view(np.uint32), vo)
            assert np.array_equal(c.cpu().numpy().view(np.uint64), co)
    ko, vo = O.dump()
    kg, vg = T.dump()
    assert np.array_equal(kg, ko) and np.array_equal(vg, vo)
    T.close()


@pytest.mark.parametrize("n,length", [(5000, 90_000_000), (200_000, 25_000_000)])
def test_listing_long_sequences_in_parallel(n, length):
    """The kernels that stage such a batch take some tens of microseconds, where one thread that writes the long sequence's
    segments takes 1.6 and 5.9 ms; at the first call and at later ones, whose list has had to hold them."""
    import torch
    off = torch.full((n + 1,), 100, dtype=torch.int64, device="cuda").cumsum(0) - 100
    off[-1] += length - 100
    bases = torch.full((int(off[-1]) + 16,), ord("A"), dtype=torch.uint8, device="cuda")
    c = torch.zeros(n, dtype=torch.int64, device="cuda")
    T = kache.Table(31, 4, 1000)
    torch.cuda.synchronize()
    other = []
    for _ in range(4):
        T.profile(True)
        T.count_dev(bases.data_ptr(), off.data_ptr(), n, c.data_ptr())
        other.append(T.profile_read(5)[0])
        T.profile(False)
    print(other)
    assert max(other) < 1 and int(c.sum()) == 0
    T.close()


def test_a_warp_per_segment_of_a_middling_batch():
    """4,100 sequences of 5,125 segments, which the GPU's resident warps can take one each: the lookup staged with them
    takes no longer than one over the listed segments (1.45 times as long where it is launched for a segment each)."""
    import torch
    lens = np.tile([500, 500, 500, 1000], 1025)
    b = _batch(lens, 3)
    bases, off = _on_gpu(b)
    T = kache.Table(31, 8, 100_000_000)      # Larger than the caches.
    P = int(b.positions(31).sum())
    f = torch.zeros(P, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    T.upsert_dev(T.register(), bases.data_ptr(), off.data_ptr(), b.n, kache.KEEP, 0, 1)
    shape = T.prepare_dev(off.data_ptr(), b.n)

    def least(call):
        ms = []
        for _ in range(20):
            T.profile(True)
            call()
            torch.cuda.synchronize()
            ms.append(T.profile_read(2)[0])
            T.profile(False)
        return min(ms)

    staged = least(lambda: T.lookup_dev(bases.data_ptr(), off.data_ptr(), b.n, f.data_ptr()))
    prepared = least(lambda: T.lookup_prepared(shape, bases.data_ptr(), f.data_ptr()))
    print(staged, prepared)
    assert 0 < staged < 1.2 * prepared, (staged, prepared)
    T.prepared_free(shape)
    T.close()


def test_segment_lists_in_little_memory():
    """Calls with memory for no more than 24 bytes per sequence and 8 per segment (and, merged, 12 per sequence), where a list
    takes 32 per segment: its segments are then listed and run a part at a time. A shape prepared with room for one list."""
    import torch
    n = 100_000
    lens = np.full(n, 60)
    lens[5], lens[n - 3] = 400_000, 20_000
    b = _batch(lens, 9)
    bases, off = _on_gpu(b)
    T, O = kache.Table(31, 4, 5_000_000), oracle.OracleTable(31, 4, 5_000_000)
    u, uo = T.register(), O.register()
    P = int(b.positions(31).sum())
    f, v, c = (torch.zeros(m, dtype=t, device="cuda") for m, t in ((P, torch.uint8), (P, torch.int32), (n, torch.int64)))
    p, q = bases.data_ptr(), off.data_ptr()
    cut = n // 3
    first = int(b.slice(0, cut).positions(31).sum())
    s = q + 8 * cut
    torch.cuda.synchronize()
    few = b.slice(0, 5)
    assert T.upsert_dev(u, p, q, 5, kache.ADD, 1, 1) == O.upsert(uo, few, kache.ADD, 1, 1)     # The retry marks are made.
    segs = int(((b.positions(31) + 511) // 512).sum())
    left = kache.lib().kache_b200_testing_device_memory
    try:
        left(24 * n + 12 * segs)
        assert T.upsert_dev(u, p, q, n, kache.ADD, 1, 1) == O.upsert(uo, b, kache.ADD, 1, 1)
        assert T.update_dev(p, q, n, kache.ADD, 3) == O.update(b, kache.ADD, 3)
        T.lookup_dev(p, q, n, f.data_ptr(), v.data_ptr())
        T.count_dev(p, q, n, c.data_ptr())
        fo, vo, _ = O.lookup(b)
        co = O.count(b)
        assert np.array_equal(f.cpu().numpy(), fo) and np.array_equal(v.cpu().numpy().view(np.uint32), vo)
        assert np.array_equal(c.cpu().numpy().view(np.uint64), co)
        left(16 * n)
        hits = [int((fo[:first] == 1).sum()), int((fo[first:] == 1).sum())]
        f.fill_(7)
        torch.cuda.synchronize()
        assert T.run_dev_batches(kache.RUN_LOOKUP, [(p, q, cut, f.data_ptr(), v.data_ptr()), (p, s, n - cut, f.data_ptr() + first, v.data_ptr() + 4 * first)]) == hits
        assert np.array_equal(f.cpu().numpy(), fo)
        assert sum(T.run_dev_batches(kache.RUN_UPSERT, [(p, q, cut), (p, s, n - cut)], kache.ADD, 1, 1, u)) == O.upsert(uo, b, kache.ADD, 1, 1)
        left(30 * segs)     # With the 8 per segment that the table holds.
        shape = T.prepare_dev(q, n)
        f.fill_(7)
        torch.cuda.synchronize()
        T.lookup_prepared(shape, p, f.data_ptr(), v.data_ptr())
        torch.cuda.synchronize()
        fo, vo, _ = O.lookup(b)
        assert np.array_equal(f.cpu().numpy(), fo) and np.array_equal(v.cpu().numpy().view(np.uint32), vo)
        T.prepared_free(shape)
    finally:
        left(-1)
    kg, vg = T.dump()
    ko, vo = O.dump()
    assert np.array_equal(kg, ko) and np.array_equal(vg, vo)
    T.close()


@pytest.mark.parametrize("k,l,vb", [(31, 22, 4), (32, 20, 0), (27, 16, 1)])
@pytest.mark.parametrize("n,low,high", [(16_384, 25, 40), (16_391, 0, 125), (40_003, 33, 37), (20_000, 120, 127), (16_390, 30, 33)])
def test_groups_of_short_sequences(k, l, vb, n, low, high):
    """Short sequences, whose k-mers are a warp's rows together in groups of eight: empty ones and ones shorter than k among
    them, and, at 124 bases, the longest that a group takes; from the device, as one batch and as several that begin
    inside a group of eight, and from the host."""
    import torch
    rng = np.random.default_rng(n)
    b = _batch(rng.integers(low, high, n), n + k)
    bases, off = _on_gpu(b)
    T, O = kache.Table(k, vb, 1000, 0.8, False, l, capi=False), oracle.OracleTable(k, vb, 1000, 0.8, False)
    u, uo = T.register(), O.register()
    p, q = bases.data_ptr(), off.data_ptr()
    cuts = [0, 3, 3, n // 3 | 1, n - 5, n]
    first = [int(b.slice(0, c).positions(k).sum()) if c else 0 for c in cuts]
    P = first[-1]
    f, w, v, c = (torch.zeros(max(m, 1), dtype=t, device="cuda") for m, t in ((P, torch.uint8), (P, torch.uint8), (P * max(vb, 1), torch.uint8), (n, torch.int64)))
    vp = v.data_ptr() if vb else None
    torch.cuda.synchronize()

    def parts(*outs):
        return [(p, q + 8 * a, e - a) + tuple(o and o + size * (a if seq else x) for o, size, seq in outs) for a, e, x in zip(cuts, cuts[1:], first)]

    for i in range(2):
        assert T.upsert_dev(u, p, q, n, kache.ADD, 1, 1) == O.upsert(uo, b, kache.ADD, 1, 1)
        assert sum(T.run_dev_batches(kache.RUN_UPSERT, parts(), kache.ADD, 1, 1, u)) == O.upsert(uo, b, kache.ADD, 1, 1)
        assert T.upsert(u, b, kache.ADD, 1, 1) == O.upsert(uo, b, kache.ADD, 1, 1)
        if vb:
            half = b.slice(0, n // 2)
            assert T.update_dev(p, q, n // 2, kache.ADD_WRAP, 5) == O.update(half, kache.ADD_WRAP, 5)
            assert T.upsert_oriented_dev(u, p, q, n, kache.OR, 1, 2) == O.insert_oriented(uo, b, kache.OR, 1, 2)
        fo, vo, wo = O.lookup(b)
        co = O.count(b)
        hits = [int((fo[x:y] == 1).sum()) for x, y in zip(first, first[1:])]
        for merged in (False, True):
            f.fill_(7), w.fill_(7), v.fill_(7), c.fill_(7)
            torch.cuda.synchronize()
            if merged:
                assert T.run_dev_batches(kache.RUN_LOOKUP, parts((f.data_ptr(), 1, False), (vp, vb, False), (w.data_ptr(), 1, False))) == hits
                assert T.run_dev_batches(kache.RUN_COUNT, parts((c.data_ptr(), 8, True))) == hits
            else:
                T.lookup_dev(p, q, n, f.data_ptr(), vp, w.data_ptr())
                T.count_dev(p, q, n, c.data_ptr())
            assert np.array_equal(f.cpu().numpy()[:P], fo) and np.array_equal(w.cpu().numpy()[:P], wo)
            assert vb == 0 or np.array_equal(v.cpu().numpy()[:P * vb].view(T.vdt), vo)
            assert np.array_equal(c.cpu().numpy().view(np.uint64), co)
        assert np.array_equal(T.count(b), co)
        if vb:
            assert np.array_equal(T.count_masked(b, 1, 2), O.count_masked(b, 1, 2)) and np.array_equal(T.sum(b), O.sum(b))
        fh, vh, wh = T.lookup(b)
        assert np.array_equal(fh, fo) and np.array_equal(wh, wo) and (vb == 0 or np.array_equal(vh, vo))
    kg, vg = T.dump()
    ko, vo = O.dump()
    assert np.array_equal(kg, ko) and (vb == 0 or np.array_equal(vg, vo))
    T.close()


def test_short_sequences_in_little_memory():
    """Short sequences, which might be run in groups, with memory for the sums over them and for a quarter of their segments'
    list, 24 bytes and 8 for each, and none for groups."""
    import torch
    n = 40_000
    b = _batch(np.full(n, 40), 17)
    bases, off = _on_gpu(b)
    T, O = kache.Table(31, 4, 1_000_000), oracle.OracleTable(31, 4, 1_000_000)
    u, uo = T.register(), O.register()
    f = torch.zeros(10 * n, dtype=torch.uint8, device="cuda")
    p, q = bases.data_ptr(), off.data_ptr()
    torch.cuda.synchronize()
    assert T.upsert_dev(u, p, q, 5, kache.ADD, 1, 1) == O.upsert(uo, b.slice(0, 5), kache.ADD, 1, 1)     # The retry marks are made.
    left = kache.lib().kache_b200_testing_device_memory
    try:
        left(24 * n + 8 * n + 4096)
        assert T.upsert_dev(u, p, q, n, kache.ADD, 1, 1) == O.upsert(uo, b, kache.ADD, 1, 1)
        T.lookup_dev(p, q, n, f.data_ptr())
    finally:
        left(-1)
    assert np.array_equal(f.cpu().numpy(), O.lookup(b)[0])
    T.close()


# Groups are made where they save 500,000 units (groups_pay, device_misc.cuh) and 2,000 for each segment beside them, or
# 4,000,000. These batches' would save 0, 0, 557,056 with no segments, 552,432 with 170, 1,083,200 with 3, 2,109,024 with 8,846,
# 5,549,824 with 12,500, and of eight sequences one of which has 124 bases 1,600,000, or, of 125, 0.
@pytest.mark.parametrize("n,low,high,every,launches", [
    (17_000, 60, 140, 0, 3), (60_000, 75, 76, 0, 3), (16_384, 33, 34, 0, 4), (16_384, 33, 34, 1000, 3), (40_003, 33, 37, 0, 4), (250_000, 0, 60, 200, 3),
    (250_000, 31, 46, 200, 4), (80_000, 124, 0, 0, 4), (80_000, 125, 0, 0, 3),
])
def test_groups_only_where_they_pay(n, low, high, every, launches):
    """Lookups and counts of reads of `low` to `high` - 1 bases, one in `every` of 1,100: by how many launches, and against the
    oracle, as one batch and as two."""
    import torch
    lens = np.random.default_rng(n).integers(low, high, n) if high else np.resize([31, 31, 0, 33, 31, 30, 31, low], n)
    if every:
        lens[5::every] = 1100
    b = _batch(lens, n + low)
    bases, off = _on_gpu(b)
    T, O = kache.Table(31, 4, 1_000_000), oracle.OracleTable(31, 4, 1_000_000)
    p, q = bases.data_ptr(), off.data_ptr()
    torch.cuda.synchronize()
    u, uo = T.register(), O.register()
    for s in range(0, n // 2, 5000):        # In batches too small for groups.
        part = b.slice(s, min(n // 2, s + 5000))
        assert T.upsert(u, part, kache.ADD, 1, 1) == O.upsert(uo, part, kache.ADD, 1, 1)
    P = int(b.positions(31).sum())
    f, v, c = (torch.full((m,), 7, dtype=t, device="cuda") for m, t in ((P, torch.uint8), (P, torch.int32), (n, torch.int64)))
    torch.cuda.synchronize()
    before = kache.kernel_launches()
    T.lookup_dev(p, q, n, f.data_ptr(), v.data_ptr())
    assert kache.kernel_launches() - before == launches
    fo, vo, _ = O.lookup(b)
    co = O.count(b)
    assert np.array_equal(f.cpu().numpy(), fo) and np.array_equal(v.cpu().numpy().view(np.uint32), vo)
    T.count_dev(p, q, n, c.data_ptr())
    assert np.array_equal(c.cpu().numpy().view(np.uint64), co)
    cut = n // 3 | 1
    x = int(b.slice(0, cut).positions(31).sum())
    f.fill_(7)
    torch.cuda.synchronize()
    assert T.run_dev_batches(kache.RUN_LOOKUP, [(p, q, cut, f.data_ptr()), (p, q + 8 * cut, n - cut, f.data_ptr() + x)]) == [int((fo[:x] == 1).sum()), int((fo[x:] == 1).sum())]
    assert np.array_equal(f.cpu().numpy(), fo)
    assert T.upsert_dev(u, p, q, n, kache.ADD, 1, 1) == O.upsert(uo, b, kache.ADD, 1, 1)
    kg, vg = T.dump()
    ko, vo = O.dump()
    assert np.array_equal(kg, ko) and np.array_equal(vg, vo)
    T.close()
