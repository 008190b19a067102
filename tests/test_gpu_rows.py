"""Rows of 32 consecutive k-mers upserted, updated and counted by a warp together, against the oracle: segment and row
edges, keys repeated within a row (homopolymers, tandem repeats), the same new keys from many warps at once, full
buckets and the overflow table, for operations that commute and operations that wait for a racing insert."""
import numpy as np
import pytest

import kache
import oracle
import synth
from kache import Batch

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _rand(rng, n):
    return ACGT[rng.integers(0, 4, n)].tobytes()


def _edge_reads(k, seed):
    """Reads with 0, 1, 31, 32, 33, 511, 512, 513, ... k-mers, and repeats of periods 1 to 33 (keys again within a row)."""
    rng = np.random.default_rng(seed)
    reads = [_rand(rng, k - 1 + m) for m in (0, 1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 511, 512, 513, 1025)]
    for period in (1, 2, 3, 5, 7, 16, 31, 32, 33):
        unit = _rand(rng, period)
        reads.append((unit * (300 // period + 2))[:300])
    reads += [b"A" * 200, b"T" * 200, b"AC" * 100, b"N" + b"G" * 90 + b"N" + b"C" * 90]
    half = _rand(rng, 150)
    comp = half.translate(bytes.maketrans(b"ACGT", b"TGCA"))[::-1]
    return reads + [half + comp, half[:40] + b"N" + half[40:], half.lower()]


@pytest.mark.parametrize("k,l,vb", [(31, 22, 8), (31, 22, 1), (27, 16, 2), (32, 20, 4)])
@pytest.mark.parametrize("op,x,init", [(kache.ADD_WRAP, 1, 1), (kache.MIN, 3, 9), (kache.ASSIGN, 7, 7), (kache.KEEP, 0, 5)])
def test_row_edges_and_repeats(k, l, vb, op, x, init):
    reads = _edge_reads(k, 5)
    for n, copies in ((100_000, 1), (200, 60)):     # A roomy table; one that overflows, with every new key raced for.
        b = Batch.of(reads * copies)
        G = kache.Table(k, vb, n, 0.8, False, l, capi=False)
        O = oracle.OracleTable(k, vb, n, 0.8, False)
        ug, uo = G.register(), O.register()
        for _ in range(2):
            assert G.upsert(ug, b, op, x, init) == O.upsert(uo, b, op, x, init)
            assert G.capacity() == O.capacity()
        if op != kache.KEEP:
            assert G.update(b, op, x, capi=False) == O.update(b, op, x)
        kg, vg = G.dump()
        ko, vo = O.dump()
        assert G.size() == O.size() and np.array_equal(kg, ko) and np.array_equal(vg, vo)
        f, v, w = G.lookup(b)
        fo, v_o, wo = O.lookup(b)
        assert np.array_equal(f, fo) and np.array_equal(v, v_o) and np.array_equal(w, wo)
        assert np.array_equal(G.count(b), O.count(b))
        G.close()


@pytest.mark.parametrize("vb", [0, 4])
def test_counts_past_full_buckets(vb):
    """Per-sequence counts of 5,000 reads, half of them absent, on a table at its load factor, whose full buckets send
    keys to secondary buckets and the overflow table."""
    g = synth.genome(999_900, seed=81)
    index = Batch(*synth.stretches(g, 100_000))
    other = synth.genome(500_000, seed=82)
    reads = synth.reads_fixed(g, 2500, 150, seed=83), synth.reads_fixed(other, 2500, 150, seed=84)
    q = Batch(np.concatenate([r[0][:2500 * 150] for r in reads]), np.arange(5001, dtype=np.uint64) * np.uint64(150))
    G = kache.Table(31, vb, 1_000_000)
    O = oracle.OracleTable(31, vb, 1_000_000)
    assert G.insert(G.register(), index, kache.KEEP, 0) == O.insert(O.register(), index, kache.KEEP, 0)
    assert G.stats().overflow_keys > 0
    assert np.array_equal(G.count(q), O.count(q))
    G.close()


def _dev(bases, off):
    import torch
    return torch.from_numpy(np.ascontiguousarray(bases)).cuda(), torch.from_numpy(off.view(np.int64)).cuda()


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 4096, 4097, 9001])
def test_staging_edges(n):
    """Device batches of as many sequences as its staging's blocks and launches divide by, some empty or shorter than k,
    alone and as several batches (one of them empty): upserts, lookups, updates and counts against the oracle."""
    import torch
    rng = np.random.default_rng(n)
    lens = rng.choice([0, 5, 30, 31, 32, 62, 63, 100], n)
    lens[0] = 700
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(lens)
    b = Batch(np.concatenate([ACGT[rng.integers(0, 4, int(off[-1]))], np.zeros(16, np.uint8)]), off)
    bases, offs = _dev(b.bases, b.off)
    G, O = kache.Table(31, 4, 1000), oracle.OracleTable(31, 4, 1000)
    u, uo = G.register(), O.register()
    torch.cuda.synchronize()
    cut = n // 3
    parts = [(bases.data_ptr(), offs.data_ptr(), cut), (bases.data_ptr(), offs.data_ptr() + 8 * cut, 0), (bases.data_ptr(), offs.data_ptr() + 8 * cut, n - cut)]
    assert G.upsert_dev(u, bases.data_ptr(), offs.data_ptr(), n, kache.ADD, 1, 1) == O.upsert(uo, b, kache.ADD, 1, 1)
    assert sum(G.run_dev_batches(kache.RUN_UPSERT, parts, kache.ADD, 2, 2, u)) == O.upsert(uo, b, kache.ADD, 2, 2)
    assert G.update_dev(bases.data_ptr(), offs.data_ptr(), n, kache.ADD, 1) == O.update(b, kache.ADD, 1)
    assert G.capacity() == O.capacity()
    fo, vo, _ = O.lookup(b)
    P = len(fo)
    f, v, c = (torch.full((max(m, 1),), 7, dtype=t, device="cuda") for m, t in ((P, torch.uint8), (P, torch.int32), (n, torch.int64)))
    torch.cuda.synchronize()
    G.lookup_dev(bases.data_ptr(), offs.data_ptr(), n, f.data_ptr(), v.data_ptr())
    G.count_dev(bases.data_ptr(), offs.data_ptr(), n, c.data_ptr())
    assert np.array_equal(f.cpu().numpy()[:P], fo) and np.array_equal(v.cpu().numpy()[:P].view(np.uint32), vo)
    assert np.array_equal(c.cpu().numpy().view(np.uint64), O.count(b))
    first = int(b.slice(0, cut).positions(31).sum()) if cut else 0
    f.fill_(7), c.fill_(7)
    torch.cuda.synchronize()
    hits = G.run_dev_batches(kache.RUN_LOOKUP, [parts[0] + (f.data_ptr(),), parts[1] + (f.data_ptr(),), parts[2] + (f.data_ptr() + first,)])
    sums = G.run_dev_batches(kache.RUN_COUNT, [parts[0] + (c.data_ptr(),), parts[1] + (c.data_ptr(),), parts[2] + (c.data_ptr() + 8 * cut,)])
    assert np.array_equal(f.cpu().numpy()[:P], fo) and np.array_equal(c.cpu().numpy().view(np.uint64), O.count(b))
    assert hits == sums == [int((fo[:first] == 1).sum()), 0, int((fo[first:] == 1).sum())]
    G.close()


@pytest.mark.parametrize("n,length", [(150_000, 150), (3, 4_000_000)])
def test_large_launches_equal_prepared_ones(n, length):
    """Batches whose warps take segments from a counter, and few sequences of more segments than a block lists: staged
    lookups and counts equal prepared ones, whose shares are fixed, and the update's total is theirs."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(5)
    bases = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")[torch.randint(0, 4, (n * length + 64,), device="cuda", generator=g)]
    bases[n * length // 2:n * length] = bases[:n * length - n * length // 2].clone()    # Each half's k-mers again.
    off = torch.arange(n + 1, dtype=torch.int64, device="cuda") * length
    half = torch.arange(n // 2 + 1, dtype=torch.int64, device="cuda") * length
    G = kache.Table(31, 4, 10_000_000)
    u, P = G.register(), n * (length - 30)
    f, h = (torch.zeros(P, dtype=torch.uint8, device="cuda") for _ in range(2))
    v, w = (torch.zeros(P, dtype=torch.int32, device="cuda") for _ in range(2))
    c, d = (torch.zeros(n, dtype=torch.int64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    G.upsert_dev(u, bases.data_ptr(), half.data_ptr(), n // 2, kache.ADD, 1, 1)
    p = G.prepare_dev(off.data_ptr(), n)
    G.lookup_dev(bases.data_ptr(), off.data_ptr(), n, f.data_ptr(), v.data_ptr())
    G.lookup_prepared(p, bases.data_ptr(), h.data_ptr(), w.data_ptr())
    G.count_prepared(p, bases.data_ptr(), d.data_ptr())
    G.count_dev(bases.data_ptr(), off.data_ptr(), n, c.data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(f, h) and torch.equal(v, w) and torch.equal(c, d)
    present = int((f == 1).sum())
    assert present == int(c.sum()) == G.update_dev(bases.data_ptr(), off.data_ptr(), n, kache.ADD, 1) and 0 < present
    assert int(v[f == 1].min()) >= 1
    G.prepared_free(p)
    G.close()


@pytest.mark.parametrize("op,x,init", [(kache.ADD_WRAP, 1, 1), (kache.MIN, 3, 9)])
def test_upserts_by_the_work_counter(op, x, init):
    """121,000 reads of 121 k-mers, whose warps take segments from a counter, one of an operation that commutes and one
    that waits for a racing insert; as one batch and as two."""
    import torch
    g = synth.genome(1_000_000, seed=85)
    b = Batch(*synth.reads_fixed(g, 121_000, 151, seed=86))
    bases, offs = _dev(b.bases, b.off)
    G, O = kache.Table(31, 4, 30_000_000), oracle.OracleTable(31, 4, 30_000_000)
    u, uo = G.register(), O.register()
    torch.cuda.synchronize()
    p, o, cut = bases.data_ptr(), offs.data_ptr(), 500
    assert G.upsert_dev(u, p, o, b.n, op, x, init) == O.upsert(uo, b, op, x, init)
    parts = [(p, o, cut), (p, o + 8 * cut, b.n - cut)]
    assert G.run_dev_batches(kache.RUN_UPSERT, parts, op, x, init, u) == [0, 0]
    O.upsert(uo, b, op, x, init)
    assert sum(G.run_dev_batches(kache.RUN_UPDATE, parts, kache.ADD, 2)) == O.update(b, kache.ADD, 2)
    kg, vg = G.dump()
    ko, vo = O.dump()
    assert G.size() == O.size() and np.array_equal(kg, ko) and np.array_equal(vg, vo)
    f, _, _ = O.lookup(b)
    d = torch.zeros(len(f), dtype=torch.uint8, device="cuda")
    c = torch.zeros(b.n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    first = 121 * cut
    hits = G.run_dev_batches(kache.RUN_LOOKUP, [parts[0] + (d.data_ptr(),), parts[1] + (d.data_ptr() + first,)])
    assert hits == [int((f[:first] == 1).sum()), int((f[first:] == 1).sum())]
    assert G.run_dev_batches(kache.RUN_COUNT, [parts[0] + (c.data_ptr(),), parts[1] + (c.data_ptr() + 8 * cut,)]) == hits
    assert np.array_equal(d.cpu().numpy(), f) and np.array_equal(c.cpu().numpy().view(np.uint64), O.count(b))
    G.close()


@pytest.mark.parametrize("vb", [0, 2, 8])
def test_overflow_grows_behind_a_staged_upsert(vb):
    """Device upserts of 10,000 keys of one minimizer, of which 96 have room in buckets: the overflow table's 2,048 slots
    fill up, and the k-mers left over are upserted again in larger ones, from the list that was staged."""
    import torch
    b = Batch(*synth.one_minimizer(1000, 87))
    bases, offs = _dev(b.bases, b.off)
    G, O = kache.Table(31, vb, 20_000), oracle.OracleTable(31, vb, 20_000)
    u, uo = G.register(), O.register()
    torch.cuda.synchronize()
    p, o = bases.data_ptr(), offs.data_ptr()
    G.profile(True)
    ins = G.upsert_dev(u, p, o, b.n, kache.ADD, 1, 1)
    assert G.profile_read(0)[1] > 2     # The launch, and at least two more after the overflow table's growth.
    assert ins == O.upsert(uo, b, kache.ADD, 1, 1) and G.stats().overflow_keys > 9000
    assert sum(G.run_dev_batches(kache.RUN_UPSERT, [(p, o, 300), (p, o + 2400, 700)], kache.ADD, 1, 1, u)) == O.upsert(uo, b, kache.ADD, 1, 1)
    kg, vg = G.dump()
    ko, vo = O.dump()
    assert np.array_equal(kg, ko) and (vb == 0 or np.array_equal(vg, vo))
    c = torch.zeros(b.n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    G.count_dev(p, o, b.n, c.data_ptr())
    assert np.array_equal(c.cpu().numpy().view(np.uint64), O.count(b))
    G.close()


def test_slot_given_up_for_a_lower_claim():
    """A read's ten new keys of one bucket, the fourth of which has a claim there already that was never published: the keys
    claim slots side by side, the fourth then finds the earlier claim in the slot that the first one lost, and leaves its
    own slot as a hole. Nobody sees the hole, and later keys of the bucket go past it."""
    b = Batch(*synth.one_minimizer(200, 88))
    one = b.slice(0, 1)
    kmer = bytes(b.bases[3:34])
    G, O = kache.Table(31, 4, 20_000), oracle.OracleTable(31, 4, 20_000)
    u, uo = G.register(), O.register()
    assert kache.lib().kache_b200_testing_plant_claim(G.h, kmer, 1000) == kache.KACHE_OK
    O.upsert(uo, one, kache.ADD, 1, 1)
    assert G.upsert(u, one, kache.ADD, 1, 1) == 9
    O.upsert(uo, b.slice(1, 200), kache.ADD, 1, 1)
    assert G.upsert(u, b.slice(1, 200), kache.ADD, 1, 1) == O.size() - 10
    ko, vo = O.dump()
    fo, _, _ = O.lookup(b)
    kg, vg = G.dump()
    f, v, _ = G.lookup(b)
    missing = np.setdiff1d(ko, kg)      # The planted k-mer's, which is not published.
    assert len(missing) == 1 and len(kg) == len(ko) - 1
    assert np.array_equal(kg, ko[ko != missing]) and np.array_equal(vg, vo[ko != missing])
    assert fo[3] == 1 and f[3] == 0 and np.array_equal(np.delete(f, 3), np.delete(fo, 3))
    assert G.size() == len(kg) == G.reduce(kache.REDUCE_KEYS)
    G.close()


@pytest.mark.parametrize("vb", [2, 4])
def test_histogram_past_a_blocks_bins(vb):
    """Counts on both sides of the 8,192 that a block holds, and of the largest asked for."""
    g = synth.genome(5000, seed=89)
    G, O = kache.Table(31, vb, 10_000), oracle.OracleTable(31, vb, 10_000)
    u, uo = G.register(), O.register()
    for i, x in enumerate((1, 8190, 8191, 8192, 8193, 9999, 10_000, 10_001, 65_535)):
        b = Batch(*synth.stretches(g[500 * i:500 * i + 130 + i], 1000))
        assert G.upsert(u, b, kache.ASSIGN, x, x) == O.upsert(uo, b, kache.ASSIGN, x, x)
    for m in (0, 1, 8190, 8191, 8192, 8193, 10_000, 70_000):
        assert np.array_equal(G.histogram(m), O.histogram(m))
    G.close()


@pytest.mark.parametrize("vb", [1, 2, 4])
@pytest.mark.parametrize("x", [1, 200, 255])
def test_wrapping_adds_to_hot_keys(vb, x):
    """Values of 1, 2 and 4 bytes that wrap around many times, added to from all warps at once; then an operation that
    compares the whole values."""
    x = x * 257 if vb == 2 else x
    b = Batch.of([b"ACGTTGCAAC" * 15] * 3000 + [b"A" * 150] * 1000 + [_rand(np.random.default_rng(i % 50), 150) for i in range(3000)])
    G, O = kache.Table(31, vb, 20_000), oracle.OracleTable(31, vb, 20_000)
    u, uo = G.register(), O.register()
    for _ in range(2):
        assert G.upsert(u, b, kache.ADD_WRAP, x, 3) == O.upsert(uo, b, kache.ADD_WRAP, x, 3)
        assert G.update(b, kache.ADD_WRAP, x, capi=False) == O.update(b, kache.ADD_WRAP, x)
        assert np.array_equal(G.dump()[1], O.dump()[1])
    assert G.update(b, kache.MAX, 77, capi=False) == O.update(b, kache.MAX, 77)
    assert G.update(b, kache.ADD, 100) == O.update(b, kache.ADD, 100)
    assert np.array_equal(G.dump()[1], O.dump()[1])
    G.close()
