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
