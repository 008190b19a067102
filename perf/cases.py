"""The work that programs built on the streaming k-mer table have it do, as cases that can be timed and compared.

A case names a job (what calls a pass makes) and its sizes. Inputs are seeded and made on the GPU: uniform genomes,
reads of fixed or log-normal lengths at uniform starts, half of them reverse-complemented, with substitutions and N's.
All outputs are whole numbers that do not depend on the order in which concurrent inserts land.

Jobs (one pass each):
  find        look up every k-mer of the reads: found flags and values                  (lookup_dev)
  stream      empty a map, count its reads in calls of `call` reads, look them all up   (clear, upsert_dev, lookup_dev)
  count_find  empty a map, count one read set in it, look up a second one               (clear, upsert_dev, lookup_dev)
  counter     count the occurrences of an index's k-mers in a batch of reads, then the
              histogram of the counts and the coverage along the batch's first reads    (update_dev, histogram, lookup_dev)
  oriented    empty a strand map, mark the strands of long reads' k-mers in batches of
              `call` reads, look the batches up with orientations                       (clear, run_dev_batches)
  grow        empty a set sized for 1M keys, insert a genome in calls of `call` pieces
              while it doubles, look up reads of the genome                             (clear, upsert_dev, lookup_dev)
  served      a mix of upsert / find / count requests, one call per kind                (run_dev_batches)
  screen      per read, how many of its k-mers are in a set                             (count_dev)
  host        empty a map, count reads held in host memory and look them up, through
              the C interface                                                           (clear, insert, lookup)
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kache-hash_b200"))
import kache  # noqa: E402

MINIMIZER = {31: 22, 27: 16, 32: 20}
VALUES = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}    # As wide as the table's values.
HIST = 10000        # Largest count of a histogram, as the counter's callers ask for it.
SAMPLE = 16384      # Reads of a counted batch whose coverage is looked up.


def listed():
    return [
        # A short call: 64 reads, the batch of the reference's own measuring loop, against a map of a bacterial genome.
        {"name": "find_64_reads", "job": "find", "k": 31, "value_bytes": 8, "genome": 5_000_000, "reads": 64, "length": 150, "sigma": 0.0},
        # The same reads arriving as they would from a parser: calls of 64 reads into a small map, then one lookup.
        {"name": "stream_64_read_calls", "job": "stream", "k": 31, "value_bytes": 8, "genome": 50_000, "reads": 1024, "call": 64, "length": 150, "sigma": 0.0},
        # A strand map <27, u8, 16> fed calls of one small batch of long reads: few long sequences, ragged lengths.
        {"name": "oriented_256_long_reads", "job": "oriented", "k": 27, "value_bytes": 1, "genome": 1_000_000, "reads": 256, "call": 256, "length": 10_000, "sigma": 0.8},
        # Saturating 16-bit counts of reads of uneven lengths, some shorter than k: an odd, middling batch.
        {"name": "count_find_u16_ragged", "job": "count_find", "k": 31, "value_bytes": 2, "genome": 700_001, "reads": 20_011, "held": 30_011, "length": 150, "sigma": 0.6},
        # Host callers of the C interface with pageable buffers.
        {"name": "host_50k_reads", "job": "host", "k": 31, "value_bytes": 8, "genome": 2_000_000, "reads": 50_000, "length": 150, "sigma": 0.0},
        # Screening a sequencer's reads against a set of a host genome's k-mers (half the reads are from elsewhere).
        {"name": "screen_1m_reads_set", "job": "screen", "k": 31, "value_bytes": 0, "genome": 10_000_000, "reads": 1_000_000, "length": 150, "sigma": 0.0},
        # Looking up an assembly's contigs (1 Mbp each) in a <32, u32, 20> map: the longest sequences.
        {"name": "find_contigs_k32", "job": "find", "k": 32, "value_bytes": 4, "genome": 40_000_000, "reads": 40, "length": 1_000_000, "sigma": 0.0},
        # The headline benchmark: 10x reads of a 5 Mbp genome counted, then 1M held-out reads looked up.
        {"name": "count_find_10m_keys", "job": "count_find", "k": 31, "value_bytes": 8, "genome": 5_000_000, "reads": 333_333, "held": 1_000_000, "length": 150, "sigma": 0.0},
        # The strand map over 16 batches of 256 long reads, one call per kind of request.
        {"name": "oriented_16_batches", "job": "oriented", "k": 27, "value_bytes": 1, "genome": 10_000_000, "reads": 4096, "call": 256, "length": 10_000, "sigma": 0.8},
        # A set that grows from 1M keys by doubling as a genome streams in, in calls of 65,536 pieces.
        {"name": "grow_set_100m", "job": "grow", "k": 32, "value_bytes": 0, "genome": 100_000_000, "reads": 100_000, "call": 65_536, "length": 150, "sigma": 0.0},
        # The k-mer counter: a batch of 2^20 reads counted against the index of a 100 Mbp genome.
        {"name": "counter_1m_reads", "job": "counter", "k": 31, "value_bytes": 4, "genome": 100_000_000, "reads": 1 << 20, "length": 150, "sigma": 0.6},
        # A service's mix of upsert / find / count requests (60/30/10) against a map of a 50 Mbp genome.
        {"name": "served_300_requests", "job": "served", "k": 31, "value_bytes": 4, "genome": 50_000_000, "reads": 1_500_000, "requests": 300, "length": 150, "sigma": 0.0},
    ]


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    job = rng.choice(["find", "stream", "count_find", "counter", "oriented", "grow", "served", "screen", "host"])
    k, vb = rng.choice([31, 31, 27, 32]), rng.choice([1, 2, 4, 8])
    length = rng.choice([75, 100, 150, 150, 251])
    sigma = rng.choice([0.0, 0.0, 0.3, 0.6])
    c = {"job": job, "k": k, "value_bytes": vb, "genome": span(100_000, 50_000_000), "length": length, "sigma": sigma}
    if job == "find":
        if rng.random() < 0.3:
            c.update(length=span(2_000, 1_000_000), sigma=0.0)
        c["reads"] = span(64, 100_000_000 // c["length"]) if c["length"] < 50_000 else rng.randint(1, 40)
        c["genome"] = max(c["genome"], 2 * c["length"])
    elif job == "stream":
        c.update(genome=span(20_000, 500_000), reads=span(256, 8192), call=span(32, 512))
    elif job == "count_find":
        c.update(reads=span(1000, 40_000_000 // length), held=span(1000, 100_000_000 // length))
    elif job == "counter":
        c.update(k=31, value_bytes=4, reads=span(20_000, 140_000_000 // length))
    elif job == "oriented":
        c.update(k=rng.choice([27, 31]), value_bytes=rng.choice([1, 2]), reads=span(64, 4096), call=rng.choice([64, 256]), length=10_000, sigma=0.8)
        c["genome"] = max(c["genome"], 400_000)
    elif job == "grow":
        c.update(value_bytes=0, genome=span(2_000_000, 80_000_000), reads=span(1000, 200_000), call=rng.choice([16_384, 65_536]))
    elif job == "served":
        c.update(k=31, value_bytes=rng.choice([4, 8]), reads=span(20_000, 150_000_000 // length), requests=rng.randint(20, 300))
    elif job == "screen":
        c.update(value_bytes=rng.choice([0, 0, 4]), reads=span(64, 100_000_000 // length))
    else:
        c.update(k=31, value_bytes=rng.choice([4, 8]), genome=span(100_000, 3_000_000), reads=span(100, 80_000))
    return c


# ---- Inputs --------------------------------------------------------------------------------------------------------

def _gen(seed, what):
    return torch.Generator(device="cuda").manual_seed((seed * 1_000_003 + what) & 0x7FFFFFFF)


def _genome(n, seed):
    return torch.randint(0, 4, (n,), dtype=torch.uint8, device="cuda", generator=_gen(seed, 1))


def _offsets(case, n, what):
    """Offsets of n sequences: all of the case's length, or log-normal about it (25-1000 bases for short reads, 1-100 kb
    for long ones), the same for every seed, so that a case's outputs have one shape."""
    length, sigma = case["length"], case["sigma"]
    if sigma:
        x = torch.randn(n, device="cuda", generator=_gen(0, what)).mul_(sigma).exp_().mul_(length)
        lens = x.clamp_(*((1000, 100_000) if length >= 5000 else (25, 1000))).long().clamp_(max=case["genome"])
    else:
        lens = torch.full((n,), min(length, case["genome"]), dtype=torch.int64, device="cuda")
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=off[1:])
    return off


def _ascii():
    return torch.tensor(list(b"ACGTN"), dtype=torch.uint8, device="cuda")


def _reads(case, g, n, seed, what, foreign=0.0, sub=0.005, n_rate=0.0005):
    """n reads of the genome as (ASCII bases, offsets); a share `foreign` of them are random sequence instead."""
    off = _offsets(case, n, what)
    gen = _gen(seed, what + 1)
    total = int(off[-1])
    lens = off[1:] - off[:-1]
    first = (torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) * (g.numel() - lens + 1)).long()
    back = torch.rand(n, device="cuda", generator=gen) < 0.5
    first = torch.where(back, first + lens - 1, first)
    other = torch.rand(n, device="cuda", generator=gen) < foreign
    out = torch.empty(total + 64, dtype=torch.uint8, device="cuda")
    out[total:] = 0
    table, piece = _ascii(), 1 << 25
    for b in range(0, total, piece):
        j = torch.arange(b, min(total, b + piece), device="cuda")
        q = torch.searchsorted(off, j, right=True) - 1
        j -= off[q]
        flip = back[q]
        c = g[torch.where(flip, first[q] - j, first[q] + j)] ^ (flip.to(torch.uint8) * 3)
        u = torch.rand(c.numel(), device="cuda", generator=gen)
        step = torch.randint(1, 4, (c.numel(),), dtype=torch.uint8, device="cuda", generator=gen)
        c = torch.where(u < sub, (c + step) & 3, c)
        if foreign:
            c = torch.where(other[q], torch.randint(0, 4, (c.numel(),), dtype=torch.uint8, device="cuda", generator=gen), c)
        c = torch.where(u >= 1 - n_rate, torch.full_like(c, 4), c)
        out[b:b + c.numel()] = table[c.long()]
    return out, off


def _pieces(g, length):
    """The genome as pieces of `length` bases, end to end."""
    n = -(-g.numel() // length)
    off = (torch.arange(n + 1, device="cuda") * length).clamp_(max=g.numel())
    return torch.cat([_ascii()[g.long()], torch.zeros(64, dtype=torch.uint8, device="cuda")]), off


def _positions(off, k):
    return int((off[1:] - off[:-1] - k + 1).clamp_(min=0).sum())


def _requests(case):
    """(kind, first read, end read) of a service's requests, log-normal in size, over the read pool."""
    gen = torch.Generator().manual_seed(3)
    m = case["requests"]
    x = torch.randn(m, generator=gen).mul_(1.5).exp_()
    ends = (torch.cumsum(x, 0) / x.sum() * case["reads"]).round().long().tolist()
    u = torch.rand(m, generator=gen).tolist()
    return [(0 if v < 0.6 else 1 if v < 0.9 else 2, a, b) for v, a, b in zip(u, [0] + ends[:-1], ends) if b > a]


def _inputs(case, seed):
    """Every array of bases and offsets that a case's calls read."""
    job, g = case["job"], _genome(case["genome"], seed)
    x = {"reads": _reads(case, g, case["reads"], seed, 10, foreign=0.5 if job == "screen" else 0.0, sub=0.01 if job == "served" else 0.005)}
    if job in ("find", "counter", "served", "screen"):
        x["index"] = _pieces(g, 1_000_000)
    if job == "find":
        x["index2"] = _reads(dict(case, length=min(1000, case["genome"]), sigma=0.0), g, max(1, case["genome"] // 1000), seed, 20)
    if job == "count_find":
        x["held"] = _reads(case, g, case["held"], seed, 30)
    if job == "grow":
        x["pieces"] = _pieces(g, 150)
    return x


# ---- A program's state and its calls -------------------------------------------------------------------------------

def _table(case):
    k, job, g = case["k"], case["job"], case["genome"]
    # Sized for the keys expected; sets and services that are only read, or that new keys keep reaching, with headroom.
    keys = {"stream": 2 * g, "count_find": 2 * g, "grow": 1_000_000, "host": 2 * g, "screen": 4 * g,
            "served": 3 * g + 100 * case["reads"]}.get(job, g)
    lf, pow2 = (0.9, True) if job == "counter" else (0.8, False)
    return kache.Table(k, case["value_bytes"], max(keys, 1000), lf, pow2, MINIMIZER[k], capi=k == 31 and job == "host")


def prepare(case, seed):
    k, job, vb = case["k"], case["job"], case["value_bytes"]
    x = _inputs(case, seed)
    t = _table(case)
    torch.cuda.synchronize()    # The table works on a stream of its own.
    s = {"case": case, "t": t, "user": t.register(), "x": x}
    if "index" in x:      # The index is in the table before the calls that count.
        b, o = x.pop("index")
        t.upsert_dev(s["user"], b.data_ptr(), o.data_ptr(), o.numel() - 1, kache.KEEP, 0, 0 if job in ("counter", "served") else 1)
    if "index2" in x:     # Values that differ from k-mer to k-mer.
        b, o = x.pop("index2")
        t.upsert_dev(s["user"], b.data_ptr(), o.data_ptr(), o.numel() - 1, kache.ADD_WRAP, 1, 1)

    def outputs(off, values=True):
        p = max(_positions(off, k), 1)
        s["found"] = torch.zeros(p, dtype=torch.uint8, device="cuda")
        s["values"] = torch.zeros(p, dtype=VALUES[vb], device="cuda") if vb and values else None
        s["fwd"] = torch.zeros(p, dtype=torch.uint8, device="cuda") if job == "oriented" else None

    b, o = x["reads"]
    if job == "host":
        s["batch"] = kache.Batch(b.cpu().numpy(), o.cpu().numpy().astype("uint64"))
    elif job == "count_find":
        outputs(x["held"][1])
    elif job == "counter":
        s["sample"] = min(SAMPLE, case["reads"])
        outputs(o[:s["sample"] + 1])
    elif job == "screen":
        s["counts"] = torch.zeros(case["reads"], dtype=torch.int64, device="cuda")
    elif job == "oriented":
        outputs(o)
        first = torch.zeros(o.numel(), dtype=torch.int64, device="cuda")
        torch.cumsum((o[1:] - o[:-1] - k + 1).clamp_(min=0), 0, out=first[1:])
        first = first.tolist()
        cuts = [(i, min(i + case["call"], case["reads"])) for i in range(0, case["reads"], case["call"])]
        s["ups"] = [(b.data_ptr(), o.data_ptr() + 8 * i, e - i) for i, e in cuts]
        s["looks"] = [(b.data_ptr(), o.data_ptr() + 8 * i, e - i, s["found"].data_ptr() + first[i], s["values"].data_ptr() + vb * first[i],
                       s["fwd"].data_ptr() + first[i]) for i, e in cuts]
    elif job == "served":
        reqs = _requests(case)
        size = {i: _positions(o[i:e + 1], k) if kind == 1 else e - i for kind, i, e in reqs}
        total = [sum(size[i] for kind, i, _ in reqs if kind == q) for q in range(3)]
        s["found"] = torch.zeros(max(total[1], 1), dtype=torch.uint8, device="cuda")
        s["values"] = torch.zeros(max(total[1], 1), dtype=VALUES[vb], device="cuda")
        s["counts"] = torch.zeros(max(total[2], 1), dtype=torch.int64, device="cuda")
        s["runs"], at = ([], [], []), [0, 0, 0]
        for kind, i, e in reqs:
            a = at[kind]
            out = [(), (s["found"].data_ptr() + a, s["values"].data_ptr() + vb * a), (s["counts"].data_ptr() + 8 * a,)][kind]
            s["runs"][kind].append((b.data_ptr(), o.data_ptr() + 8 * i, e - i) + out)
            at[kind] += size[i]
    else:
        outputs(o)
    torch.cuda.synchronize()
    return s


def _look(s, b, off, n):
    v = s["values"]
    s["t"].lookup_dev(b.data_ptr(), off.data_ptr(), n, s["found"].data_ptr(), None if v is None else v.data_ptr(), None)
    return {"found": s["found"]} if v is None else {"found": s["found"], "values": v}


def _calls(s, b, off, n, call, op, x, init):
    """Upserts of n sequences in calls of `call`: the keys inserted."""
    return sum(s["t"].upsert_dev(s["user"], b.data_ptr(), off.data_ptr() + 8 * i, min(call, n - i), op, x, init) for i in range(0, n, call))


def run(s):
    c, t, x = s["case"], s["t"], s["x"]
    job, n, (b, o) = c["job"], c["reads"], x["reads"]
    add = kache.ADD if c["value_bytes"] < 4 else kache.ADD_WRAP
    if job == "find":
        return _look(s, b, o, n)
    if job == "screen":
        t.count_dev(b.data_ptr(), o.data_ptr(), n, s["counts"].data_ptr())
        return {"counts": s["counts"]}
    if job == "counter":
        present = t.update_dev(b.data_ptr(), o.data_ptr(), n, kache.ADD_WRAP, 1)
        return {"present": present, "histogram": t.histogram(HIST).astype("int64"), **_look(s, b, o, s["sample"])}
    if job == "served":
        ups, looks, counts = s["runs"]
        r = {"inserted": sum(t.run_dev_batches(kache.RUN_UPSERT, ups, kache.ADD, 1, 1, s["user"])) if ups else 0,
             "hits": t.run_dev_batches(kache.RUN_LOOKUP, looks) if looks else [],
             "sums": t.run_dev_batches(kache.RUN_COUNT, counts) if counts else []}
        return {**{q: v if q == "inserted" else torch.tensor(v) for q, v in r.items()}, "found": s["found"], "values": s["values"], "counts": s["counts"]}
    t.clear()
    if job == "host":
        ins = t.insert(s["user"], s["batch"], kache.ADD, 1)
        found, values, _ = t.lookup(s["batch"], fwd=False)
        return {"inserted": ins, "found": found, "values": values.astype("int64")}
    if job == "stream":
        return {"inserted": _calls(s, b, o, n, c["call"], add, 1, 1), **_look(s, b, o, n)}
    if job == "count_find":
        hb, ho = x["held"]
        return {"inserted": t.upsert_dev(s["user"], b.data_ptr(), o.data_ptr(), n, add, 1, 1), **_look(s, hb, ho, c["held"])}
    if job == "grow":
        pb, po = x["pieces"]
        return {"inserted": _calls(s, pb, po, po.numel() - 1, c["call"], kache.KEEP, 0, 0), **_look(s, b, o, n)}
    ins = sum(t.run_dev_batches(kache.RUN_UPSERT_ORIENTED, s["ups"], kache.OR, 1, 2, s["user"]))
    hits = t.run_dev_batches(kache.RUN_LOOKUP, s["looks"])
    return {"inserted": ins, "hits": torch.tensor(hits), "found": s["found"], "values": s["values"], "fwd": s["fwd"]}


def work(case):
    """The bytes of one pass: every base and offset read once, every per-position output written once, and every distinct
    k-mer that the pass's calls touch read (and, where they change it, written) once, as its key and value."""
    k, job, vb, g = case["k"], case["job"], case["value_bytes"], case["genome"]
    mean = case["length"] * math.exp(case["sigma"] ** 2 / 2) if case["sigma"] else min(case["length"], g)
    bases = case["reads"] * mean
    pos = case["reads"] * max(mean - k + 1, 1)
    out, keys, extra = 1 + vb, min(g, pos), 8 * case["reads"]
    entry = 8 + vb
    total = bases + extra
    if job == "find":
        total += pos * out + keys * entry
    elif job == "stream" or job == "host":
        total += bases + extra + pos * out + 3 * keys * entry
    elif job == "count_find":
        held = case["held"] * max(mean - k + 1, 1)
        total += case["held"] * (mean + 8) + held * out + 2 * keys * entry + min(g, held) * entry
    elif job == "counter":
        sample = min(SAMPLE, case["reads"]) * max(mean - k + 1, 1)
        total += 2 * keys * entry + g * entry + sample * out + 8 * HIST
    elif job == "oriented":
        total += bases + extra + pos * (out + 1) + 3 * keys * entry
    elif job == "grow":
        total += g * (1 + 8 * (150 - k + 1) / 150) + pos * out + min(g, pos) * 8
    elif job == "served":
        total += 0.3 * pos * out + 1.6 * keys * entry
    else:
        total += 8 * case["reads"] + min(g, pos) * entry
    return {"bytes": float(total), "flops": 0.0}


# ---- What the calls return, from sorted arrays ---------------------------------------------------------------------

def _kmers(bases, off, k):
    """The canonical k-mers at all positions of the sequences, in order, whether each is one (only ACGT) and whether it
    occurs as its canonical form. As 64-bit patterns with the top bit flipped, so that signed order is theirs."""
    n = int(off[-1])
    codes = torch.full((256,), 4, dtype=torch.int64, device="cuda")
    for i, ch in enumerate(b"ACGT"):
        codes[ch] = i
    c = codes[bases[:n].long()]
    bad = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(c == 4, 0, out=bad[1:])
    f, r = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.int64, device="cuda")
    for j in range(k):
        m = n - j
        if m <= 0:
            break
        f[:m] |= (c[j:] & 3) << (2 * (k - 1 - j))
        r[:m] |= (3 - (c[j:] & 3)) << (2 * j)
    lens = (off[1:] - off[:-1] - k + 1).clamp_(min=0)
    q = torch.repeat_interleave(torch.arange(lens.numel(), device="cuda"), lens)
    start = torch.cumsum(lens, 0) - lens
    p = torch.arange(q.numel(), device="cuda") - start[q] + off[:-1][q]
    top = torch.iinfo(torch.int64).min
    f, r = f[p] ^ top, r[p] ^ top
    ok = bad[p + k] == bad[p]
    return torch.minimum(f, r), ok, f <= r, q


def _at(keys, query):
    """Each query's index in the sorted distinct keys, and whether it is there."""
    if not keys.numel():
        return torch.zeros_like(query), torch.zeros_like(query, dtype=torch.bool)
    i = torch.searchsorted(keys, query).clamp_(max=keys.numel() - 1)
    return i, keys[i] == query


def _found(keys, vals, batch, k, vb, fwd=False):
    q, ok, f, _ = _kmers(*batch, k)
    i, hit = _at(keys, q)
    hit &= ok
    r = {"found": torch.where(ok, hit.to(torch.uint8), torch.full_like(ok, 2, dtype=torch.uint8))}
    if vb:
        r["values"] = torch.where(hit, vals[i], torch.zeros_like(i)).to(VALUES[vb])
    if fwd:
        r["fwd"] = (ok & f).to(torch.uint8)
    return r


def exact(case, seed):
    k, job, vb = case["k"], case["job"], case["value_bytes"]
    x = _inputs(case, seed)
    (b, o), n = x["reads"], case["reads"]
    most = {1: 255, 2: 65535}.get(vb, 1 << 62)

    def valid(name, kk=k):
        q, ok, f, s = _kmers(*x[name], kk)
        return q[ok], f[ok], s[ok]

    if job in ("find", "counter", "served", "screen"):
        keys = torch.unique(valid("index")[0])
        vals = torch.full((keys.numel(),), 0 if job in ("counter", "served") else 1, dtype=torch.int64, device="cuda")
    if job == "find":
        more, num = torch.unique(valid("index2")[0], return_counts=True)
        i, hit = _at(keys, more)
        vals.index_add_(0, i[hit], num[hit])
        keys, order = torch.sort(torch.cat([keys, more[~hit]]))
        return _found(keys, torch.cat([vals, num[~hit]])[order], (b, o), k, vb)    # Wrapping, as the narrower values do.
    if job == "screen":
        q, _, s = valid("reads")
        return {"counts": torch.bincount(s[_at(keys, q)[1]], minlength=n)}
    if job == "counter":
        q, _, _ = valid("reads")
        i, hit = _at(keys, q)
        vals = torch.bincount(i[hit], minlength=keys.numel())
        h = torch.bincount(vals.clamp(max=HIST + 1), minlength=HIST + 2)[:HIST + 1]
        h[0] = 0
        m = min(SAMPLE, n)
        return {"present": int(hit.sum()), "histogram": h, **_found(keys, vals, (b, o[:m + 1]), k, vb)}
    if job == "served":
        reqs = _requests(case)

        def slice_kmers(i, e):
            at = int(o[i])
            q, ok, _, s = _kmers(b[at:], o[i:e + 1] - at, k)
            return q, ok, s

        ups = [q[ok] for q, ok, _ in (slice_kmers(i, e) for kind, i, e in reqs if kind == 0)]
        more, num = torch.unique(torch.cat(ups), return_counts=True) if ups else (keys[:0], keys[:0])
        i, hit = _at(keys, more)
        vals.index_add_(0, i[hit], num[hit])
        keys, order = torch.sort(torch.cat([keys, more[~hit]]))
        vals = torch.cat([vals, num[~hit]])[order]
        out, hits, sums = {"found": [], "values": [], "counts": []}, [], []
        for kind, i, e in reqs:
            at, sub = int(o[i]), o[i:e + 1] - int(o[i])
            if kind == 1:
                r = _found(keys, vals, (b[at:], sub), k, vb)
                out["found"].append(r["found"]), out["values"].append(r["values"]), hits.append(int((r["found"] == 1).sum()))
            elif kind == 2:
                q, ok, s = slice_kmers(i, e)
                out["counts"].append(torch.bincount(s[ok & _at(keys, q)[1]], minlength=e - i))
                sums.append(int(out["counts"][-1].sum()))
        return {"inserted": int((~hit).sum()), "hits": torch.tensor(hits), "sums": torch.tensor(sums),
                **{q: torch.cat(v) if v else torch.zeros(1, dtype=d, device="cuda") for (q, v), d in zip(out.items(), (torch.uint8, VALUES[vb], torch.int64))}}
    if job == "grow":
        keys = torch.unique(valid("pieces")[0])
        return {"inserted": keys.numel(), **_found(keys, None, (b, o), k, 0)}
    if job == "oriented":
        q, f, _ = valid("reads")
        keys, at = torch.unique(q, return_inverse=True)
        vals = torch.zeros(keys.numel(), dtype=torch.int64, device="cuda")
        for bit, m in ((1, f), (2, ~f)):
            vals[at[m]] |= bit
        r = _found(keys, vals, (b, o), k, vb, True)
        lens = (o[1:] - o[:-1] - k + 1).clamp_(min=0)
        start = torch.cumsum(lens, 0) - lens
        ends = torch.cat([start, lens.sum().reshape(1)]).tolist()
        hits = [int((r["found"][ends[i]:ends[min(i + case["call"], n)]] == 1).sum()) for i in range(0, n, case["call"])]
        return {"inserted": keys.numel(), "hits": torch.tensor(hits), **r}
    keys, num = torch.unique(valid("reads")[0], return_counts=True)
    num = num.clamp_(max=most)
    r = {"inserted": keys.numel(), **_found(keys, num, x["held"] if job == "count_find" else (b, o), k, vb)}
    if job == "host":
        r["values"] = r["values"].long()
    return r
