// The warp describer and the streaming kernel: one warp describes a segment of a sequence, 32 k-mer positions per
// row, and hands each row's k-mers to a visitor (upsert, update, lookup, count, ...), one k-mer per lane.
//
// What it computes per position is the reference describers' description (include/Kmer_Batch.hpp:191-250,
// include/Kmer_Lanes.hpp:164-244) with this library's placement hash (device_common.cuh): the canonical key, its
// orientation, its checksum and its minimizer hash. How:
//   - each row of 32 bases is loaded coalesced (lane j reads base j); three ballots per row hold its ACGT flags and its
//     codes' high and low bits, base j at bit j;
//   - lane j's k-mer is a window of k bits of each plane, one funnel shift of two consecutive rows. First base lowest,
//     its complement is the reverse complement's plane; bit-reversed, it is the forward plane;
//   - the l-mer at a k-mer's start is a shift of its forward planes and a mask of its reverse ones. Each lane hashes
//     that one; the minima of neighbouring pairs of hashes go to a per-warp ring in shared memory, and a k-mer's
//     minimizer hash, the least of the w = k - l + 1 hashes from its own position on, is the least of ceil(w / 2) pair
//     minima;
//   - non-ACGT characters split sequences (DNA_Utility.hpp:199-224): a window with one is not a k-mer.
// Every operation runs so, also those without per-position outputs: consecutive k-mers share minimizers, so a row of 32
// touches about seven buckets where 32 lanes on 32 different reads would touch 32 (a lane per segment, rolling its k-mers,
// took 9.19 ms for 130M upserts into a 6.7 GB map, rows 2.8 ms; 7.1 against 3.6 ms for 190M updates).
//
// What bounds it is instructions (327 per row in a lookup of 150 bp reads, issue slots two thirds used), then the latency
// of three dependent loads; so more resident warps pay even at the price of some spills: six blocks of 256 threads per SM
// (40 registers) against five (48, half the spills), with the work counter: an upsert of 40M positions and a lookup of 120M 2.90
// against 2.98 ms, counts of 1M reads 1.33 against 1.39, 190M updates with a histogram 4.52 against 4.77, 40M lookups of
// contigs 0.55 against 0.58. (Four and three, with fixed shares of segments, when six took 1.81 and 1.08 ms: lookup 1.80,
// overlapping two rows, and 2.29 ms, upsert 1.15 and 1.46.)
// Sequences are cut into segments of up to `seg_positions` positions; each segment re-reads the k - 1 bases it
// shares with the next, so segments, like the reference's lanes (include/Streaming_Kmer_Hash_Table.hpp:1751-1781),
// need no state from one another.
#pragma once

#include "device_table.cuh"

namespace kache_b200
{

// A segment: up to seg_len consecutive k-mer positions of one sequence, with all that a warp needs to start on it in one
// 32-byte entry.
struct alignas(16) Segment
{
    uint64_t base;      // Its first base, as an offset from the batch's bases.
    uint64_t pos;       // Its first position, counted over the batch's sequences.
    uint64_t q;         // Its sequence.
    uint32_t npos;      // Its positions. (Of a group, see below: group_word.)
    uint32_t batch;     // Its batch, of several run as one.
};

// A group: group_seqs sequences, in order and of one batch, of up to group_len bases each, whose k-mers are a warp's rows of 32
// together (group_kernel); its entry has its first sequence's q, and base and pos where that starts. Sequences of few k-mers
// leave most lanes of a row idle by themselves: 2M reads of 33 bases, three 31-mers each, took 1,040 us to count and 1,484 to
// upsert, in groups 341 and 503.
constexpr uint32_t group_seqs = 8, group_len = 124;

__device__ __forceinline__ uint32_t group_word(const uint32_t npos, const uint32_t bases) { return bases << 10 | npos; }

// What visitors get of a segment.
struct Seg_Of
{
    uint64_t q, pos;
    uint32_t batch;
};

// A batch on the device: its segments in sequence order. Several batches run as one have no bases in common (null): their
// segments' offsets are addresses.
struct Dev_Batch
{
    const uint8_t* bases;
    const Segment* segs;
    // Groups, and for them where each sequence starts, as Segment::base says, and the positions before it.
    const Segment* groups;
    const uint64_t* start;
    const uint64_t* pos_off;
};

constexpr int stream_warps = 8;

// One row of 32 bases: base j's flag (one of A, C, G, T) and code bits at bit j.
struct Row
{
    uint32_t hi, lo, valid;
};

constexpr int base_table_bytes = 256;

// Fills a block's table of base_bits by character, in shared memory (one load per base in place of the tests).
__device__ __forceinline__ void fill_base_table(uint8_t* tab)
{
    for(uint32_t ch = threadIdx.x; ch < base_table_bytes; ch += blockDim.x)
        tab[ch] = base_bits(ch);
    __syncthreads();
}

// A row of characters, one per lane.
__device__ __forceinline__ Row pack_row(const uint32_t ch, const uint8_t* tab)
{
    constexpr uint32_t all = 0xFFFFFFFFu;
    const uint32_t t = tab[ch];
    Row r;
    r.valid = __ballot_sync(all, t & 1u);
    r.lo = __ballot_sync(all, t & 2u);
    r.hi = __ballot_sync(all, t & 4u);
    return r;
}

// A k-mer as the visitors get it.
struct Kmer_Desc
{
    uint64_t key;       // Its canonical form's planes.
    uint32_t pos;       // Position in the segment.
    uint32_t h;         // Minimizer hash.
    bool fwd;           // Occurs as its canonical form.
    bool valid;         // All k characters are ACGT.
    bool in;            // The position exists (is in the segment).
};

constexpr int ring_words = 96;  // A warp's ring: two rows of 32, then a copy of the first row (entries up to w <= 32).

// A row's k-mers as a row ahead of the visits holds them: the canonical key and two flags.
struct Row_Kmers
{
    uint64_t key;
    bool fwd, acgt;
};

// This lane's k-mer in the window that starts in row a, and the hash of the l-mer that it starts with.
template <int k, int l>
__device__ __forceinline__ Row_Kmers window(const Row& a, const Row& b, const uint32_t lane, uint32_t& lmer)
{
    constexpr uint32_t km = (k == 32 ? ~0u : (1u << k) - 1), lm = (1u << l) - 1;
    const uint32_t hi = __funnelshift_r(a.hi, b.hi, lane), lo = __funnelshift_r(a.lo, b.lo, lane);
    const Planes f{__brev(hi) >> (32 - k), __brev(lo) >> (32 - k)}, r{~hi & km, ~lo & km};
    const bool gt = planes_greater(f, r);
    Row_Kmers x;
    x.key = gt ? key_of(r) : key_of(f);
    x.fwd = !gt;
    x.acgt = (__funnelshift_r(a.valid, b.valid, lane) & km) == km;
    lmer = lmer_hash(Planes{f.hi >> (k - l), f.lo >> (k - l)}, Planes{r.hi & lm, r.lo & lm});
    return x;
}

// Describes a segment of npos positions, whose bases start at seq, to the visitor, by a whole warp.
template <int k, int l, typename Visitor>
__device__ __forceinline__ void describe_segment(const uint8_t* const seq, const uint32_t npos, uint32_t* const ring, const uint8_t* const tab,
                                                 const uint32_t lane, Visitor& vis)
{
    constexpr int w = k - l + 1;
    static_assert(k <= 32 && l < k && w <= 32, "k-mers in a machine word, minimizers of at least two l-mers");
    constexpr uint32_t all = 0xFFFFFFFFu;
    const uint32_t bases = npos + k - 1;
    // Characters are asked for a row ahead of their use: L1 returns loads in order, so one waited for at once would wait
    // for the table's sectors that other warps miss in front of it.
    const auto load = [&](const uint32_t o) -> uint32_t { return o + lane < bases ? __ldg(seq + o + lane) : 0u; };
    const uint32_t ch0 = load(0), ch1 = load(32);
    uint32_t ch = load(64);

    // Ring entry 32 (r & 1) + j is min(H[i - 1], H[i]) for position i = 32 r + j of the segment, where H are the l-mer
    // hashes; rows r and r + 1 are held. An even row's first entries are also at 64 + j, so that a window of an odd row
    // reads past its end.
    const Row r0 = pack_row(ch0, tab);
    Row r1 = pack_row(ch1, tab);
    uint32_t hash;      // Of this lane's l-mer in the newest row described.
    Row_Kmers x = window<k, l>(r0, r1, lane, hash);
    const uint32_t left = __shfl_up_sync(all, hash, 1);
    ring[lane] = min(left, hash);   // Entry 0 is never read.

    // The k-mers of the row at offset o, whose windows were taken when the row before was described; takes the next
    // row's windows, whose first hashes this row's minimizers need.
    const auto describe = [&](const uint32_t o)
    {
        const uint32_t half = o & 32;
        __syncwarp();       // The previous row's reads of the ring are done.
        const Row r2 = pack_row(ch, tab);
        ch = load(o + 96);
        const uint32_t last = __shfl_sync(all, hash, 31);
        const Row_Kmers y = window<k, l>(r1, r2, lane, hash);
        const uint32_t up = __shfl_up_sync(all, hash, 1), pair = min(lane ? up : last, hash);
        ring[(half ^ 32) + lane] = pair;
        if(half && lane < w)
            ring[64 + lane] = pair;
        __syncwarp();

        Kmer_Desc d;
        d.pos = o + lane;
        d.in = d.pos < npos;
        d.valid = d.in && x.acgt;
        d.key = x.key;
        d.fwd = x.fwd;
        // Pairs (i - 1, i) at i = j + 1, j + 3, ...: w / 2 of them cover [j, j + w - 1] for even w; for odd w the
        // pair at j + w - 1 adds the last hash.
        const uint32_t* at = ring + half + lane;
        d.h = at[1];
#pragma unroll
        for(int i = 3; i < w; i += 2)
            d.h = min(d.h, at[i]);
        if constexpr(w % 2 == 1)
            d.h = min(d.h, at[w - 1]);
        r1 = r2, x = y;
        return d;
    };

#pragma unroll 1
    for(uint32_t o = 0; o < npos; o += 32)
        vis.visit(describe(o), lane);
    __syncwarp();
}

template <int k, int l, typename Visitor>
__global__ void __launch_bounds__(32 * stream_warps, Visitor::min_blocks) stream_kernel(const Dev_Batch batch, const uint64_t seg_b, const uint64_t segs_end,
                                                                                        const unsigned long long* run, unsigned long long* taken, Visitor vis)
{
    // The segments [seg_b, segs_end), or as many as `run` says, counted by the kernel before.
    const uint64_t seg_e = run ? static_cast<uint64_t>(*run) : segs_end;
    __shared__ uint32_t ring_all[stream_warps][ring_words];
    __shared__ uint8_t tab[base_table_bytes];
    fill_base_table(tab);
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    vis.begin();
    // After its first segment a warp takes more, a few at a time, from the counter `taken` (zero before the launch); without
    // one every warp has a fixed share (see Engine::shares).
    const uint64_t warps = uint64_t(gridDim.x) * stream_warps, nsegs = seg_e > seg_b ? seg_e - seg_b : 0;
    const uint64_t some = max(uint64_t(1), min(uint64_t(4), nsegs / (warps * 8)));
    const auto take = [&]() -> uint64_t
    {
        unsigned long long g = 0;
        if(lane == 0)
            g = atomicAdd(taken, static_cast<unsigned long long>(some));
        return warps + __shfl_sync(0xFFFFFFFFu, g, 0);
    };
    // A segment's entry is asked for a segment ahead, a word per lane.
    const auto ask = [&](const uint64_t g) -> uint32_t
    {
        return g < nsegs && lane < sizeof(Segment) / 4 ? __ldg(reinterpret_cast<const uint32_t*>(batch.segs + seg_b + g) + lane) : 0u;
    };
    uint64_t g = uint64_t(blockIdx.x) * stream_warps + wid, left = 1;
    for(uint32_t entry = ask(g); g < nsegs; )
    {
        const auto word = [&](const int i) { return __shfl_sync(0xFFFFFFFFu, entry, i); };
        const auto wide = [&](const int i) { return uint64_t(word(i + 1)) << 32 | word(i); };
        const uint64_t base = wide(0);
        const Seg_Of s{wide(4), wide(2), word(7)};
        const uint32_t npos = word(6);
        if(!taken)
            g += warps;
        else if(--left)
            ++g;
        else
            g = take(), left = some;
        entry = ask(g);
        vis.begin_segment(s);
        describe_segment<k, l>(batch.bases + base, npos, ring_all[wid], tab, lane, vis);
        vis.end_segment(s, lane);
    }
    vis.end(lane);
}

// The planes of a group's bases, end to end in `planes`: 32 words each of high and low code bits and of flags.
__device__ __forceinline__ void pack_group(const uint8_t* const seq, const uint32_t bases, uint32_t* const planes, const uint8_t* const tab, const uint32_t lane)
{
#pragma unroll 1
    for(uint32_t o = 0; o < bases; o += 128)
    {
        uint32_t ch[4];
#pragma unroll
        for(int i = 0; i < 4; ++i)
            ch[i] = o + 32 * i + lane < bases ? __ldg(seq + o + 32 * i + lane) : 0u;
#pragma unroll
        for(int i = 0; i < 4; ++i)
        {
            const Row r = pack_row(ch[i], tab);
            if(lane == 0)
                planes[o / 32 + i] = r.hi, planes[32 + o / 32 + i] = r.lo, planes[64 + o / 32 + i] = r.valid;
        }
    }
    __syncwarp();
}

// The k-mer at position j of a group, whose sequence number i starts at first (in lane i) of its positions and `from` of its
// bases; its sequence's number goes to `i`. The lanes' k-mers are not all neighbours, so each lane hashes the w l-mers of
// its own.
template <int k, int l>
__device__ __forceinline__ Kmer_Desc group_kmer(const uint32_t j, const uint32_t* const planes, const uint32_t first, const uint32_t from, uint32_t& i)
{
    constexpr uint32_t all = 0xFFFFFFFFu, km = (k == 32 ? ~0u : (1u << k) - 1), lm = (1u << l) - 1;
    i = 0;      // The last one that starts at or before j.
#pragma unroll
    for(uint32_t step = group_seqs / 2; step; step /= 2)
        i += __shfl_sync(all, first, i + step) <= j ? step : 0;
    const uint32_t b = __shfl_sync(all, from, i) + (j - __shfl_sync(all, first, i));
    const uint32_t* p = planes + (b >> 5);
    const uint32_t hi = __funnelshift_r(p[0], p[1], b), lo = __funnelshift_r(p[32], p[33], b);
    const Planes f{__brev(hi) >> (32 - k), __brev(lo) >> (32 - k)}, r{~hi & km, ~lo & km};
    const bool gt = planes_greater(f, r);
    Kmer_Desc d;
    d.key = gt ? key_of(r) : key_of(f);
    d.fwd = !gt;
    d.valid = (__funnelshift_r(p[64], p[65], b) & km) == km;
    d.h = ~0u;
#pragma unroll
    for(int x = 0; x <= k - l; ++x)
        d.h = min(d.h, lmer_hash(Planes{(f.hi >> (k - l - x)) & lm, (f.lo >> (k - l - x)) & lm}, Planes{(r.hi >> x) & lm, (r.lo >> x) & lm}));
    return d;
}

// The kernel over groups [grp_b, grp_end), or as many as `run` says, counted by the kernel before. A row costs some 430
// instructions, where a segment's costs 330 and its start 120: which sequences make a group is staging's choice (`group_saves`).
// A kernel of its own, behind the one over segments: as a branch of that one it cost the rows of 150 bp reads 4 to 6 %, whose
// registers are few enough as it is, and with one loop for both kinds of row they took three times as long.
template <int k, int l, typename Visitor>
__global__ void __launch_bounds__(32 * stream_warps, Visitor::min_blocks) group_kernel(const Dev_Batch batch, const uint64_t grp_b, const uint64_t grp_end, const unsigned long long* run, Visitor vis)
{
    __shared__ uint32_t planes_all[stream_warps][96];
    __shared__ uint8_t tab[base_table_bytes];
    fill_base_table(tab);
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr uint32_t all = 0xFFFFFFFFu;
    uint32_t* const planes = planes_all[wid];
    vis.begin();
    const uint64_t grp_e = run ? static_cast<uint64_t>(*run) : grp_end, warps = uint64_t(gridDim.x) * stream_warps;
    for(uint64_t g = grp_b + uint64_t(blockIdx.x) * stream_warps + wid; g < grp_e; g += warps)
    {
        const Segment e = batch.groups[g];
        const Seg_Of s{e.q, e.pos, e.batch};
        const uint32_t npos = e.npos & 0x3FFu;
        // Lane i has where the group's sequence i starts, in its bases and in its positions.
        uint32_t from = 0, first = ~0u;
        if(lane < group_seqs)
            from = static_cast<uint32_t>(batch.start[s.q + lane] - e.base), first = static_cast<uint32_t>(batch.pos_off[s.q + lane] - s.pos);
        pack_group(batch.bases + e.base, e.npos >> 10, planes, tab, lane);
        vis.begin_segment(s);
#pragma unroll 1
        for(uint32_t o = 0; o < npos; o += 32)
        {
            uint32_t i;
            Kmer_Desc d = group_kmer<k, l>(min(o + lane, npos - 1), planes, first, from, i);
            d.pos = o + lane;
            d.in = d.pos < npos;
            d.valid = d.valid && d.in;
            vis.visit(d, lane);
            if constexpr(requires { vis.end_group_row(s, i, lane); })
                vis.end_group_row(s, i, lane);
        }
        vis.end_segment(s, lane);
        __syncwarp(all);
    }
    vis.end(lane);
}

// ---- Visitors -------------------------------------------------------------------------------------------------

// Per-warp counter flush: one atomic per warp at the end of the kernel.
__device__ __forceinline__ void warp_flush(unsigned long long* ctr, const unsigned long long c, const uint32_t lane)
{
    if(lane == 0 && c)
        atomicAdd(ctr, c);
}

// Finds a row's k-mers, for visitors that insert nothing: `hit` where the key is present, its value then in `val` (with
// val_), its place in (at, slot) (value_word). What few lanes need, candidates past the second and what lies beyond a full
// bucket, is behind a branch of the whole warp.
template <bool set_, bool val_>
struct Found
{
    bool hit;
    uint32_t at;
    uint64_t slot;
    unsigned long long val;

    __device__ __forceinline__ Found(const Dev_Table& T, const Kmer_Desc& d)
    {
        const Probe p = probe_primary<set_, false, val_>(T, d.valid, d.key, d.h);
        at = bucket_of(d.h, T.cap), slot = p.slot, val = p.val;
        hit = p.slot < B;
        const bool on = !hit && (p.rest != 0 || p.full);
        if(__any_sync(0xFFFFFFFFu, on))
        {
            if(on)
                hit = find_on<set_, false, val_>(T, at, slot, p.rest, p.full, ~d.key, d.h, val);
            __syncwarp();
        }
    }
};

// Upsert / insert / upsert_oriented (include/Streaming_Kmer_Hash_Table.hpp:2219-2514): returns the keys inserted;
// k-mers that found the overflow table full set their bit in `retry_out` and change nothing. In retry mode, only
// the positions whose bit is set in `retry_in` run.
template <bool set_, typename V, typename Fn>
struct Upsert_Visitor
{
    static constexpr int min_blocks = 6;
    Dev_Table T;
    Fn fn;
    unsigned long long* inserted;
    unsigned int* retry_out;
    const unsigned int* retry_in;
    unsigned int* retried;      // Set to 1 if any bit of retry_out was set.
    unsigned long long* per;        // If set, the keys inserted are added there per sequence, or
    bool by_batch;                  // per batch.
    unsigned long long ins = 0;     // By this warp, before its current segment.
    uint32_t seg_ins = 0;           // In the current segment,
    uint64_t seg_pos = 0;           // whose first position this is.

    __device__ __forceinline__ void begin() {}
    __device__ __forceinline__ void begin_segment(const Seg_Of& s) { seg_ins = 0, seg_pos = s.pos; }
    __device__ __forceinline__ void end_segment(const Seg_Of& s, const uint32_t lane)
    {
        ins += seg_ins;
        if(per && lane == 0 && seg_ins)
            atomicAdd(per + (by_batch ? s.batch : s.q), static_cast<unsigned long long>(seg_ins));
    }

    __device__ __forceinline__ void visit(const Kmer_Desc& d, const uint32_t lane)
    {
        constexpr uint32_t all = 0xFFFFFFFFu;
        bool active = d.valid;
        if(retry_in && active)
        {
            const uint64_t gpos = seg_pos + d.pos;
            active = (retry_in[gpos >> 5] >> (gpos & 31)) & 1;
        }

        const unsigned long long key_st = ~d.key;
        const Probe p = probe_primary<set_, true, false>(T, active, d.key, d.h);
        uint32_t j = p.slot, r = j < B ? FOUND : NONE, at = active ? bucket_of(d.h, T.cap) : no_bucket;
        uint64_t ov_i = 0;
        const uint32_t need_m = __ballot_sync(all, active && r == NONE);
        if(need_m)
        {
            // Of lanes with one key, the first upserts it; the others then update it where it is. (The chain reads the
            // bucket again: its checksums would take registers that other warps need.)
            const bool need = active && r == NONE;
            uint32_t lead = lane;
            if(need)
                lead = __ffs(__match_any_sync(need_m, key_st)) - 1;
            warp_claim<set_>(T, key_st, d.h, checksum_of(d.key), lane, need && lead == lane, at, j, r, ov_i);
            if(__any_sync(all, lead != lane))
            {
                const uint32_t r_l = __shfl_sync(all, r, lead), at_l = __shfl_sync(all, at, lead), j_l = __shfl_sync(all, j, lead);
                const uint64_t ov_l = __shfl_sync(all, ov_i, lead);
                if(lead != lane)
                    r = r_l == OV_FULL ? OV_FULL : FOUND_PENDING, at = at_l, j = j_l, ov_i = ov_l;
            }
        }

        // A claimed slot is published after its value is written; where the operation commutes, from a zeroed value, it is
        // published at once and its initial value is then one more update.
        const bool comm = fn.commutes(), main = at != no_bucket;
        unsigned long long* const val = main ? key_word<set_>(T, at, j) + 1 : T.ov + 4 * ov_i + 1;
        if(r == INSERTED)
        {
            if constexpr(!set_)
                if(!comm)
                    write_val<V>(val, fn.initial(d.fwd)), __threadfence();
            if(main)
                *reinterpret_cast<volatile uint8_t*>(cs_of(T, at, j)) = static_cast<uint8_t>(checksum_of(d.key));
            else
            {
                *reinterpret_cast<volatile unsigned long long*>(val + 1) = 1ull;
                atomicAdd(T.ov_count, 1ull);
            }
        }
        else if(r == OV_FULL)
        {
            const uint64_t gpos = seg_pos + d.pos;
            atomicOr(retry_out + (gpos >> 5), 1u << (gpos & 31));
            *retried = 1;
        }
        const uint32_t ins_m = __ballot_sync(all, r == INSERTED);
        seg_ins += __popc(ins_m);

        if constexpr(!set_)
        {
            if(comm)
            {
                if(r == INSERTED || ((r == FOUND || r == FOUND_PENDING) && !fn.is_noop()))
                    fn.apply_or_init(val, d.fwd, r == INSERTED);
            }
            else if(r == FOUND || r == FOUND_PENDING)
            {
                if(r == FOUND_PENDING && !await_published(Landing{val, main ? cs_of(T, at, j) : nullptr, main ? nullptr : val + 1, 0}, T.wait_polls))
                    atomicOr(T.err, ERR_WAIT);
                fn.apply(val, d.fwd);
            }
        }
    }

    __device__ __forceinline__ void end(const uint32_t lane) { warp_flush(inserted, ins, lane); }
};

// Present-only update (include/Streaming_Kmer_Hash_Table.hpp:2650-2691): returns the k-mers present, repeats counted.
// Nothing is inserted meanwhile, so checksums and keys are read through L1; only values change, atomically.
template <typename V, typename Fn>
struct Update_Visitor
{
    static constexpr int min_blocks = 6;
    Dev_Table T;
    Fn fn;
    unsigned long long* present;
    unsigned long long* per_batch;  // If set, the k-mers present are added there per batch.
    unsigned long long cnt = 0;     // By this warp, before its current segment.
    uint32_t seg_cnt = 0;           // In the current segment.

    __device__ __forceinline__ void begin() {}
    __device__ __forceinline__ void begin_segment(const Seg_Of&) { seg_cnt = 0; }
    __device__ __forceinline__ void end_segment(const Seg_Of& s, const uint32_t lane)
    {
        cnt += seg_cnt;
        if(per_batch && lane == 0 && seg_cnt)
            atomicAdd(per_batch + s.batch, static_cast<unsigned long long>(seg_cnt));
    }

    __device__ __forceinline__ void visit(const Kmer_Desc& d, const uint32_t)
    {
        const Found<false, false> f(T, d);
        if(f.hit)
            fn.apply(value_word<false>(T, f.at, f.slot), d.fwd);
        seg_cnt += __popc(__ballot_sync(0xFFFFFFFFu, f.hit));
    }

    __device__ __forceinline__ void end(const uint32_t lane) { warp_flush(present, cnt, lane); }
};

// Per-position lookup (capi/Kmer_Table.hpp:163-190): found (0 absent, 1 present, 2 not a k-mer), value, orientation
// at pos_off[q] + i.
template <bool set_, typename V>
struct Lookup_Visitor
{
    static constexpr int min_blocks = 6;
    Dev_Table T;
    uint8_t* found;
    V* values;
    uint8_t* fwd;
    uint64_t obase = 0;     // The current segment's first position in them.

    __device__ __forceinline__ void begin() {}
    __device__ __forceinline__ void begin_segment(const Seg_Of& s) { obase = s.pos; }
    __device__ __forceinline__ void end_segment(const Seg_Of&, uint32_t) {}
    __device__ __forceinline__ void end(uint32_t) {}

    __device__ __forceinline__ void visit(const Kmer_Desc& d, const uint32_t) { look(d); }
    // Looks the k-mer up and writes its outputs; whether it is present.
    __device__ __forceinline__ bool look(const Kmer_Desc& d)
    {
        const Found<set_, !set_> f(T, d);
        if(!d.in)
            return false;
        const uint64_t o = obase + d.pos;
        found[o] = d.valid ? (f.hit ? 1 : 0) : 2;
        if constexpr(!set_)
            if(values)
                values[o] = f.hit ? value_of<V>(f.val) : V(0);
        if(fwd)
            fwd[o] = d.valid && d.fwd;
        return f.hit;
    }
};

// Lookups of several batches run as one: each segment's outputs go to its own batch's arrays, at its positions within
// that batch, and the positions found are added at per_batch.
template <bool set_, typename V>
struct Lookup_Batches_Visitor : Lookup_Visitor<set_, V>
{
    const uint64_t* outs;       // Per batch, 8 words: found, values, fwd at words 4-6 (device addresses, or 0).
    const uint64_t* pos_base;   // Per batch: the merged position of its first k-mer.
    unsigned long long* per_batch;
    uint32_t hits = 0;          // In the current segment.

    __device__ __forceinline__ void begin_segment(const Seg_Of& s)
    {
        const uint64_t* o = outs + 8 * uint64_t(s.batch);
        this->found = reinterpret_cast<uint8_t*>(o[4]);
        this->values = reinterpret_cast<V*>(o[5]);
        this->fwd = reinterpret_cast<uint8_t*>(o[6]);
        this->obase = s.pos - pos_base[s.batch];
        hits = 0;
    }
    __device__ __forceinline__ void visit(const Kmer_Desc& d, const uint32_t)
    {
        const bool hit = this->look(d);
        hits += __popc(__ballot_sync(0xFFFFFFFFu, hit));
    }
    __device__ __forceinline__ void end_segment(const Seg_Of& s, const uint32_t lane)
    {
        if(lane == 0 && hits)
            atomicAdd(per_batch + s.batch, static_cast<unsigned long long>(hits));
    }
};

// Per-sequence reductions over lookups (capi/Kmer_Table.hpp:134-161): 0 count, 1 masked count, 2 sum. A segment
// belongs to one sequence, so each warp adds its segment's total once; of a group's row, each sequence's lanes add theirs.
template <bool set_, typename V, int mode_>
struct Seq_Reduce_Visitor
{
    static constexpr int min_blocks = 6;
    Dev_Table T;
    unsigned long long* out;
    V m_fwd, m_rev;
    // Of the current segment: a lane's sum (2), or the warp's count (0, 1), by votes: added up by lane, and by five shuffles of
    // 64 bits at its end, counts of 1.5M reads of 56 bases, a row each, took 791 us against 754, of 1M reads 1329 against 1295.
    unsigned long long acc = 0;
    uint32_t cnt = 0;
    uint32_t ones = 0;      // The lanes that counted in the current row.

    __device__ __forceinline__ void begin() {}
    __device__ __forceinline__ void begin_segment(const Seg_Of&) { acc = 0, cnt = 0; }
    // What the k-mer adds.
    __device__ __forceinline__ unsigned long long term(const Kmer_Desc& d) const
    {
        const Found<set_, !set_ && mode_ != 0> f(T, d);
        if(!f.hit)
            return 0;
        if constexpr(mode_ == 0)
            return 1;
        else if constexpr(mode_ == 1)
            return (value_of<V>(f.val) & (d.fwd ? m_fwd : m_rev)) != 0;
        else
            return static_cast<unsigned long long>(value_of<V>(f.val));
    }
    __device__ __forceinline__ void visit(const Kmer_Desc& d, const uint32_t)
    {
        const unsigned long long x = term(d);
        if constexpr(mode_ == 2)
            acc += x;
        else
            ones = __ballot_sync(0xFFFFFFFFu, x != 0), cnt += __popc(ones);
    }
    // After a group's row, whose lanes are of the group's sequences i in order: adds what each sequence's lanes have to its
    // word of `counts`. Returns how many counted.
    __device__ __forceinline__ uint32_t flush_row(unsigned long long* counts, const uint32_t i, const uint32_t lane)
    {
        constexpr uint32_t all = 0xFFFFFFFFu;
        if constexpr(mode_ == 2)
        {
            if(acc)
                atomicAdd(counts + i, acc);
            acc = 0;
            return 0;
        }
        else
        {
            const uint32_t left = __shfl_up_sync(all, i, 1), heads = __ballot_sync(all, lane == 0 || i != left);
            if(heads >> lane & 1)
            {
                const uint32_t from = all << lane, next = heads & (from << 1);
                const uint32_t n = __popc(ones & (next ? from & ((next & (0u - next)) - 1) : from));
                if(n)
                    atomicAdd(counts + i, static_cast<unsigned long long>(n));
            }
            cnt = 0;
            return __popc(ones);
        }
    }
    __device__ __forceinline__ void end_group_row(const Seg_Of& s, const uint32_t i, const uint32_t lane) { flush_row(out + s.q, i, lane); }
    __device__ __forceinline__ unsigned long long seg_total() const
    {
        if constexpr(mode_ != 2)
            return cnt;
        unsigned long long a = acc;
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
            a += __shfl_xor_sync(0xFFFFFFFFu, a, o);
        return a;
    }
    __device__ __forceinline__ void end_segment(const Seg_Of& s, const uint32_t lane)
    {
        const unsigned long long a = seg_total();
        if(lane == 0 && a)
            atomicAdd(out + s.q, a);
    }
    __device__ __forceinline__ void end(uint32_t) {}
};

// Counts of several batches run as one: per sequence in its own batch's array, and per batch at per_batch.
template <bool set_, typename V>
struct Count_Batches_Visitor : Seq_Reduce_Visitor<set_, V, 0>
{
    const uint64_t* outs;       // Per batch, 8 words: its first merged sequence at word 3, its counts' address at word 4.
    unsigned long long* per_batch;

    uint32_t grouped = 0;       // Found in the rows of the current group.

    __device__ __forceinline__ void end_group_row(const Seg_Of& s, const uint32_t i, const uint32_t lane)
    {
        const uint64_t* o = outs + 8 * uint64_t(s.batch);
        grouped += this->flush_row(reinterpret_cast<unsigned long long*>(o[4]) + (s.q - o[3]), i, lane);
    }
    __device__ __forceinline__ void end_segment(const Seg_Of& s, const uint32_t lane)
    {
        const unsigned long long a = this->seg_total(), n = a + grouped;
        grouped = 0;
        if(lane == 0 && n)
        {
            const uint64_t* o = outs + 8 * uint64_t(s.batch);
            if(a)
                atomicAdd(reinterpret_cast<unsigned long long*>(o[4]) + (s.q - o[3]), a);
            atomicAdd(per_batch + s.batch, n);
        }
    }
};

// The descriptions that callers can see, for checking the describer: the key's 2-bit encoding, and the reference's
// checksum and minimizer hash of it.
template <int k, int l>
struct Describe_Visitor
{
    static constexpr int min_blocks = 4;
    uint64_t* key;
    uint64_t* h;
    uint8_t* cs;
    uint8_t* fwd;
    uint8_t* valid;
    uint64_t obase = 0;

    __device__ __forceinline__ void begin() {}
    __device__ __forceinline__ void begin_segment(const Seg_Of& s) { obase = s.pos; }
    __device__ __forceinline__ void end_segment(const Seg_Of&, uint32_t) {}
    __device__ __forceinline__ void end(uint32_t) {}
    __device__ __forceinline__ void visit(const Kmer_Desc& d, const uint32_t)
    {
        if(!d.in)
            return;
        const uint64_t o = obase + d.pos, e = encoding_of(d.key);
        key[o] = d.valid ? e : 0, h[o] = d.valid ? described_minimizer<k, l>(e) : 0, cs[o] = d.valid ? described_checksum(e) : 0;
        fwd[o] = d.valid && d.fwd, valid[o] = d.valid;
    }
};

}
