// The table in HBM and its lock-free per-k-mer operations.
//
// Layout (structure of arrays, one entry per bucket of B = 32 slots):
//   cs[cap][32]     u8   checksums; 0 = empty. One 32-byte sector per bucket, so two 16-byte loads of it test all 32
//                        slots (slot j's is byte cs_byte(j)).
//   spill[cap][8]   u32  the 255-bit spill filter of minimizers whose keys left the (full) bucket
//                        (include/Streaming_Kmer_Hash_Table.hpp:91-97,1064-1093). Bit 0 is unused.
//   slots[cap][32]       maps: {u64 ~key, u64 value} (16 B; a key and its value share one sector);
//                        sets: {u64 ~key} (8 B). The key (its planes, device_common.cuh) is stored complemented, so
//                        zeroed memory is empty: no canonical k-mer is all T's, whose complement would be 0.
//   ov[ov_cap]           the overflow table: {u64 ~key, u64 value, u64 ready, u64 pad}, linear probing.
//
// Concurrency without locks, in place of the reference's bucket spin locks (include/Streaming_Kmer_Hash_Table.hpp:
// 1125-1212): an insert claims a slot by atomicCAS of its key word from 0. An inserter by itself tries a bucket's slots in
// order from the first empty checksum on; a run of lanes with one bucket tries neighbouring slots side by side, but as a
// whole every one from there on (warp_claim). So whoever claims a slot for a key, or meets another's claim of it, has tried
// all lower slots that were open, and the lowest slot that holds the key is the one that all settle on. A claim that a
// lower one of its key makes void stays as a hole: checksum 0, a key that no k-mer has. Holes are rare (two warps have to
// claim one new key in one bucket within the same few hundred nanoseconds) and last until a rebuild leaves them out; one
// costs its slot and, for each new key of its bucket, a swap that fails, also where the bucket is full. The last slot is
// never a hole and is claimed only by who has tried all others, so its checksum says that the bucket is full.
// The claimer then writes the value, fences, and publishes the checksum; a racing inserter of the same key
// that met the claim waits (boundedly) for that checksum before applying its update. (Where updates commute from a zeroed
// value nobody fences or waits, see Op_Fn::commutes.) Every inserter of a key scans the
// same chain -- primary bucket, then secondary p, then q, then the overflow table -- so a key has one copy. A full
// primary bucket gets its spill-filter bit set before any key of its minimizer goes beyond it, which keeps the
// reference's lookup rule: absent past a full primary bucket unless its filter marks the minimizer
// (include/Streaming_Kmer_Hash_Table.hpp:2555-2571).
#pragma once

#include "device_common.cuh"

namespace kache_b200
{

template <typename V> struct Val_Of { typedef V type; static constexpr bool is_set = false; };
template <> struct Val_Of<void> { typedef uint8_t type; static constexpr bool is_set = true; };

struct Dev_Table
{
    uint8_t* cs;
    uint32_t* spill;
    unsigned long long* slots;
    uint64_t cap;           // Buckets.
    unsigned long long* ov; // Overflow slots, 4 words each.
    uint64_t ov_mask;       // Overflow capacity - 1 (a power of 2).
    uint32_t ov_probe;      // Most slots an overflow probe visits.
    unsigned long long* ov_count;   // Keys in the overflow table.
    unsigned int* err;      // Nonzero after a bounded wait gave up.
    uint32_t wait_polls;    // Most polls of a wait for a racing insert's publication.
};

constexpr uint32_t default_wait_polls = 1u << 22;

constexpr uint32_t no_bucket = ~0u;     // No bucket's index: there are at most 2^32 - 1.
constexpr uint32_t ERR_WAIT = 1;    // A wait for a racing insert's publication ran out.

template <bool set_> __host__ __device__ constexpr int slot_words() { return set_ ? 1 : 2; }

// Loads that must see other SMs' writes within the same kernel bypass L1.
__device__ __forceinline__ unsigned long long ld_cg(const unsigned long long* p) { return __ldcg(p); }
__device__ __forceinline__ uint4 ld_cg4(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ uint8_t ld_volatile_u8(const uint8_t* p) { return *reinterpret_cast<const volatile uint8_t*>(p); }

// Atomics on the table's words that return nothing, as reductions: no lane waits for their results.
__device__ __forceinline__ void red_add(unsigned long long* p, const unsigned long long x) { asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "l"(x) : "memory"); }
__device__ __forceinline__ void red_add(unsigned int* p, const unsigned int x) { asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "r"(x) : "memory"); }
__device__ __forceinline__ void red_or(unsigned long long* p, const unsigned long long x) { asm volatile("red.relaxed.gpu.global.or.b64 [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "l"(x) : "memory"); }
__device__ __forceinline__ void red_or(unsigned int* p, const unsigned int x) { asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "r"(x) : "memory"); }
__device__ __forceinline__ void red_max(unsigned long long* p, const unsigned long long x) { asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "l"(x) : "memory"); }
__device__ __forceinline__ void red_max(unsigned int* p, const unsigned int x) { asm volatile("red.relaxed.gpu.global.max.u32 [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "r"(x) : "memory"); }
__device__ __forceinline__ void red_min(unsigned long long* p, const unsigned long long x) { asm volatile("red.relaxed.gpu.global.min.u64 [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "l"(x) : "memory"); }
__device__ __forceinline__ void red_min(unsigned int* p, const unsigned int x) { asm volatile("red.relaxed.gpu.global.min.u32 [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "r"(x) : "memory"); }

// Reads a stored value as V.
template <typename V>
__device__ __forceinline__ V read_val(const unsigned long long* w)
{
    if constexpr(sizeof(V) == 8)
        return static_cast<V>(*w);
    else
        return static_cast<V>(*reinterpret_cast<const uint32_t*>(w));
}

template <typename V>
__device__ __forceinline__ void write_val(unsigned long long* w, const V v)
{
    if constexpr(sizeof(V) == 8)
        *w = static_cast<unsigned long long>(v);
    else
        *reinterpret_cast<uint32_t*>(w) = static_cast<uint32_t>(v);
}

// Applies `f` to the value at `w` atomically: a compare-and-swap loop on the value's word (the low 32 bits for
// values of up to 4 bytes, whose upper bytes stay 0), as the reference updates values in place
// (include/Streaming_Kmer_Hash_Table.hpp:1239-1253).
template <typename V, typename F>
__device__ __forceinline__ void cas_update(unsigned long long* w, const F& f)
{
    if constexpr(sizeof(V) == 8)
    {
        unsigned long long old = __ldcg(w), assumed;
        do
        {
            assumed = old;
            old = atomicCAS(w, assumed, static_cast<unsigned long long>(f(static_cast<V>(assumed))));
        } while(old != assumed);
    }
    else
    {
        unsigned int* p = reinterpret_cast<unsigned int*>(w);
        unsigned int old = __ldcg(p), assumed;
        do
        {
            assumed = old;
            old = atomicCAS(p, assumed, static_cast<unsigned int>(f(static_cast<V>(assumed))));
        } while(old != assumed);
    }
}

// The closed set of value operations of the C interface (capi/Kmer_Table.hpp:30-43), with a wrapping add for the
// template API's `v + x`: `f(v)` for a present key, `x` for an absent one. Atomic fast paths where one
// instruction does the operation exactly.
template <typename V>
struct Op_Fn
{
    uint32_t op;
    V x;
    V init;

    __device__ __forceinline__ V operator()(const V v) const
    {
        constexpr V mx = static_cast<V>(~V(0));
        switch(op)
        {
        case OP_KEEP: return v;
        case OP_ASSIGN: return x;
        case OP_ADD: return v > static_cast<V>(mx - x) ? mx : static_cast<V>(v + x);
        case OP_OR: return static_cast<V>(v | x);
        case OP_MIN: return v < x ? v : x;
        case OP_ADD_WRAP: return static_cast<V>(v + x);
        default: return v > x ? v : x;
        }
    }

    __device__ __forceinline__ V initial(bool) const { return init; }
    __device__ __forceinline__ bool is_noop() const { return op == OP_KEEP; }

    // Whether every update of a key combines with the others in any order, starting from a zeroed value: then an
    // inserter folds its initial value in atomically (op(0, init) = init for these ops) and nobody waits for it.
    __device__ __forceinline__ bool commutes() const
    {
        return op == OP_KEEP || op == OP_ADD || op == OP_ADD_WRAP || op == OP_OR || op == OP_MAX;
    }

    // For operations that commute: an occurrence's update, the key's first one giving it its initial value.
    __device__ __forceinline__ void apply_or_init(unsigned long long* w, bool, const bool first) const
    {
        if(op != OP_KEEP)
            Op_Fn<V>{op, first ? init : x, init}.apply(w, true);
        else if(first)
            write_val<V>(w, init);
    }

    __device__ __forceinline__ void apply(unsigned long long* w, bool) const
    {
        if(op == OP_KEEP)
            return;
        constexpr V mx = static_cast<V>(~V(0));
        if constexpr(sizeof(V) == 8)
        {
            switch(op)
            {
            case OP_ADD:
                // Saturating add as an atomic add, then the saturated value wherever an add carried past the maximum:
                // every add that overflows sees it (old > max - x) and stores the maximum after its own add, and an
                // add landing on a value an overflow left small either overflows in turn or is overwritten by that
                // fix-up, so the word ends at min(max, v + sum x) as the serial order would leave it. Nothing reads
                // values while inserts run.
                if(atomicAdd(w, static_cast<unsigned long long>(x)) > static_cast<unsigned long long>(mx - x))
                    atomicExch(w, static_cast<unsigned long long>(mx));
                return;
            case OP_ASSIGN: atomicExch(w, static_cast<unsigned long long>(x)); return;
            case OP_OR: red_or(w, static_cast<unsigned long long>(x)); return;
            case OP_MIN: red_min(w, static_cast<unsigned long long>(x)); return;
            case OP_MAX: red_max(w, static_cast<unsigned long long>(x)); return;
            case OP_ADD_WRAP: red_add(w, static_cast<unsigned long long>(x)); return;
            default: break;
            }
        }
        else
        {
            unsigned int* p = reinterpret_cast<unsigned int*>(w);
            switch(op)
            {
            case OP_ADD:    // As above, on the value's 32-bit word (values of 1 or 2 bytes saturate below its top).
                if(atomicAdd(p, static_cast<unsigned int>(x)) > static_cast<unsigned int>(mx - x))
                    atomicExch(p, static_cast<unsigned int>(mx));
                return;
            case OP_ASSIGN: atomicExch(p, static_cast<unsigned int>(x)); return;
            case OP_OR: red_or(p, static_cast<unsigned int>(x)); return;
            case OP_MIN: red_min(p, static_cast<unsigned int>(x)); return;
            case OP_MAX: red_max(p, static_cast<unsigned int>(x)); return;
            case OP_ADD_WRAP:
                // A value of 1 or 2 bytes is the low part of its word, which the words' adds keep right by themselves; an
                // add that carries out of it takes the carry off again, so the part above ends at 0. (A compare-and-swap
                // loop took 1.16 ms for 12M updates of 20,000 keys, this 0.22.)
                if constexpr(sizeof(V) == 4)
                    red_add(p, static_cast<unsigned int>(x));
                else if((atomicAdd(p, static_cast<unsigned int>(x)) & mx) + x > mx)
                    red_add(p, 0u - (1u << (8 * sizeof(V))));
                return;
            default: break;
            }
        }
        cas_update<V>(w, *this);
    }
};

// The oriented operations (capi/Kmer_Table.hpp:50-61): operand x_fwd for an occurrence as the canonical form,
// x_rev for one as its reverse complement; an absent key gets f(0, fwd) (include/Streaming_Kmer_Hash_Table.hpp:682).
template <typename V>
struct Oriented_Op_Fn
{
    uint32_t op;
    V x_fwd, x_rev;

    __device__ __forceinline__ Op_Fn<V> at(const bool fwd) const { return Op_Fn<V>{op, fwd ? x_fwd : x_rev, V(0)}; }
    __device__ __forceinline__ V initial(const bool fwd) const { return at(fwd)(V(0)); }
    __device__ __forceinline__ bool is_noop() const { return false; }
    __device__ __forceinline__ bool commutes() const { return op == OP_ADD || op == OP_ADD_WRAP || op == OP_OR || op == OP_MAX; }
    __device__ __forceinline__ void apply_or_init(unsigned long long* w, const bool fwd, bool) const { at(fwd).apply(w, fwd); }
    __device__ __forceinline__ void apply(unsigned long long* w, const bool fwd) const { at(fwd).apply(w, fwd); }
};

// Adapts a user's device functor `f(v)` with the value `val` for absent keys (the C++ template API's upsert).
template <typename V, typename F>
struct User_Fn
{
    F f;
    V val;
    __device__ __forceinline__ V initial(bool) const { return val; }
    __device__ __forceinline__ bool is_noop() const { return false; }
    __device__ __forceinline__ bool commutes() const { return false; }
    __device__ __forceinline__ void apply_or_init(unsigned long long* w, bool, bool) const { cas_update<V>(w, f); }
    __device__ __forceinline__ void apply(unsigned long long* w, bool) const { cas_update<V>(w, f); }
};

// Adapts a user's device functor `f(v, fwd)` (the C++ template API's upsert_oriented): absent keys get f(V(), fwd).
template <typename V, typename F>
struct User_Oriented_Fn
{
    F f;
    __device__ __forceinline__ V initial(const bool fwd) const { return f(V(), fwd); }
    __device__ __forceinline__ bool is_noop() const { return false; }
    __device__ __forceinline__ bool commutes() const { return false; }
    __device__ __forceinline__ void apply_or_init(unsigned long long* w, const bool fwd, bool) const { apply(w, fwd); }
    __device__ __forceinline__ void apply(unsigned long long* w, const bool fwd) const
    {
        const F& g = f;
        cas_update<V>(w, [&](const V v){ return g(v, fwd); });
    }
};

// Outcome of one k-mer's upsert chain.
enum Outcome : uint32_t
{
    NONE = 0,
    INSERTED = 1,       // This lane claimed the slot; it still writes the value and publishes.
    FOUND = 2,          // Present and published: apply the update.
    FOUND_PENDING = 3,  // Present, claimed by a racing lane that has yet to publish: wait, then apply.
    OV_FULL = 4         // The overflow table had no room within its probe bound: retry after it grows.
};

template <bool set_>
__device__ __forceinline__ unsigned long long* key_word(const Dev_Table& T, const uint64_t b, const uint32_t j)
{
    return T.slots + (b * B + j) * slot_words<set_>();
}

// A bucket's checksums: words 0..3 and 4..7.
struct Checksums
{
    uint4 lo, hi;

    __device__ __forceinline__ bool full() const { return (hi.w >> 24) != 0; }  // The last slot is claimed after all others.
    // The first slot whose checksum is empty, or B. (The inexact test can flag a byte above an empty one of its word,
    // which is a higher slot.)
    __device__ __forceinline__ uint32_t first_empty() const
    {
        const uint32_t m = candidates32<false>(lo, hi, 0);
        return m ? __ffs(m) - 1 : B;
    }
};

template <bool cg_>
__device__ __forceinline__ Checksums bucket_cs(const Dev_Table& T, const uint32_t b)
{
    const uint8_t* p = T.cs + uint64_t(b) * B;
    if constexpr(cg_)
        return Checksums{ld_cg4(p), ld_cg4(p + 16)};
    else
        return Checksums{*reinterpret_cast<const uint4*>(p), *reinterpret_cast<const uint4*>(p + 16)};
}

__device__ __forceinline__ uint8_t* cs_of(const Dev_Table& T, const uint32_t b, const uint32_t j) { return T.cs + uint64_t(b) * B + cs_byte(j); }

// Looks for the key among the published slots of bucket b. Returns FOUND with its slot at `j`, or NONE with the first
// slot whose checksum is empty at `j` (B if there is none).
template <bool set_>
__device__ __forceinline__ uint32_t bucket_probe(const Dev_Table& T, const uint32_t b, const unsigned long long key_st, const uint32_t c, uint32_t& j)
{
    const Checksums s = bucket_cs<true>(T, b);
    uint32_t r = NONE;
    j = s.first_empty();
    for(uint32_t cand = candidates32<true>(s.lo, s.hi, c); cand != 0 && r == NONE; cand &= cand - 1)
        if(ld_cg(key_word<set_>(T, b, __ffs(cand) - 1)) == key_st)
            r = FOUND, j = __ffs(cand) - 1;
    return r;
}

// Tries the bucket b for the key, one lane by itself: its published candidates, then the claim scan. Returns FOUND,
// FOUND_PENDING (claimed by another lane, published or not) or INSERTED with the slot at `j`, or NONE if the bucket is full
// without the key.
template <bool set_>
__device__ __forceinline__ uint32_t bucket_upsert(const Dev_Table& T, const uint32_t b, const unsigned long long key_st, const uint32_t c, uint32_t& j)
{
    uint32_t r = bucket_probe<set_>(T, b, key_st, c, j);
    // The claim scan: a compare-and-swap straight away (a slot with an empty checksum is most likely unclaimed), whose
    // result, if it fails, is the racing claimer's key.
    while(r == NONE && j < B)
    {
        const unsigned long long cur = atomicCAS(key_word<set_>(T, b, j), 0ull, key_st);
        if(cur == 0)
            r = INSERTED;
        else if(cur == key_st)
            r = FOUND_PENDING;
        else
            ++j;
    }
    return r;
}

// Tries the overflow table. Returns FOUND_PENDING or INSERTED with the slot index at `i_out`, or OV_FULL.
__device__ __forceinline__ uint32_t overflow_upsert(const Dev_Table& T, const unsigned long long key_st, uint64_t& i_out)
{
    uint64_t i = ov_hash(key_st) & T.ov_mask;
    uint32_t r = OV_FULL;
    for(uint32_t t = 0; r == OV_FULL && t < T.ov_probe; ++t, i = (i + 1) & T.ov_mask)
    {
        unsigned long long* kw = T.ov + 4 * i;
        unsigned long long cur = ld_cg(kw);
        if(cur == 0)
        {
            cur = atomicCAS(kw, 0ull, key_st);
            if(cur == 0)
                r = INSERTED, i_out = i;
        }
        if(cur == key_st)
            r = FOUND_PENDING, i_out = i;
    }
    return r;
}

// Where an upsert chain ended: a value word and the flag that publishes it (a checksum byte, or an overflow slot's
// ready word).
struct Landing
{
    unsigned long long* val;
    uint8_t* cs;            // Non-null in the main table.
    unsigned long long* ready;  // Non-null in the overflow table.
    uint32_t c;
};

// The upsert chain of one k-mer (include/Streaming_Kmer_Hash_Table.hpp:2431-2490, lock-free): primary bucket; if
// full, mark its spill filter, then the secondary buckets in order; then the overflow table.
template <bool set_>
__device__ __forceinline__ uint32_t upsert_chain(const Dev_Table& T, const uint64_t key, const uint32_t h, const uint32_t c, Landing& L)
{
    const unsigned long long key_st = ~key;
    uint32_t j;
    const uint32_t b = bucket_of(h, T.cap);
    uint32_t r = bucket_upsert<set_>(T, b, key_st, c, j);
    uint32_t at = b;
    if(r == NONE)
    {
        const uint32_t fp = filter_pos(h);
        uint32_t* sw = T.spill + uint64_t(b) * 8 + (fp >> 5);
        const uint32_t bit = 1u << (fp & 31);
        if(!(__ldcg(sw) & bit))
            atomicOr(sw, bit);

        at = second_bucket(h, T.cap);
        r = bucket_upsert<set_>(T, at, key_st, c, j);
        if(r == NONE)
            at = third_bucket(h, T.cap), r = bucket_upsert<set_>(T, at, key_st, c, j);
    }

    if(r != NONE)
    {
        unsigned long long* kw = key_word<set_>(T, at, j);
        L.val = set_ ? nullptr : kw + 1, L.cs = cs_of(T, at, j), L.ready = nullptr, L.c = c;
        return r;
    }

    uint64_t i;
    r = overflow_upsert(T, key_st, i);
    L.val = T.ov + 4 * i + 1, L.cs = nullptr, L.ready = T.ov + 4 * i + 2, L.c = c;
    return r;
}

// The upsert chain of the lanes of a whole warp that `want` it (no two with the same key). On entry `at` is a lane's
// primary bucket (no_bucket in lanes without a k-mer). On return r is as upsert_chain's, with the slot at (at, j), or with
// at = no_bucket at overflow slot `ov_i`. All stages of the chain go through one loop, with one probe and one swap in it:
// the kernel's code is large enough that its size costs time (unrolled twice, 40M upserts took 1.28 ms against 1.04).
//
// The lanes hold consecutive k-mers, so the new ones come in runs of neighbours that share a minimizer, hence a bucket.
// A run claims together: its lane of rank i tries slot j + i at once with the others, where lanes trying the same slot
// one after another would take as many rounds of compare-and-swaps as the run has keys. What keeps one copy of each key
// is that a run as a whole tries every slot from the first empty one on, as a single inserter would: a lane whose key a
// failed swap of its run shows in a lower slot takes that slot, and leaves a slot that it has itself claimed higher up
// as a hole: unpublished for good (its checksum stays 0, so nothing iterates it), its key replaced by one that no k-mer
// has (so no lookup takes it for a candidate, and inserters pass it by as another key's claim). The lowest slot that
// holds a key is the one that everybody settles on, since an inserter either finds it published when it first probes the
// bucket, or its run tries that slot. A hole is never the last slot, which marks a bucket full: only a lane of rank 0,
// whose claim is the lowest tried, takes that one.
constexpr unsigned long long hole_key = 1;  // ~key of T...TG, whose reverse complement CA...A is the lesser.

template <bool set_>
__device__ __forceinline__ void warp_claim(const Dev_Table& T, const unsigned long long key_st, const uint32_t h, const uint32_t c, const uint32_t lane,
                                           const bool want, uint32_t& at, uint32_t& j, uint32_t& r, uint64_t& ov_i)
{
    constexpr uint32_t all = 0xFFFFFFFFu;
    const uint32_t le = all >> (31 - lane), lt = le >> 1;
    uint32_t stage = 0;         // 0: the primary bucket; 1 and 2: the secondary ones.
    bool probe = want;
    for(;;)
    {
        if(probe)
            r = bucket_probe<set_>(T, at, key_st, c, j);
        const bool open = want && r == NONE, in = open && j < B;
        if(!__any_sync(all, open))
            return;
        probe = open && !in && stage < 2;
        if(probe)
        {
            // A full bucket: a primary one's spill filter is marked before the key goes beyond it.
            if(stage == 0)
            {
                const uint32_t fp = filter_pos(h);
                uint32_t* sw = T.spill + uint64_t(at) * 8 + (fp >> 5);
                const uint32_t bit = 1u << (fp & 31);
                if(!(__ldcg(sw) & bit))
                    atomicOr(sw, bit);
            }
            at = stage == 0 ? second_bucket(h, T.cap) : third_bucket(h, T.cap);
            ++stage;
        }
        else if(open && !in)
        {
            at = no_bucket;
            r = overflow_upsert(T, key_st, ov_i);
        }

        const uint32_t in_m = __ballot_sync(all, in);
        if(in_m == 0)
            continue;
        // This lane's run: the lanes from the last change of bucket on, up to the next.
        const uint32_t left = __shfl_up_sync(all, at, 1);
        const uint32_t heads = __ballot_sync(all, lane == 0 || at != left);
        const uint32_t from = all << (31 - __clz(heads & le)), next = heads & ~le;
        const uint32_t run = next ? from & ((next & (0u - next)) - 1) : from;
        // Lanes of a run whose probes saw different first empty slots do not claim together: those unlike the first
        // probe afresh.
        const uint32_t first = __shfl_sync(all, j, in ? __ffs(in_m & run) - 1 : lane);
        const bool ok = in && j == first;
        const uint32_t ok_run = __ballot_sync(all, ok) & run;
        const uint32_t rank = __popc(ok_run & lt), slot = j + rank;
        const bool tries = ok && (rank == 0 || slot < B - 1);
        unsigned long long cur = 0;
        uint32_t got = slot;
        if(tries)
        {
            cur = atomicCAS(key_word<set_>(T, at, slot), 0ull, key_st);
            if(cur == 0)
                r = INSERTED;
            else if(cur == key_st)
                r = FOUND_PENDING;
        }
        const uint32_t tried = __popc(__ballot_sync(all, tries) & run);
        // Where a swap lost, its run's lanes compare their keys with what it showed: every run at once, lane by lane
        // from its first.
        const uint32_t lost = __ballot_sync(all, tries && r == NONE);
        if(lost)
            for(uint32_t left_m = run & lost; __any_sync(all, left_m); left_m &= left_m - 1)
            {
                const uint32_t s = left_m ? __ffs(left_m) - 1 : lane;
                const unsigned long long k_s = __shfl_sync(all, cur, s);
                const uint32_t slot_s = __shfl_sync(all, slot, s);
                if(ok && left_m && k_s == key_st && (r == NONE || slot_s < got))
                {
                    if(r == INSERTED)
                        *reinterpret_cast<volatile unsigned long long*>(key_word<set_>(T, at, got)) = hole_key;
                    r = FOUND_PENDING, got = slot_s;
                }
            }
        if(ok)
            j = r == NONE ? j + tried : got;
        probe = probe || (in && !ok);
    }
}

// Publishes a claimed slot whose value nobody waits for.
__device__ __forceinline__ void publish(const Landing& L)
{
    if(L.cs)
        *reinterpret_cast<volatile uint8_t*>(L.cs) = static_cast<uint8_t>(L.c);
    else
        *reinterpret_cast<volatile unsigned long long*>(L.ready) = 1ull;
}

// Waits, boundedly (`polls` polls), for a racing insert of the same key to publish. Returns false if the wait ran out.
__device__ __forceinline__ bool await_published(const Landing& L, const uint32_t polls)
{
    bool done = false;
    for(uint32_t t = 0; !done && t < polls; ++t)
    {
        done = L.cs ? ld_volatile_u8(L.cs) != 0 : *reinterpret_cast<const volatile unsigned long long*>(L.ready) != 0;
        if(!done && t > 64)
            __nanosleep(64);
    }
    __threadfence();
    return done;
}

// The key and value of a map's slot at kw (16-byte aligned), in one load.
template <bool cg_>
__device__ __forceinline__ void load_slot(const unsigned long long* kw, unsigned long long& k, unsigned long long& v)
{
    const ulonglong2 s = cg_ ? __ldcg(reinterpret_cast<const ulonglong2*>(kw)) : *reinterpret_cast<const ulonglong2*>(kw);
    k = s.x, v = s.y;
}

// Compares the key of the slot at kw with key_st (a stored, complemented key), keeping a map's value in `val`.
template <bool set_, bool cg_>
__device__ __forceinline__ bool slot_is(const unsigned long long* kw, const unsigned long long key_st, unsigned long long& val)
{
    unsigned long long k;
    if constexpr(set_)
        k = cg_ ? ld_cg(kw) : *kw;
    else
        load_slot<cg_>(kw, k, val);
    return k == key_st;
}

// Looks for the key, which the first probe of its primary bucket did not find, among the candidates `cand` left there and
// then, if that bucket is full, past it: absent unless its spill filter marks the minimizer; else the secondary buckets;
// then the overflow table iff both are full (include/Streaming_Kmer_Hash_Table.hpp:2548-2574). On entry `at` is the primary
// bucket; if the key is found, its slot is `slot` of bucket `at`, or with at = no_bucket of the overflow table, and with
// val_ a map's value goes to `val`. (This and the other chains here leave their loops in one place each: with returns out
// of nested loops, lanes of a warp went on apart past the end of the chain, and the votes behind it missed them.)
template <bool set_, bool cg_, bool val_>
__device__ __forceinline__ bool find_on(const Dev_Table& T, uint32_t& at, uint64_t& slot, uint32_t cand, const bool full, const unsigned long long key_st,
                                        const uint32_t h, unsigned long long& val)
{
    const uint32_t c = checksum_of(~key_st);
    bool hit = false, both_full = true, on;
    uint32_t t = 0;     // 0: the primary bucket; 1 and 2: the secondary ones.
    do
    {
        while(cand != 0 && !hit)
        {
            slot = __ffs(cand) - 1;
            cand &= cand - 1;
            const unsigned long long* kw = key_word<set_>(T, at, static_cast<uint32_t>(slot));
            if constexpr(val_ && !set_)
                hit = slot_is<set_, cg_>(kw, key_st, val);
            else
                hit = (cg_ ? ld_cg(kw) : *kw) == key_st;
        }
        on = !hit && full && t < 2;
        if(on && t == 0)
        {
            const uint32_t fp = filter_pos(h);
            const uint32_t* sw = T.spill + uint64_t(at) * 8 + (fp >> 5);
            on = ((cg_ ? __ldcg(sw) : *sw) >> (fp & 31)) & 1;
        }
        if(on)
        {
            at = ++t == 1 ? second_bucket(h, T.cap) : third_bucket(h, T.cap);
            const Checksums s = bucket_cs<cg_>(T, at);
            cand = candidates32<false>(s.lo, s.hi, c);
            both_full = both_full && s.full();
        }
    } while(on);
    on = !hit && t == 2 && both_full;
    if(on)
    {
        at = no_bucket;
        slot = ov_hash(key_st) & T.ov_mask;
        for(uint32_t n = 0; on && n < T.ov_probe; ++n)
        {
            unsigned long long k, v;
            load_slot<cg_>(T.ov + 4 * slot, k, v);
            hit = k == key_st;
            on = !hit && k != 0;
            if constexpr(val_)
                val = v;
            slot = on ? (slot + 1) & T.ov_mask : slot;
        }
    }
    return hit;
}

// The value word (the key word of a set) of slot j of bucket `at`, or with at = no_bucket of the overflow table.
template <bool set_>
__device__ __forceinline__ unsigned long long* value_word(const Dev_Table& T, const uint32_t at, const uint64_t j)
{
    return at == no_bucket ? T.ov + 4 * j + 1 : key_word<set_>(T, at, static_cast<uint32_t>(j)) + (set_ ? 0 : 1);
}

// Finds a key, one lane by itself: its value word (the key word of a set), or null.
template <bool set_, bool cg_>
__device__ __forceinline__ unsigned long long* find_chain(const Dev_Table& T, const uint64_t key, const uint32_t h, const uint32_t c)
{
    uint32_t at = bucket_of(h, T.cap);
    uint64_t j = 0;
    const Checksums s = bucket_cs<cg_>(T, at);
    unsigned long long val;
    const bool hit = find_on<set_, cg_, false>(T, at, j, candidates32<false>(s.lo, s.hi, c), s.full(), ~key, h, val);
    return hit ? value_word<set_>(T, at, j) : nullptr;
}

// The first probe of a lane's k-mer, in its primary bucket.
struct Probe
{
    uint32_t slot;      // The key's slot there, B if it was not found.
    uint32_t rest;      // Candidate slots not tried.
    bool full;          // Whether the bucket is full.
    unsigned long long val;     // With val_, the value in a map of the key found.
};

// Probes the primary bucket of the k-mer `key` of minimizer hash h where `valid`. The first two candidates are read
// together: one lane in fourteen or so has a candidate besides its key, so most warps have some, and a warp waits for a
// second read as long as for the first.
template <bool set_, bool cg_, bool val_>
__device__ __forceinline__ Probe probe_primary(const Dev_Table& T, const bool valid, const uint64_t key, const uint32_t h)
{
    const unsigned long long key_st = ~key;
    const uint32_t b = bucket_of(h, T.cap);
    uint32_t cand = 0;
    Probe p{B, 0, false, 0};
    if(valid)
    {
        const Checksums s = bucket_cs<cg_>(T, b);
        // Exactly where inserts run (cg_): a slot claimed but not yet published is no candidate.
        cand = candidates32<cg_>(s.lo, s.hi, checksum_of(key));
        p.full = s.full();
    }
    const uint32_t j1 = top_bit(cand), more = cand & ~(1u << (j1 & 31)), j2 = top_bit(more);
    unsigned long long k1, v1, k2, v2;
    const auto read = [&](const uint32_t j, unsigned long long& k, unsigned long long& v)
    {
        const unsigned long long* kw = key_word<set_>(T, b, j);
        if constexpr(val_ && !set_)
            load_slot<cg_>(kw, k, v);
        else
            k = cg_ ? ld_cg(kw) : *kw;
    };
    if(cand)
        read(j1, k1, v1);
    if(more)
        read(j2, k2, v2);
    if(cand && k1 == key_st)
        p.slot = j1;
    if constexpr(val_ && !set_)
        p.val = v1;
    if(more && k2 == key_st)
    {
        p.slot = j2;
        if constexpr(val_ && !set_)
            p.val = v2;
    }
    p.rest = more & ~(1u << (j2 & 31));
    return p;
}

// For failure-injection tests: claims a slot of the key's primary bucket for it, as a racing inserter would, and
// leaves it unpublished (its checksum stays 0), so that a later inserter of the key that must see its value first
// waits on it. One thread; *ok is set to 1 if a slot was claimed.
template <int k, int l, bool set_>
__global__ void plant_claim_kernel(const Dev_Table T, const uint64_t key, unsigned long long* ok)
{
    const uint64_t b = bucket_of(minimizer_hash<k, l>(key), T.cap);
    const uint32_t j = bucket_cs<false>(T, static_cast<uint32_t>(b)).first_empty();
    *ok = 0;
    if(j == B)
        return;
    unsigned long long* kw = key_word<set_>(T, b, j);
    *ok = atomicCAS(kw, 0ull, ~key) == 0ull;
}

// The value of a found key, as read with it.
template <typename V>
__device__ __forceinline__ V value_of(const unsigned long long w)
{
    if constexpr(sizeof(V) == 8)
        return static_cast<V>(w);
    else
        return static_cast<V>(static_cast<uint32_t>(w));
}

}
