// The table-wide kernels: resize (rehash into a doubled table), overflow growth, iteration (for_each), reductions,
// histograms, placement statistics, single-k-mer lookups, and the device-side batch preparation.
#pragma once

#include "device_table.cuh"
#include "device_stream.cuh"

namespace kache_b200
{

// Inserts one key with its value, known absent (every key of a table is distinct), into `T`. Returns INSERTED or
// OV_FULL. No other thread inserts the same key, so none waits for the value: no fence before publishing.
template <bool set_>
__device__ __forceinline__ uint32_t place_key(const Dev_Table& T, const uint64_t key, const uint32_t h, const unsigned long long val)
{
    Landing L{};
    const uint32_t r = upsert_chain<set_>(T, key, h, checksum_of(key), L);
    if(r == INSERTED)
    {
        if constexpr(!set_)
            *L.val = val;
        publish(L);
        if(!L.cs)
            atomicAdd(T.ov_count, 1ull);
    }
    return r;
}

// Resize, second phase: the old slots marked in `marks` (keys not at their primary bucket, and the overflow table's
// slots) go through the insertion chain of the new table. A warp takes 32 words of marks (1024 slots), lists their set
// bits in shared memory, and then works through the list a slot per lane, so that lanes stay busy however sparse the
// marks are. Keys that find the new overflow table full set their bit in `retry_out`.
template <int k, int l, bool set_>
__global__ void __launch_bounds__(256) rest_kernel(const Dev_Table from, const Dev_Table to, const unsigned int* marks, const uint64_t total,
                                                   unsigned int* retry_out, unsigned int* retried)
{
    __shared__ uint16_t list_all[8][1024];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint16_t* list = list_all[wid];
    const uint64_t main_slots = from.cap * B, words = (total + 31) / 32;
    const uint64_t warps = uint64_t(gridDim.x) * 8;
    for(uint64_t wb = uint64_t(blockIdx.x) * 8 + wid; wb * 32 < words; wb += warps)
    {
        const uint64_t wi = wb * 32 + lane;
        uint32_t word = wi < words ? marks[wi] : 0u;
        if(wi * 32 + 32 > total && wi < words)
            word &= (total - wi * 32) >= 32 ? ~0u : ((1u << (total - wi * 32)) - 1);
        const uint32_t cnt = __popc(word);
        uint32_t pre = cnt;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, pre, o);
            if(lane >= static_cast<uint32_t>(o))
                pre += y;
        }
        const uint32_t n = __shfl_sync(0xFFFFFFFFu, pre, 31);
        pre -= cnt;
        for(uint32_t w = word, i = pre; w; w &= w - 1, ++i)
            list[i] = static_cast<uint16_t>(lane * 32 + __ffs(w) - 1);
        __syncwarp();
        for(uint32_t r = lane; r < n; r += 32)
        {
            const uint64_t s = wb * 1024 + list[r];
            unsigned long long key_st, val = 0;
            if(s < main_slots)
            {
                key_st = from.slots[s * slot_words<set_>()];
                if constexpr(!set_)
                    val = from.slots[s * 2 + 1];
            }
            else
            {
                const uint64_t i = s - main_slots;
                key_st = from.ov[4 * i];
                val = from.ov[4 * i + 1];
            }
            if(key_st == 0)
                continue;
            const uint64_t key = ~key_st;
            if(place_key<set_>(to, key, minimizer_hash<k, l>(key), val) == OV_FULL)
            {
                atomicOr(retry_out + (s >> 5), 1u << (s & 31));
                *retried = 1;
            }
        }
        __syncwarp();
    }
}

// Resize, first phase (include/Streaming_Kmer_Hash_Table.hpp:1494-1570, out of place): a warp per old bucket b.
// The keys whose primary bucket is b move to their primary bucket in the new table, one of the 2^d buckets
// [b * 2^d, (b + 1) * 2^d) when the capacity grows 2^d-fold, since bucket_of is monotone in the capacity; the warp
// writes each of those buckets whole (checksums, keys, values, a cleared spill filter), so the new arrays need no
// clearing. Keys held in b as a secondary bucket get their bit set in `rest`, for the second phase (rest_kernel).
template <int k, int l, bool set_>
__global__ void __launch_bounds__(256) split_kernel(const Dev_Table from, const Dev_Table to, const uint32_t d, unsigned int* rest)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = uint64_t(gridDim.x) * (blockDim.x / 32);
    for(uint64_t b = uint64_t(blockIdx.x) * (blockDim.x / 32) + (threadIdx.x >> 5); b < from.cap; b += warps)
    {
        const uint64_t s = b * B + lane;
        const uint8_t c = *cs_of(from, static_cast<uint32_t>(b), lane);
        unsigned long long key_st = 0, val = 0;
        uint32_t dest = 0xFFFFFFFFu;
        if(c)
        {
            key_st = from.slots[s * slot_words<set_>()];
            if constexpr(!set_)
                val = from.slots[s * 2 + 1];
            const uint32_t h = minimizer_hash<k, l>(~key_st);
            if(bucket_of(h, from.cap) == b)
                dest = bucket_of(h, to.cap) - static_cast<uint32_t>(b << d);
        }
        const uint32_t other = __ballot_sync(0xFFFFFFFFu, c != 0 && dest == 0xFFFFFFFFu);
        if(lane == 0 && other)
            rest[s >> 5] = other;   // s >> 5 == b: one word per old bucket.
        for(uint32_t t = 0; t < (1u << d); ++t)
        {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, dest == t);
            const uint64_t nb = (b << d) + t;
            // Lane j writes slot j of the new bucket: the rank-j key moving there, or an empty slot.
            const uint32_t n = __popc(m);
            const uint32_t src = lane < n ? __fns(m, 0, static_cast<int>(lane) + 1) : 0;
            const unsigned long long k_j = __shfl_sync(0xFFFFFFFFu, key_st, src);
            const unsigned long long v_j = __shfl_sync(0xFFFFFFFFu, val, src);
            const uint32_t c_j = __shfl_sync(0xFFFFFFFFu, static_cast<uint32_t>(c), src);
            const uint64_t ns = nb * B + lane;
            to.slots[ns * slot_words<set_>()] = lane < n ? k_j : 0ull;
            if constexpr(!set_)
                to.slots[ns * 2 + 1] = lane < n ? v_j : 0ull;
            *cs_of(to, static_cast<uint32_t>(nb), lane) = lane < n ? static_cast<uint8_t>(c_j) : 0;
            if(lane < 8)
                to.spill[nb * 8 + lane] = 0;
        }
    }
}

// Doubles the overflow table: re-inserts its keys into `to`'s overflow table, which has nothing else.
static __global__ void __launch_bounds__(256) ov_move_kernel(const unsigned long long* from, const uint64_t from_slots, const Dev_Table to)
{
    for(uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < from_slots; i += uint64_t(gridDim.x) * blockDim.x)
    {
        const unsigned long long key_st = from[4 * i];
        if(key_st == 0)
            continue;
        // The target has twice the slots, so a free one lies within its capacity.
        uint64_t j = ov_hash(key_st) & to.ov_mask;
        for(uint64_t t = 0; t <= to.ov_mask; ++t, j = (j + 1) & to.ov_mask)
            if(atomicCAS(to.ov + 4 * j, 0ull, key_st) == 0ull)
            {
                to.ov[4 * j + 1] = from[4 * i + 1];
                to.ov[4 * j + 2] = 1;
                break;
            }
    }
}

// Collects the keys (as their 2-bit encodings) and values of buckets [b_b, b_e) and overflow slots [o_b, o_e), in
// no particular order (include/Streaming_Kmer_Hash_Table.hpp:2705-2725): a warp claims its output range with one
// atomic.
template <bool set_>
__global__ void __launch_bounds__(256) collect_kernel(const Dev_Table T, const uint64_t b_b, const uint64_t b_e, const uint64_t o_b, const uint64_t o_e,
                                                      uint64_t* keys, uint64_t* vals, unsigned long long* count)
{
    const uint64_t n_main = (b_e - b_b) * B, total = n_main + (o_e - o_b);
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for(uint64_t s0 = uint64_t(blockIdx.x) * blockDim.x; s0 < total; s0 += stride)
    {
        const uint64_t s = s0 + threadIdx.x;
        bool have = false;
        unsigned long long key_st = 0, val = 0;
        if(s < n_main)
        {
            const uint64_t slot = b_b * B + s;
            if(*cs_of(T, static_cast<uint32_t>(slot / B), slot % B))
            {
                have = true;
                key_st = T.slots[slot * slot_words<set_>()];
                if constexpr(!set_)
                    val = T.slots[slot * 2 + 1];
            }
        }
        else if(s < total)
        {
            const uint64_t i = o_b + (s - n_main);
            key_st = T.ov[4 * i];
            if(key_st)
                have = true, val = T.ov[4 * i + 1];
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, have);
        unsigned long long base = 0;
        if(lane == 0 && m)
            base = atomicAdd(count, static_cast<unsigned long long>(__popc(m)));
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if(have)
        {
            const uint64_t o = base + __popc(m & ((1u << lane) - 1));
            keys[o] = encoding_of(~key_st);
            if(vals)
                vals[o] = val;
        }
    }
}

// The value of slot s of the table, its main slots first and then the overflow table's, if it holds a key.
template <bool set_>
__device__ __forceinline__ bool slot_value(const Dev_Table& T, const uint64_t s, unsigned long long& raw)
{
    const uint64_t n_main = T.cap * B;
    if(s < n_main)
    {
        // A set has no values, so its checksums can be taken in the order they lie in.
        if((set_ ? T.cs[s] : *cs_of(T, static_cast<uint32_t>(s / B), s % B)) == 0)
            return false;
        if constexpr(!set_)
            raw = T.slots[s * 2 + 1];
        return true;
    }
    const uint64_t i = s - n_main;
    if(T.ov[4 * i] == 0)
        return false;
    raw = T.ov[4 * i + 1];
    return true;
}

// Reductions of the C interface over all keys (capi/Kmer_Table.hpp:203-230): 0 keys with v & m nonzero (all keys
// in a set), 1 popcount of v & m, 2 sum of v & m.
template <bool set_, typename V>
__global__ void __launch_bounds__(256) reduce_kernel(const Dev_Table T, const uint32_t what, const uint64_t mask, unsigned long long* out)
{
    const uint64_t total = T.cap * B + T.ov_mask + 1;
    unsigned long long acc = 0;
    for(uint64_t s = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; s < total; s += uint64_t(gridDim.x) * blockDim.x)
    {
        unsigned long long raw = 0;
        if(!slot_value<set_>(T, s, raw))
            continue;
        const uint64_t x = static_cast<uint64_t>(static_cast<V>(raw)) & mask;
        if(set_)
            acc += 1;
        else if(what == 0)
            acc += x != 0;
        else if(what == 1)
            acc += __popcll(x);
        else
            acc += x;
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1)
        acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
    if((threadIdx.x & 31) == 0 && acc)
        atomicAdd(out, acc);
}

// The histogram of the values in [1, hmax] (counter/Kmer_Set_Counter.cpp:96-119), added to hist[0..hmax]. Counts of k-mers
// crowd on a few values, so a block counts those up to hist_bins in shared memory and adds its bins up at the end; one
// global atomic per key on those few words took 41.8 ms over 100M keys, against 0.62 with the blocks' bins (reading the 2.1 GB table takes 0.33).
constexpr uint32_t hist_bins = 8192;    // 32 KB: six blocks per SM.

template <typename V>
__global__ void __launch_bounds__(256) histogram_kernel(const Dev_Table T, const uint64_t hmax, unsigned long long* hist)
{
    __shared__ uint32_t bins[hist_bins];
    const uint32_t held = static_cast<uint32_t>(min(hmax + 1, static_cast<uint64_t>(hist_bins)));
    for(uint32_t i = threadIdx.x; i < held; i += blockDim.x)
        bins[i] = 0;
    __syncthreads();
    const uint64_t total = T.cap * B + T.ov_mask + 1;
    // A block's share of the slots stays below 2^32, so its bins cannot overflow.
    for(uint64_t s = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; s < total; s += uint64_t(gridDim.x) * blockDim.x)
    {
        unsigned long long raw = 0;
        if(!slot_value<false>(T, s, raw))
            continue;
        const uint64_t v = static_cast<uint64_t>(static_cast<V>(raw));
        if(v < held)
            atomicAdd(bins + v, 1u);
        else if(v <= hmax)
            atomicAdd(hist + v, 1ull);
    }
    __syncthreads();
    for(uint32_t i = threadIdx.x; i < held; i += blockDim.x)
        if(i > 0 && bins[i])
            atomicAdd(hist + i, static_cast<unsigned long long>(bins[i]));
}

// Placement statistics (include/Streaming_Kmer_Hash_Table.hpp:1108-1120,2729-2752): keys in their primary bucket
// and keys in another, from recomputed minimizer hashes.
template <int k, int l, bool set_>
__global__ void __launch_bounds__(256) distribution_kernel(const Dev_Table T, unsigned long long* prim_sec)
{
    const uint64_t n_main = T.cap * B;
    unsigned long long p = 0, s2 = 0;
    for(uint64_t s = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; s < n_main; s += uint64_t(gridDim.x) * blockDim.x)
    {
        if(!*cs_of(T, static_cast<uint32_t>(s / B), s % B))
            continue;
        const uint64_t key = ~T.slots[s * slot_words<set_>()];
        if(bucket_of(minimizer_hash<k, l>(key), T.cap) == s / B)
            p++;
        else
            s2++;
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1)
        p += __shfl_xor_sync(0xFFFFFFFFu, p, o), s2 += __shfl_xor_sync(0xFFFFFFFFu, s2, o);
    if((threadIdx.x & 31) == 0)
        atomicAdd(prim_sec, p), atomicAdd(prim_sec + 1, s2);
}

// Single k-mer lookups (include/Streaming_Kmer_Hash_Table.hpp:2608-2645) of canonical keys: out[2i] = found,
// out[2i+1] = value.
template <int k, int l, bool set_, typename V>
__global__ void get_kernel(const Dev_Table T, const uint64_t* keys, const uint64_t n, unsigned long long* out)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if(i >= n)
        return;
    const uint64_t key = keys[i];
    const unsigned long long* v = find_chain<set_, false>(T, key, minimizer_hash<k, l>(key), checksum_of(key));
    out[2 * i] = v != nullptr;
    out[2 * i + 1] = (v && !set_) ? static_cast<unsigned long long>(read_val<V>(v)) : 0ull;
}

// The staging of a device batch, or of several run as one: its sequences are counted, the counts summed, and its segments
// listed, with no host read in between. The launch behind it takes its number of segments from ctr[6]: none if the batch
// has more segments or positions than the caller made room for, which the host reads with the launch's results. Up to
// small_stage_max sequences take one block (stage_small_kernel), more take two launches (stage_count_kernel,
// stage_list_kernel). A million sequences take 26 and 30 us; a counting kernel, two scans, a search per segment and the
// host's read of the counts before it took 45 us of kernels and about 30 of waiting.
constexpr uint32_t small_stage_max = 4096;      // Sequences of a block (at most 4 per thread).
constexpr uint32_t small_segs_max = 16384;      // Segments that a block lists.
constexpr uint32_t stage_block = 1024;

struct Stage
{
    // One batch's n + 1 offsets; or (null) several batches, 8 words each -- bases, offsets, sequences, first merged
    // sequence, out0, out1, out2, 0 -- in batch order, with, to be filled, the address of each merged sequence's first
    // base, its batch, and each batch's first merged position.
    const uint64_t* off;
    const uint64_t* desc;
    uint64_t count;
    uint64_t* addr;
    uint32_t* batch_of;
    uint64_t* pos_base;
    bool zero_out0;             // Zeroes each sequence's word of its batch's out0.
    bool group;                 // May make groups (of more than small_stage_max sequences).
    uint64_t n;
    int k;
    uint32_t sms;
    uint64_t max_segs, max_pos;
    uint64_t *npos, *pos_off, *seg_off;     // Positions of each sequence, with in_group; n + 1 sums of positions and of segments.
    unsigned long long* blocks;     // Three words per block of stage_count_kernel: the positions before it, the entries, and the segments were there no groups.
    Segment *segs, *groups;
    unsigned long long* ctr;    // [0] and the low half of [2] are zeroed; [3..6]: positions, segments, segment length, segments to run; [7]: zero between launches; [8] is zeroed; [9]: whether the segments fit the list; [10], [11]: groups to run, and listed.
    unsigned long long* zero;   // zero_n words zeroed.
    uint64_t zero_n;
};

// The length of sequence q. Of several batches, `lo` is a batch at or before q's (or, at first, no less than 0 with
// `seek`), and becomes q's; the sequence's entries are filled.
__device__ __forceinline__ uint64_t stage_length(const Stage& a, const uint64_t q, uint64_t& lo, const bool seek)
{
    if(a.desc == nullptr)
        return a.off[q + 1] - a.off[q];
    if(seek)
        for(uint64_t hi = a.count; hi - lo > 1; )   // The last batch whose first merged sequence is at or before q.
        {
            const uint64_t mid = (lo + hi) / 2;
            if(a.desc[8 * mid + 3] <= q)
                lo = mid;
            else
                hi = mid;
        }
    while(lo + 1 < a.count && a.desc[8 * (lo + 1) + 3] <= q)
        ++lo;
    const uint64_t* d = a.desc + 8 * lo;
    const uint64_t j = q - d[3], b0 = reinterpret_cast<const uint64_t*>(d[1])[j];
    a.addr[q] = d[0] + b0;
    a.batch_of[q] = static_cast<uint32_t>(lo);
    if(a.zero_out0)
        reinterpret_cast<uint64_t*>(d[4])[j] = 0;
    return reinterpret_cast<const uint64_t*>(d[1])[j + 1] - b0;
}

constexpr uint64_t in_group = uint64_t(1) << 63;

// Segments and groups are counted together, in 34 bits and 30.
constexpr int group_shift = 34;
constexpr uint64_t segs_mask = (uint64_t(1) << group_shift) - 1;
__device__ __forceinline__ uint64_t entries(const uint64_t q, const uint64_t np, const bool g)
{
    return g ? uint64_t(q % group_seqs == 0) << group_shift : (np + seg_positions - 1) / seg_positions;
}

// Groups of short sequences (device_stream.cuh), the first a multiple of group_seqs, are made where that saves instructions, in
// units of ten a warp: 55 for a row of a group (43, but its lanes have several sequences' k-mers and so more buckets: reads of
// 75 bases at 45 were no faster in groups) and 1 for 23 of its bases against 31 for a row of a sequence and 13 to start on
// one. And a batch has groups only if they save more than the launch over them takes, at 14 ps a unit with all SMs at work:
// some 7 us, and up to 50 beside a launch over segments that fills the SMs by itself. (Lookups of 60,000 reads of about 100
// bases, a few of them in groups, took 149 us with those and 118 without; of 60,000 of 33, 55 with and 69 without.)
__device__ __forceinline__ bool groups_pay(const uint64_t saved, const uint64_t segs) { return saved >= min(500'000 + 2'000 * segs, uint64_t(4'000'000)); }

// What the group of the calling lane's sequence q, of batch `lo`, saves in those units; 0 if it is not to be one. A whole warp,
// with consecutive sequences.
__device__ __forceinline__ uint32_t group_saves(const Stage& a, const uint64_t q, const uint64_t len, const uint64_t np, const uint64_t lo)
{
    constexpr uint32_t all = 0xFFFFFFFFu;
    if(!a.group)
        return 0;
    const int leader = static_cast<int>(threadIdx.x & 31 & ~(group_seqs - 1));
    const uint64_t lo_leader = __shfl_sync(all, lo, leader);    // (All lanes take part: not behind a condition.)
    const bool ok = q < a.n && len <= group_len && lo == lo_leader;
    const uint32_t no = (__ballot_sync(all, !ok) >> leader) & ((1u << group_seqs) - 1);
    // Bases, positions and rows of the sequences by themselves, in 12 bits, 12 and 8.
    uint32_t x = ok ? static_cast<uint32_t>(len << 20 | np << 8 | (np + 31) / 32) : 0;
#pragma unroll
    for(uint32_t o = 1; o < group_seqs; o *= 2)
        x += __shfl_xor_sync(all, x, o);
    const uint32_t bases = x >> 20, pos = x >> 8 & 0xFFFu, rows = x & 0xFFu;
    const uint32_t with = 55 * ((pos + 31) / 32) + bases / 23 + 10, without = 31 * rows + 13 * group_seqs;
    return no == 0 && pos > 0 && with < without ? without - with : 0;
}

// The group that starts at sequence q: `pos` positions, from `first` on, the last sequence's np_last among them.
__device__ __forceinline__ Segment stage_group(const Stage& a, const uint64_t q, const uint64_t pos, const uint64_t first, const uint64_t np_last)
{
    const uint64_t* at = (a.desc ? a.addr : a.off) + q;
    const uint64_t bases = at[group_seqs - 1] - at[0] + (np_last ? np_last + a.k - 1 : 0);
    return Segment{at[0], first, q, group_word(static_cast<uint32_t>(pos), static_cast<uint32_t>(bases)), a.desc ? a.batch_of[q] : 0};
}

// Segment number i of sequence q, which starts at `first` of its np positions.
__device__ __forceinline__ Segment stage_segment(const Stage& a, const uint64_t q, const uint64_t i, const uint64_t np, const uint64_t first, const uint64_t seg_len)
{
    const uint64_t p0 = i * seg_len;
    return Segment{(a.desc ? a.addr[q] : a.off[q]) + p0, first + p0, q, static_cast<uint32_t>(min(np - p0, seg_len)), a.desc ? a.batch_of[q] : 0};
}

// Makes each of x the inclusive sum of its own over the block's threads in order; warps[.][31] is then the block's.
template <int n_>
__device__ __forceinline__ void block_sums(unsigned long long (&x)[n_], unsigned long long (*warps)[32])
{
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const auto warp_sum = [&](unsigned long long& a)
    {
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, a, o);
            if(lane >= static_cast<uint32_t>(o))
                a += y;
        }
    };
    __syncthreads();    // The words' last use is over.
#pragma unroll
    for(int i = 0; i < n_; ++i)
    {
        warp_sum(x[i]);
        if(lane == 31)
            warps[i][wid] = x[i];
    }
    __syncthreads();
    if(wid < n_)
    {
        unsigned long long a = warps[wid][lane];
        warp_sum(a);
        warps[wid][lane] = a;
    }
    __syncthreads();
#pragma unroll
    for(int i = 0; i < n_; ++i)
        x[i] += wid ? warps[i][wid - 1] : 0;
}

// The inclusive sum of x over the block's threads in order; `warps` is 32 words of shared memory.
__device__ __forceinline__ unsigned long long block_sum(const unsigned long long x, unsigned long long* warps)
{
    unsigned long long a[1] = {x};
    block_sums<1>(a, reinterpret_cast<unsigned long long(*)[32]>(warps));
    return a[0];
}

// The sum of x over the warp.
__device__ __forceinline__ unsigned long long warp_total(unsigned long long x)
{
#pragma unroll
    for(int o = 16; o > 0; o >>= 1)
        x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
    return x;
}

static __global__ void __launch_bounds__(stage_block) stage_small_kernel(const Stage a)
{
    __shared__ unsigned long long wp[32], ws[32];
    __shared__ uint32_t first_seg[small_stage_max + 1];
    const uint32_t t = threadIdx.x;
    const uint64_t per = (a.n + stage_block - 1) / stage_block, q0 = min(a.n, uint64_t(t) * per);
    const uint32_t mine = static_cast<uint32_t>(min(a.n, q0 + per) - q0);
    uint64_t np[4], lo = 0;
    unsigned long long P = 0, S = 0;
#pragma unroll
    for(uint32_t i = 0; i < 4; ++i)
        if(i < mine)
        {
            const uint64_t len = stage_length(a, q0 + i, lo, i == 0);
            np[i] = len >= uint64_t(a.k) ? len - a.k + 1 : 0;
            P += np[i];
        }
    for(uint64_t i = t; i < a.zero_n; i += stage_block)
        a.zero[i] = 0;
    unsigned long long bp = block_sum(P, wp) - P;
    const uint64_t total = wp[31], seg_len = fitted_seg_len(total, a.sms);
#pragma unroll
    for(uint32_t i = 0; i < 4; ++i)
        if(i < mine)
            S += (np[i] + seg_len - 1) / seg_len;
    unsigned long long bs = block_sum(S, ws) - S;
    const uint64_t nsegs = ws[31], run = nsegs <= a.max_segs && total <= a.max_pos ? nsegs : 0;
#pragma unroll
    for(uint32_t i = 0; i < 4; ++i)
        if(i < mine)
        {
            const uint64_t q = q0 + i;
            a.pos_off[q] = bp, a.seg_off[q] = bs;
            if(run)
                first_seg[q] = static_cast<uint32_t>(bs);
            if(a.desc && a.desc[8 * uint64_t(a.batch_of[q]) + 3] == q)
                a.pos_base[a.batch_of[q]] = bp;
            bp += np[i], bs += (np[i] + seg_len - 1) / seg_len;
        }
    if(t == stage_block - 1)
    {
        a.pos_off[a.n] = total, a.seg_off[a.n] = nsegs;
        a.ctr[3] = total, a.ctr[4] = nsegs, a.ctr[5] = seg_len, a.ctr[6] = run;
        a.ctr[0] = 0, *reinterpret_cast<uint32_t*>(a.ctr + 2) = 0, a.ctr[8] = 0, a.ctr[9] = nsegs <= a.max_segs, a.ctr[10] = 0, a.ctr[11] = 0;
    }
    __syncthreads();
    for(uint32_t i = t; i < run; i += stage_block)
    {
        uint32_t l = 0, h = static_cast<uint32_t>(a.n);     // The last q with first_seg[q] <= i.
        while(h - l > 1)
        {
            const uint32_t mid = (l + h) / 2;
            if(first_seg[mid] <= i)
                l = mid;
            else
                h = mid;
        }
        const uint64_t first = a.pos_off[l];
        a.segs[i] = stage_segment(a, l, i - first_seg[l], a.pos_off[l + 1] - first, first, seg_len);
    }
}

// Larger batches, first launch: each block counts stage_block sequences, and the block that ends last sums the blocks'
// counts. The segments are listed behind it (stage_list_kernel) if they are not many more than the sequences, nor too many
// of them one block's: otherwise the host, which reads so, lists them by a thread each (segs_kernel).
static __global__ void __launch_bounds__(stage_block) stage_count_kernel(const Stage a)
{
    __shared__ unsigned long long w[3][32];
    __shared__ bool last, most[2];      // `most`: whether a block has too many segments, without groups and with.
    const uint32_t t = threadIdx.x;
    const uint64_t q = uint64_t(blockIdx.x) * stage_block + t;
    uint64_t np = 0, len = 0, lo = 0;
    if(q < a.n)
    {
        len = stage_length(a, q, lo, true);
        np = len >= uint64_t(a.k) ? len - a.k + 1 : 0;
    }
    const uint32_t saves = group_saves(a, q, len, np, lo);
    if(q < a.n)
        a.npos[q] = saves ? np | in_group : np;
    for(uint64_t i = q; i < a.zero_n; i += uint64_t(gridDim.x) * stage_block)
        a.zero[i] = 0;
    // The block's positions; its entries; the segments without groups, and above them what the groups would save, in sixteens
    // of its units.
    unsigned long long p = warp_total(np), x = a.group ? warp_total(entries(q, np, saves != 0)) : 0;
    unsigned long long y = warp_total(entries(q, np, false) | uint64_t(q % group_seqs ? 0 : saves / 16) << group_shift);
    if((t & 31) == 0)
        w[0][t >> 5] = p, w[1][t >> 5] = x, w[2][t >> 5] = y;
    __syncthreads();
    if(t < 32)
    {
        p = warp_total(w[0][t]), x = warp_total(w[1][t]), y = warp_total(w[2][t]);
        if(t == 0)
        {
            __stcg(a.blocks + 3 * blockIdx.x, p), __stcg(a.blocks + 3 * blockIdx.x + 1, x), __stcg(a.blocks + 3 * blockIdx.x + 2, y);
            __threadfence();
            last = atomicAdd(a.ctr + 7, 1ull) == gridDim.x - 1, most[0] = most[1] = false;
            __threadfence();
        }
    }
    __syncthreads();
    if(!last)
        return;
    unsigned long long P = 0, S = 0, Q = 0;
    for(uint64_t b0 = 0; b0 < gridDim.x; b0 += stage_block)
    {
        const uint64_t b = b0 + t;
        const bool in = b < gridDim.x;
        p = in ? __ldcg(a.blocks + 3 * b) : 0, x = in ? __ldcg(a.blocks + 3 * b + 1) : 0, y = in ? __ldcg(a.blocks + 3 * b + 2) : 0;
        unsigned long long to[3] = {p, x, y};
        block_sums(to, w);
        if((y & segs_mask) > small_segs_max)
            most[0] = true;
        if((x & segs_mask) > small_segs_max)
            most[1] = true;
        if(in)
            a.blocks[3 * b] = P + to[0] - p, a.blocks[3 * b + 1] = S + to[1] - x, a.blocks[3 * b + 2] = Q + to[2] - y;
        P += w[0][31], S += w[1][31], Q += w[2][31];
    }
    __syncthreads();
    if(t == 0)
    {
        const bool g = groups_pay((Q >> group_shift) * 16, S & segs_mask);
        const uint64_t segs = (g ? S : Q) & segs_mask, groups = g ? S >> group_shift : 0;
        const bool fits = segs <= a.max_segs && !most[g], run = fits && P <= a.max_pos;
        a.pos_off[a.n] = P, a.seg_off[a.n] = segs;
        a.ctr[3] = P, a.ctr[4] = segs, a.ctr[5] = seg_positions, a.ctr[6] = run ? segs : 0;
        a.ctr[0] = 0, *reinterpret_cast<uint32_t*>(a.ctr + 2) = 0, a.ctr[7] = 0, a.ctr[8] = 0, a.ctr[9] = fits;
        a.ctr[10] = run ? groups : 0, a.ctr[11] = groups;
    }
}

// Second launch: each block sums its own sequences and lists their segments and groups. A thread writes an entry in some 30 ns, so it
// lists its own sequence if that has up to own_segs; a longer one's are listed by its warp, an entry per lane. (A thread
// each took 5.9 ms for 5,000 sequences one of which has 90 Mbp, and 1.67 for 200,000 with one of 25 Mbp.)
constexpr uint32_t own_segs = 32;

static __global__ void __launch_bounds__(stage_block) stage_list_kernel(const Stage a)
{
    __shared__ unsigned long long w[2][32];
    const uint64_t q = uint64_t(blockIdx.x) * stage_block + threadIdx.x;
    constexpr uint32_t all = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31;
    uint64_t np = q < a.n ? a.npos[q] : 0;
    const bool groups = a.ctr[11] != 0, g = groups && (np & in_group);
    np &= ~in_group;
    const uint64_t x = entries(q, np, g), ns = x & segs_mask;
    unsigned long long to_here[2] = {np, x};
    block_sums(to_here, w);
    const unsigned long long first = a.blocks[3 * blockIdx.x] + to_here[0] - np, before = a.blocks[3 * blockIdx.x + (groups ? 1 : 2)] + to_here[1] - x;
    const uint64_t first_seg = before & segs_mask;
    if(q < a.n)
    {
        a.pos_off[q] = first, a.seg_off[q] = first_seg;
        if(a.desc && a.desc[8 * uint64_t(a.batch_of[q]) + 3] == q)
            a.pos_base[a.batch_of[q]] = first;
    }
    if(__any_sync(all, g))
    {
        // The positions up to the group's end, from its last lane.
        const int end = static_cast<int>(lane | (group_seqs - 1));
        const uint64_t to = __shfl_sync(all, first + np, end), np_last = __shfl_sync(all, np, end);
        if(x >> group_shift)
            a.groups[before >> group_shift] = stage_group(a, q, to - first, first, np_last);
    }
    if(a.ctr[6] == 0)
        return;
    if(ns <= own_segs)
        for(uint64_t i = 0; i < ns; ++i)
            a.segs[first_seg + i] = stage_segment(a, q, i, np, first, seg_positions);
    for(uint32_t m = __ballot_sync(all, ns > own_segs); m; m &= m - 1)
    {
        const int s = __ffs(m) - 1;
        const uint64_t q_s = q - lane + s, np_s = __shfl_sync(all, np, s), ns_s = __shfl_sync(all, ns, s);
        const uint64_t first_s = __shfl_sync(all, first, s), at = __shfl_sync(all, first_seg, s);
        for(uint64_t i = lane; i < ns_s; i += 32)
            a.segs[at + i] = stage_segment(a, q_s, i, np_s, first_s, seg_positions);
    }
}

// Lists the segments [sb, se) of a staged batch at `segs`, one thread per segment: its sequence by binary search in
// seg_off[0..n] (exclusive sums of segments per sequence), so that long sequences' many segments are listed in parallel.
static __global__ void segs_kernel(const Stage a, const uint64_t sb, const uint64_t se, const uint32_t seg_len, Segment* segs)
{
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for(uint64_t i = sb + uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < se; i += stride)
    {
        uint64_t lo = 0, hi = a.n;      // The last q with seg_off[q] <= i.
        while(hi - lo > 1)
        {
            const uint64_t mid = (lo + hi) / 2;
            if(a.seg_off[mid] <= i)
                lo = mid;
            else
                hi = mid;
        }
        const uint64_t first = a.pos_off[lo];
        segs[i - sb] = stage_segment(a, lo, i - a.seg_off[lo], a.pos_off[lo + 1] - first, first, seg_len);
    }
}

}
