// Device-side primitives of the B200 streaming k-mer table: hashing, bucket arithmetic, the per-bucket layout.
//
// The arithmetic that decides what a k-mer *is* follows kache-hash bit for bit:
//   - 2-bit codes A0 C1 G2 T3, case-insensitive: ((ch >> 2) ^ (ch >> 1)) & 3      (include/Kmer_Batch.hpp:108)
//   - canonical = min(forward, reverse complement), orientation = key == forward (include/Kmer_Batch.hpp:230-241)
//   - capacity in buckets = cap_for(n, lf, pow2)                      (include/Streaming_Kmer_Hash_Table.hpp:1004-1011)
// as does the description of a k-mer that callers can ask for (its 2-bit encoding, checksum and the least of Wang's
// hashes of its canonical l-mers: include/Kmer_Batch.hpp:24-67,204-227).
//
// Where a key sits in the table is not observable, so how it is held and placed is this library's own: a key is two
// planes of k bits, the high and the low bits of its codes, which a warp has as two ballots of 32 bases; a bucket is
// picked by the least of a 32-bit hash of the k-mer's canonical l-mers, so that consecutive k-mers share buckets, as the
// reference's minimizers have them do, at a fraction of the instructions of 64-bit hashes.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace kache_b200
{

constexpr int B = 32;                  // Slots per bucket: a bucket's 32 checksums fill one 32-byte sector.
constexpr uint64_t max_buckets = (uint64_t(1) << 32) - 1;
constexpr int seg_rows = 16;           // Rows of 32 k-mer positions that one warp describes in a segment.
constexpr int seg_positions = 32 * seg_rows;
constexpr uint64_t max_seg_index = 0xFFFFFF;   // Segment indexes take 24 bits of a segment list entry.

// The segment length for a batch of `total` positions on `sms` SMs: seg_positions, halved down to one row of 32 while
// the batch would give each SM fewer than 32 warps, so that a small call's rows run side by side instead of in turn.
__host__ __device__ __forceinline__ uint32_t fitted_seg_len(const uint64_t total, const uint32_t sms)
{
    uint32_t s = seg_positions;
    while(s > 32 && total < uint64_t(s) * sms * 32)
        s /= 2;
    return s;
}

enum Op : uint32_t { OP_KEEP = 0, OP_ASSIGN = 1, OP_ADD = 2, OP_OR = 3, OP_MIN = 4, OP_MAX = 5, OP_ADD_WRAP = 16 };

// ---- What callers can see of a k-mer ---------------------------------------------------------------------------

// Wang's hash with its shift-and-add steps written as multiplications by constants, modulo 2^64:
// ~x + (x << 21) = x * (2^21 - 1) - 1, x + (x << 3) + (x << 8) = x * 265, x + (x << 2) + (x << 4) = x * 21,
// x + (x << 31) = x * (2^31 + 1). Same value.
__host__ __device__ __forceinline__ uint64_t wang_u64(uint64_t x)
{
    x = x * ((1ull << 21) - 1) - 1;
    x = x ^ (x >> 24);
    x = x * 265;
    x = x ^ (x >> 14);
    x = x * 21;
    x = x ^ (x >> 28);
    x = x * ((1ull << 31) + 1);
    return x;
}

// The described 8-bit checksum of a 2-bit encoded key: the top byte of key times an odd constant, never 0, as the
// reference's builds without AVX-512 compute it (include/Kmer_Batch.hpp:44-67).
__host__ __device__ __forceinline__ uint8_t described_checksum(const uint64_t key)
{
    const uint8_t c = static_cast<uint8_t>((key * 0x9E3779B97F4A7C15ull) >> 56);
    return c ? c : 1;
}

__host__ __device__ __forceinline__ uint64_t kmer_mask(const int k) { return k == 32 ? ~0ull : (1ull << (2 * k)) - 1; }

// Reverse complement of a 2k-bit k-mer: complement, reverse the 32 2-bit groups, align.
__device__ __forceinline__ uint64_t revcomp(const uint64_t x, const int k)
{
    uint64_t t = __brevll(~x);
    t = ((t >> 1) & 0x5555555555555555ull) | ((t & 0x5555555555555555ull) << 1);
    return t >> (64 - 2 * k);
}

// The described minimizer hash of a 2-bit encoded canonical key: the least Wang hash of its l-mers' canonical forms
// (include/Kmer_Lanes.hpp:247-274); the l-mer at offset p of the key has its reverse complement at offset k - l - p
// of the key's reverse complement.
template <int k, int l>
__device__ __forceinline__ uint64_t described_minimizer(const uint64_t key)
{
    constexpr int w = k - l + 1;
    const uint64_t lm = kmer_mask(l);
    const uint64_t r = revcomp(key, k);
    uint64_t h = ~0ull;
    for(int p = 0; p < w; ++p)
    {
        const uint64_t f = (key >> (2 * (k - l - p))) & lm;
        const uint64_t b = (r >> (2 * p)) & lm;
        const uint64_t x = wang_u64(f < b ? f : b);
        h = x < h ? x : h;
    }
    return h;
}

// ---- Keys as planes ----------------------------------------------------------------------------------------------

// A k-mer's planes: bit k - 1 - i of `hi` and `lo` are the high and low bit of its base i's code.
struct Planes
{
    uint32_t hi, lo;
};

__host__ __device__ __forceinline__ uint32_t plane_mask(const int n) { return n == 32 ? ~0u : (1u << n) - 1; }

__host__ __device__ __forceinline__ uint64_t key_of(const Planes x) { return (uint64_t(x.hi) << 32) | x.lo; }
__host__ __device__ __forceinline__ Planes planes_of(const uint64_t key) { return Planes{static_cast<uint32_t>(key >> 32), static_cast<uint32_t>(key)}; }

// Bit i of x at bit 2i.
__host__ __device__ __forceinline__ uint64_t spread_bits(const uint32_t x)
{
    uint64_t y = x;
    y = (y | (y << 16)) & 0x0000FFFF0000FFFFull;
    y = (y | (y << 8)) & 0x00FF00FF00FF00FFull;
    y = (y | (y << 4)) & 0x0F0F0F0F0F0F0F0Full;
    y = (y | (y << 2)) & 0x3333333333333333ull;
    y = (y | (y << 1)) & 0x5555555555555555ull;
    return y;
}

// The 2-bit encoding of a key held as planes, as iteration and descriptions return it.
__host__ __device__ __forceinline__ uint64_t encoding_of(const uint64_t key)
{
    return (spread_bits(static_cast<uint32_t>(key >> 32)) << 1) | spread_bits(static_cast<uint32_t>(key));
}

// The key of a 2-bit encoding.
__host__ __device__ __forceinline__ uint64_t key_of_encoding(const uint64_t e)
{
    uint64_t key = 0;
    for(int i = 0; i < 32; ++i)
        key |= ((e >> (2 * i + 1)) & 1) << (32 + i) | ((e >> (2 * i)) & 1) << i;
    return key;
}

// Whether the k-mer f is greater than the k-mer r in the order of their 2-bit encodings: at the first base where they
// differ, the top set bit of `a` (bases where f's code is the greater) or of `b` (where r's is) decides.
__device__ __forceinline__ bool planes_greater(const Planes f, const Planes r)
{
    const uint32_t same = ~(f.hi ^ r.hi);
    const uint32_t a = (f.hi & ~r.hi) | (same & f.lo & ~r.lo);
    const uint32_t b = (r.hi & ~f.hi) | (same & r.lo & ~f.lo);
    return a > b;
}

// ---- Bases ----------------------------------------------------------------------------------------------------------

// What a row needs of a character: bit 0 whether it is one of A, C, G, T, bits 1 and 2 the low and high bit of its code.
__device__ __forceinline__ uint8_t base_bits(const uint32_t ch)
{
    const uint32_t x = (ch | 0x20u) - 'a';
    return static_cast<uint8_t>((x < 20u && ((0x80045u >> x) & 1u)) | ((ch ^ (ch >> 1)) & 6u));
}

// ---- Placement ---------------------------------------------------------------------------------------------------

// The kernels that describe and probe are bound by their instructions, most of all by the pipe of integer logic, shifts and
// compares; multiply-adds run beside it, so hashes are multiply-adds as far as they go.
// Their 32-bit factors are the five primes of xxHash, taken only as numbers of well mixed bits (lmer_hash has two of them off
// by one, to be even); what is done with them is this library's own.

// The key's 8-bit checksum in the table, 1..255 (0 marks an empty slot).
__device__ __forceinline__ uint32_t checksum_of(const uint64_t key)
{
    return __umulhi(static_cast<uint32_t>(key >> 32) * 0x27D4EB2Fu + static_cast<uint32_t>(key) * 0x9E3779B1u, 255u) + 1;
}

constexpr uint32_t lmer_seed = 0x809CB0CBu;

// The hash of an l-mer, given in both orientations: the product of two odd numbers that each orientation gives alike, so
// the order of the two does not matter and neither has to be found the lesser; its halves are then mixed. (The constants
// send the l-mer of all A's to a large hash, so that runs of A's, frequent in genomes, do not all land in one bucket.)
__device__ __forceinline__ uint32_t lmer_hash(const Planes f, const Planes r)
{
    const uint32_t a = f.hi * 0x9E3779B2u + (f.lo * 0x85EBCA76u + lmer_seed), b = r.hi * 0x9E3779B2u + (r.lo * 0x85EBCA76u + lmer_seed);
    const uint64_t x = uint64_t(a) * b;
    return static_cast<uint32_t>(x >> 32) * 0xC2B2AE3Du + static_cast<uint32_t>(x);
}

// The primary bucket of a minimizer hash. The least of several hashes has small values, so its bits are spread by a
// multiply first.
__device__ __forceinline__ uint32_t bucket_of(const uint32_t h, const uint64_t cap)
{
    return __umulhi(h * 0x9E3779B1u, static_cast<uint32_t>(cap));
}

// The index, 1..255, of a minimizer hash in its bucket's spill filter.
__host__ __device__ __forceinline__ uint32_t filter_pos(const uint32_t h)
{
    const uint32_t x = (h * 0x165667B1u) >> 24;
    return x + (x == 0);
}

// Stafford's 64-bit finaliser (variant 13).
__host__ __device__ __forceinline__ uint64_t mix64(uint64_t x)
{
    x ^= x >> 30, x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27, x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

// The secondary buckets of a minimizer hash: one copy of each key, so every inserter of a key scans them in this one
// order.
__device__ __forceinline__ uint32_t second_bucket(const uint32_t h, const uint64_t cap)
{
    return static_cast<uint32_t>(__umul64hi(mix64(h ^ 0x2545F4914F6CDD1Dull), cap));
}
__device__ __forceinline__ uint32_t third_bucket(const uint32_t h, const uint64_t cap)
{
    return static_cast<uint32_t>(__umul64hi(mix64(h + 0x9E3779B97F4A7C15ull), cap));
}

__host__ __device__ __forceinline__ uint64_t ov_hash(const uint64_t key) { return mix64(key ^ 0xD6E8FEB86659FD93ull); }

// The reverse complement of a k-mer: the complement of each code, in reverse order.
__device__ __forceinline__ Planes revcomp_planes(const Planes x, const int k)
{
    return Planes{__brev(~x.hi) >> (32 - k), __brev(~x.lo) >> (32 - k)};
}

// The minimizer hash of a canonical key: the least hash of its l-mers; the l-mer at offset p of the key has its reverse
// complement at offset k - l - p of the key's reverse complement.
template <int k, int l>
__device__ __forceinline__ uint32_t minimizer_hash(const uint64_t key)
{
    constexpr int w = k - l + 1;
    const uint32_t lm = plane_mask(l);
    const Planes f = planes_of(key), r = revcomp_planes(f, k);
    uint32_t h = ~0u;
#pragma unroll
    for(int p = 0; p < w; ++p)
        h = min(h, lmer_hash(Planes{(f.hi >> (k - l - p)) & lm, (f.lo >> (k - l - p)) & lm}, Planes{(r.hi >> p) & lm, (r.lo >> p) & lm}));
    return h;
}

// Bit 7 of each byte of the result is set iff that byte of w is zero, exactly (no carries cross bytes).
__device__ __forceinline__ uint32_t zero_bytes(const uint32_t w)
{
    return ~(((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w) & 0x80808080u;
}

// Where a bucket's checksum of slot j is among its 32 bytes: byte j / 8 of word j % 8, so that the merge below ends with
// slot j's bit at j.
__host__ __device__ __forceinline__ uint32_t cs_byte(const uint32_t j) { return 4 * (j & 7) + (j >> 3); }

// Bit j is set for the slots j of a bucket whose checksum (of the 32 bytes a, b) may equal c. With exact_, exactly for
// those. Without, for every checksum equal to c and possibly for the byte just above one in the same word (the borrow of
// the subtraction reaches it only if it equals c ^ 1): callers verify candidates by their keys.
template <bool exact_>
__device__ __forceinline__ uint32_t candidates32(const uint4 a, const uint4 b, const uint32_t c)
{
    const uint32_t cc = c * 0x01010101u;
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t m = 0;
#pragma unroll
    for(int i = 0; i < 8; ++i)
    {
        const uint32_t t = w[i] ^ cc;
        const uint32_t y = exact_ ? zero_bytes(t) : (t - 0x01010101u) & ~t & 0x80808080u;
        m = y + (m >> 1);
    }
    return m;
}

// The index of the highest set bit of x, which is not 0.
__device__ __forceinline__ uint32_t top_bit(const uint32_t x)
{
    uint32_t r;
    asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}

}
