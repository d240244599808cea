// The rules that plan an MSM batch from its sizes alone: windows, affine
// rounds and their scratch, and how large batches are divided.  Host code
// without CUDA, so that they can be checked over their whole range on the CPU.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#if defined(__CUDACC__)
#define GB_RULE __host__ __device__ constexpr
#else
#define GB_RULE constexpr
#endif

namespace gb {

static constexpr int kMaxWindowBits = 16;  // 2^15 u32 counters = 128 KB smem

// A scalar's 255 bits in windows of c and c - 1 bits, the wider ones first, so
// that no window is a remainder of a few bits whose digits would crowd a few
// buckets.  A (c - 1)-bit digit is at most 2^(c - 1), carry included, so it
// stays positive and fills all the buckets; the top window is always one of
// these (scalars are below 2^255, and 255 < windows c), so no carry is left.
GB_RULE int windows_for(int c) { return 255 / c + 1; }
GB_RULE int window_bits(int c, int j) { return j < 255 - windows_for(c) * (c - 1) ? c : c - 1; }
GB_RULE int window_offset(int c, int j)
{
    const int wide = 255 - windows_for(c) * (c - 1);
    return j < wide ? j * c : wide * c + (j - wide) * (c - 1);
}

// an MSM's digits are numbered with 31 bits
static constexpr uint64_t kMaxDigits = 0x7fffffff;

// Window size for n points, measured on GB300.  With the precomputed table an
// MSM has 2^(c - 1) buckets in all: ms a call for one and for three MSMs (*
// chosen)
//   2^8 points   c = 8 0.16 0.19, 10 0.15 0.18, 11* 0.14 0.18, 12 0.15 0.20
//   2^10         10 0.17 0.21, 11* 0.16 0.21, 12 0.16 0.23, 13 0.17 0.24
//   2^12         11 0.21 0.31, 12* 0.20 0.31, 13 0.20 0.31, 14 0.23 0.38
//   2^14         12 0.31 0.63, 13* 0.30 0.61, 14 0.32 0.63, 15 0.35 0.67
//   2^16         13 0.70 1.42, 14 0.67 1.43, 15* 0.67 1.41, 16 0.68 1.47
//   2^17         13 1.13 2.44, 15 1.08 2.38, 16* 1.03 2.41
// Without it every window has its own buckets:
//   2^10 points  8* 0.46, 9 0.47, 10 0.51
//   2^12         8 0.52, 9* 0.52, 10 0.54
//   2^14         9 0.71, 10* 0.71, 11 0.75
//   2^16         10 1.14, 11* 1.11, 12 1.13, 13 1.18
//   2^18         11 2.31, 12* 2.25, 13 2.30
inline int choose_window(size_t n, bool precomputed)
{
    auto upto = [&](int lg) { return n <= (size_t)1 << lg; };
    if (precomputed) return upto(7) ? 8 : upto(11) ? 11 : upto(12) ? 12 : upto(15) ? 13 : upto(16) ? 15 : 16;
    int c = upto(11) ? 8 : upto(13) ? 9 : upto(15) ? 10 : upto(17) ? 11 : upto(19) ? 12 : 13;
    while (c < kMaxWindowBits && n >= kMaxDigits / windows_for(c)) c++;  // 107 M points with 13 bits, 134 M with 16
    return c;
}

// Affine rounds (see msm_affine_pairs_kernel): tiles of kPairThreads x up to
// kPairsPerThread pairs, kPairBlocks blocks an SM.
static constexpr uint32_t kPairThreads = 128;
static constexpr uint32_t kPairBlocks = 4;
static constexpr uint32_t kPairsPerThread = 64;

// pairs a thread: whole waves of `slots` tiles of at most kPairsPerThread (on the
// device with 32 bits: pairs are below 2^31)
template <class U>
GB_RULE uint32_t pairs_per_thread(U pairs, U slots)
{
    const U all = (pairs + slots * kPairThreads - 1) / (slots * kPairThreads), per = all ? all : 1;
    const U waves = (per + kPairsPerThread - 1) / kPairsPerThread;
    return (uint32_t)((per + waves - 1) / waves);
}

// the bucket-ordered list's length when buckets are padded for the rounds
inline uint64_t padded_entries(uint64_t digits, uint64_t G, int rounds) { return digits + G * ((1u << rounds) - 1); }

// Scratch of the rounds: the two lists of 96-byte points that they go between
// (half and a quarter of the entries) and 48-byte prefix products, 48 to 72 bytes
// an entry where digits and references are 8.  Long lists go through the rounds
// in slices of kSliceEntries, whose results are collected: the two lists are a
// slice's then, and the last one's length is that of all entries >> rounds (2^24
// points, 4 rounds: 73.4 ms and 19.5 GB in one piece, 73.2 and 10.4 in 3 slices).
static constexpr uint64_t kSliceScratch = 8ull << 30;
static constexpr uint64_t kSliceEntries = kSliceScratch / 72 / 16 * 16;  // whole pairs in every round
inline uint64_t slice_entries(uint64_t entries) { return entries < kSliceEntries ? entries : kSliceEntries; }
inline bool sliced(uint64_t entries) { return entries > kSliceEntries; }
inline uint64_t rounds_scratch(uint64_t entries, int rounds, uint64_t slots)
{
    if (!rounds) return 0;
    const uint64_t slice = slice_entries(entries);
    const uint64_t prefix = 48ull * kPairThreads * slots * pairs_per_thread(slice / 2, slots);
    const uint64_t all = sliced(entries) ? 96 * ((entries >> rounds) + 1) : 0;
    if (rounds == 1 && all) return prefix + all;
    return prefix + all + 96 * (slice / 2 + 1) + (rounds > 1 ? 96 * (slice / 4 + 1) : 0);
}

// Rounds are taken while their scratch is below kRoundsScratch, and a batch of
// more than kGroupDigits digits or kGroupBuckets buckets (192 bytes each) is run
// as several, one after the other on the same scratch (16 MSMs of 2^20 points with
// 16 windows, 73 ms of work, against about 0.3 ms that a batch of its own costs).
static constexpr uint64_t kRoundsScratch = 16ull << 30;
static constexpr uint64_t kGroupDigits = 1ull << 28, kGroupBuckets = 1ull << 25;
// Batches with more scratch are not captured as graphs: a graph's memory stays
// with it between launches, and the gaps between the launches that it spares
// are less than 0.4 % of such a batch (64 MSMs of 2^10 .. 2^18 points, 3.5 GB
// of scratch: 14.40 ms as a graph, 14.45 without).
static constexpr uint64_t kGraphScratch = 4ull << 30;

// Affine rounds of a batch: as long as a round has pairs enough to fill the
// GPU (a round costs about 55 us whatever its size: product trees and one
// inversion a block) and buckets are long enough, as every bucket is padded to
// a multiple of 2^rounds; none if their scratch is more than most_scratch.
// Measured on GB300, entries and entries a bucket, and
// ms a call without rounds and with 1, 2, 3, 4 (* chosen):
//    1.0 M   80   0.61*  0.68   0.65
//    1.2 M   72   0.68   0.66*  0.66   0.74   0.79
//    2.0 M   80   1.04   0.99*  1.05
//    2.4 M   72   1.14   1.07   1.04*  1.08   1.20
//    4.7 M   72   2.07   1.84   1.77*  1.82   2.01
//    5.9 M   72                 2.20   2.19*  2.35
//   12.6 M  128   4.95   4.41   4.15   4.10*  4.16
//   16.8 M  128                 5.41   5.28*  5.37
//   16.8 M  512                 5.08   4.88   4.83*
//    4.2 M  7.8          2.48*  2.66   3.07   3.45
//    6.3 M   12          3.21   3.12*  3.59   4.01
//    7.2 M   27          3.25   3.06*  3.12   3.51
//   48 M     23         14.78  14.36* 14.94  17.18
inline int affine_rounds(uint64_t digits, double avg, uint64_t G, uint64_t slots, uint64_t most_scratch)
{
    static constexpr uint64_t pairs[4] = {9 << 16, 9 << 16, 11 << 16, 1 << 20};
    static constexpr double bucket[4] = {6, 11, 40, 192};
    int r = 0;
    while (r < 4 && digits >> (r + 1) >= pairs[r] && avg >= bucket[r] &&
           padded_entries(digits, G, r + 1) < 0x80000000ull)
        r++;
    return rounds_scratch(padded_entries(digits, G, r), r, slots) <= most_scratch ? r : 0;
}

// Entries of the bucket that an entry typically lies in: the items' means,
// weighted by their entries.  In an uneven batch the plain mean is of the many
// buckets of the small items, but the additions are in the buckets of the large
// ones: with chunks and the bound of a thread's span made for the mean, all of
// these went to the block-wide fix-up (2 MSMs of 2^16 points with 32 of 256
// points 5.8 ms, with 24 2.9; now 2.2 and 2.0).
struct typical_bucket {
    double squares = 0, sum = 0;
    void add(size_t n) { squares += (double)n * (double)n, sum += (double)n; }
    double entries(int c, bool precomputed) const
    {
        return sum > 0 ? squares / sum * (precomputed ? windows_for(c) : 1) / (double)(1u << (c - 1)) : 0;
    }
};

// Chunks that a bucket may span for one thread (or group) to add up its
// partials, kShortSpan at most: some 3 times the mean bucket's, as a longer
// chain holds up the launch (14 us an addition: 64 MSMs of 2^10 .. 2^18 points
// 14.42 ms with 6, 14.51 with 8), but what the typical bucket spans.
static constexpr uint32_t kShortSpan = 32;
inline uint32_t short_span(double mean, double typical, uint32_t L)
{
    return std::min<uint32_t>(kShortSpan, (uint32_t)std::max(6 + 3 * mean / L, 2 + 1.5 * typical / L));
}

// Sums of up to n points, `sums` of them: log2 of the groups of lanes for each,
// where a block has 32 groups.  Until the sums fill the GPU with a block each,
// all of a block's (a tree is the shortest chain); beyond, one for every two
// points, which is as short a chain and leaves no group idle (plain batches of
// 128 and 512 MSMs with windows of 8 bits, whose lines are 8 and 16 buckets: the
// reduction with its 1.2 ms of window doublings 4.42 -> 3.00 and 8.55 -> 5.07
// ms).
inline uint32_t sum_groups(uint64_t sums, uint32_t n, int sms)
{
    uint32_t log = 5;
    if (sums > 8 * (uint64_t)sms)
        while (log && (2u << log) > n) log--;
    return log;
}

// Of a batch against a context, items of at least 1 / kTableRatio of the
// context's K buckets use its table: with fewer points the plain engine and a
// small window is the less work.  But the plain MSMs are a batch of their own
// behind the other one (1.2 ms), so items down to 1 / kTableMinRatio use the
// table too, unless there are many.  Measured, ms by the table and plain:
//   K = 2^15  n = 512   x32 1.75 1.99  x40 2.42 2.15  x128 6.72 4.12  x384 19.4 7.19
//             n = 1024  x32 2.10 2.16  x40 2.58 2.39  x128 7.08 4.83  x384 20.4 9.13
//             n = 2048  x40 2.80 2.78  x64 4.00 3.66  x128 7.72 5.98  x384 22.3 12.6
//             n = 4095  x64 4.63 5.06  x96 6.94 6.94  x128 9.02 8.76  x384 25.6 20.0
//   K = 2^14  n = 256   x128 3.42 3.72  x192 5.15 5.01  x384 9.86 6.04
//             n = 512   x192 5.47 5.56  x256 7.04 6.99  x384 10.5 7.19
//             n = 1024  x192 6.15 6.50  x256 7.90 8.21  x384 11.7 9.09
//             n = 2047  x192 7.21 8.35  x256 9.24 10.6  x384 13.5 12.6
//   K = 2^12  n = 64    x384 3.11 5.40;  n = 511  x384 4.25 7.21
// The number of items up to which the table is taken; n: their mean length.
static constexpr size_t kTableRatio = 8, kTableMinRatio = 64;
inline size_t table_items(size_t K, size_t n)
{
    if (K >= (size_t)1 << 15) return 32 + (n * n >> 18);
    if (K >= (size_t)1 << 14) return 160 + n / 10;
    return SIZE_MAX;
}

// One group of a batch: how many of the items from `first` on fit kGroupDigits
// digits and kGroupBuckets buckets, one at least; size(i) points item i.
template <class F>
size_t group_items(size_t first, size_t items, F size, int c, bool precomputed)
{
    const uint64_t nwin = (uint64_t)windows_for(c), K = (uint64_t)1 << (c - 1);
    const uint64_t most = kGroupBuckets / (precomputed ? K : K * nwin);
    uint64_t digits = 0;
    size_t i = first;
    for (; i < items; i++) {
        digits += size(i) * nwin;
        if (i > first && (digits > kGroupDigits || i - first >= most)) break;
    }
    return i - first;
}

}  // namespace gb
