// BLS12-381 G1 multiexp (Pippenger) for sm_103a, and the MSM entry points
// of the C ABI (midnight-sppark-msm/src/bls12_381_g1_msm.cu:6164-6486).
//
// One engine serves every entry point: a BATCH of MSMs (one or many, of
// uneven sizes) goes through each pipeline stage in a single launch.
//   1. recode     : Montgomery -> canonical, signed c-bit digits per window
//                   (digit in [-2^(c-1), 2^(c-1)], carry into the next window)
//   2. histogram  : per-block shared-memory counts of bucket keys
//   3. column scan: per-key prefix over the blocks of its segment + totals
//   4. key scan   : exclusive scan of totals -> bucket start offsets
//   5. scatter    : (bucket, point) pairs placed in bucket order
//   6. accumulate : each thread sums L consecutive sorted entries into XYZZ
//                   accumulators (fixed work per thread whatever the bucket
//                   sizes), writing finished buckets directly and chunk-edge
//                   partials aside
//   7. fix-up     : buckets spanning chunks add their partials
//                   (large batches: affine rounds before it)
//   8. reduce     : sum_k (k+1) B_k per segment, by line and bit sums, then
//                   per MSM the window combination; a few MSMs' last dependent
//                   steps are the host's.
// Very large batches go through the stages in groups (gb_msm_rules.h).
//
// A "segment" owns 2^(c-1) buckets.  Two modes:
//   * precomputed (MSM contexts, whose bases are fixed): context creation
//     stores 2^(c*j) P_i for every window j, so each MSM is ONE segment and
//     needs no window combination;
//   * plain (bases passed per call): each (MSM, window) is a segment and the
//     windows are combined by Horner's rule.
// Both decode a digit's point as point_base + (d / n) * stride + d % n.
#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <atomic>
#include <tuple>
#include <set>
#include <mutex>
#include <initializer_list>
#include <vector>

#include "gb_inv_warp.cuh"
#include "gb_host_fp.h"
#include "gb_msm_rules.h"
#include "gb_runtime.cuh"

namespace gb {

static constexpr uint32_t kZeroDigit = 0xffffffffu;

static int default_acc_variant()
{
    const char *e = getenv("GB_MSM_ACC_VARIANT");
    if (e && e[0] >= '0' && e[0] <= '2') return e[0] - '0';
    return 1;  // 256 threads, 2 blocks per SM: the fastest on GB300 at n = 2^20
}

// one MSM of a batch (host view)
struct msm_item {
    const fr_t *scalars;  // device pointer, n values
    size_t n;
    size_t point_base;    // first base of this MSM in table row 0
};

// per-segment and per-sort-block descriptors (device view)
struct seg_desc {
    uint64_t digit_off;   // first digit of the segment
    uint32_t len;         // digits in the segment
    uint32_t n;           // points of the segment's MSM (digit d -> window d / n, point d % n)
    uint64_t point_base;  // base index of the MSM's first point in table row 0
    uint32_t blk0, nblk;  // sort blocks of the segment
};
struct blk_desc {
    uint32_t seg;
    uint32_t lo, hi;      // digit range within the segment
};
struct item_desc {
    const fr_t *scalars;
    uint64_t point_prefix;  // sum of n over earlier items (thread -> item map)
    uint64_t digit_base;    // digits of the item start here: [window][n]
    uint32_t n;
};

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------

__device__ __forceinline__ affine_t load_affine(const affine_t *pts, uint32_t idx)
{
    const uint4 *src = reinterpret_cast<const uint4 *>(pts + idx);
    affine_t r;
    uint4 *dst = reinterpret_cast<uint4 *>(&r);
#pragma unroll
    for (int i = 0; i < 6; i++) dst[i] = __ldg(src + i);
    return r;
}

// The canonical value of a Montgomery-form scalar s < r (s R^-1 mod r):
// Montgomery reduction alone (the product by 1 without its a * b rows),
// 8 steps of t = (t + m r) / 2^32 with m = -t0 (r's lowest limb is 1).  The
// result is below r for s < r, and the final subtraction covers s < R.
// The scalar is read with two 16-byte loads when it is 16-byte aligned.
__device__ __forceinline__ fr_t scalar_canonical(const fr_t *p)
{
    fr_t a;
    if (((uintptr_t)p & 15u) == 0) {
        const uint4 lo = __ldg(reinterpret_cast<const uint4 *>(p)), hi = __ldg(reinterpret_cast<const uint4 *>(p) + 1);
        a.v[0] = lo.x, a.v[1] = lo.y, a.v[2] = lo.z, a.v[3] = lo.w;
        a.v[4] = hi.x, a.v[5] = hi.y, a.v[6] = hi.z, a.v[7] = hi.w;
    } else {
        a = *p;
    }
    uint32_t t[9];
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] = a.v[i];
    t[8] = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint32_t m = 0u - t[0];
        uint64_t c = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint64_t v = (uint64_t)m * FrCfg::mod(j) + t[j] + c;
            t[j] = (uint32_t)v;
            c = v >> 32;
        }
        const uint64_t top = (uint64_t)t[8] + c;
#pragma unroll
        for (int j = 0; j < 7; j++) t[j] = t[j + 1];
        t[7] = (uint32_t)top;
        t[8] = (uint32_t)(top >> 32);
    }
    fr_t r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = t[i];
    fr_t::reduce_once(r.v, t[8]);
    return r;
}

// 1. recode: for item m, point i, window j: digits[base_m + j * n_m + i] =
//    (|digit| - 1) | sign << 31, or kZeroDigit.  One instance per window
//    size, so the windows unroll and the scalar's limbs stay in registers
//    (with the window a run-time value they were indexed in local memory).
template <int C>
__global__ void msm_recode_kernel(const item_desc *__restrict__ items, uint32_t nitems, uint64_t total,
                                  uint32_t *__restrict__ digits)
{
    constexpr int NWIN = windows_for(C);
    constexpr uint32_t half = 1u << (C - 1);
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    uint32_t lo = 0, hi = nitems;  // last item with point_prefix <= t
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (items[mid].point_prefix <= t) lo = mid;
        else hi = mid;
    }
    const item_desc it = items[lo];
    const uint64_t i = t - it.point_prefix;
    const fr_t s = scalar_canonical(it.scalars + i);
    uint32_t carry = 0;
    uint32_t *out = digits + it.digit_base + i;
#pragma unroll
    for (int j = 0; j < NWIN; j++) {
        const int bit = window_offset(C, j);
        const uint32_t mask = (1u << window_bits(C, j)) - 1;
        const int limb = bit >> 5, off = bit & 31;
        const uint32_t l0 = limb < 8 ? s.v[limb < 8 ? limb : 7] : 0;
        const uint32_t l1 = limb + 1 < 8 ? s.v[limb + 1 < 8 ? limb + 1 : 7] : 0;
        uint32_t raw = (uint32_t)((((uint64_t)l1 << 32) | l0) >> off) & mask;
        raw += carry;
        uint32_t d;
        if (raw == 0) {
            carry = 0;
            d = kZeroDigit;
        } else if (raw <= half) {
            carry = 0;
            d = raw - 1;
        } else {
            carry = 1;
            const uint32_t mag = (1u << C) - raw;  // digit = raw - 2^c < 0
            d = mag == 0 ? kZeroDigit : ((mag - 1) | 0x80000000u);
        }
        out[(uint64_t)j * it.n] = d;
    }
}

static void launch_recode(const item_desc *items, uint32_t nitems, uint64_t total, int c, uint32_t *digits,
                          cudaStream_t s)
{
    const unsigned grid = (unsigned)((total + 255) / 256);
    switch (c) {
    case 8: msm_recode_kernel<8><<<grid, 256, 0, s>>>(items, nitems, total, digits); break;
    case 9: msm_recode_kernel<9><<<grid, 256, 0, s>>>(items, nitems, total, digits); break;
    case 10: msm_recode_kernel<10><<<grid, 256, 0, s>>>(items, nitems, total, digits); break;
    case 11: msm_recode_kernel<11><<<grid, 256, 0, s>>>(items, nitems, total, digits); break;
    case 12: msm_recode_kernel<12><<<grid, 256, 0, s>>>(items, nitems, total, digits); break;
    case 13: msm_recode_kernel<13><<<grid, 256, 0, s>>>(items, nitems, total, digits); break;
    case 14: msm_recode_kernel<14><<<grid, 256, 0, s>>>(items, nitems, total, digits); break;
    case 15: msm_recode_kernel<15><<<grid, 256, 0, s>>>(items, nitems, total, digits); break;
    case 16: msm_recode_kernel<16><<<grid, 256, 0, s>>>(items, nitems, total, digits); break;
    default: throw cuda_error((int)cudaErrorInvalidValue, "MSM window size outside 8..16");
    }
    GB_CHECK_LAUNCH();
}

// control words of a batch, zeroed by its first kernel that has them
enum { CTL_LONGS = 0, CTL_DONE = 1, CTL_WORDS = 2 };  // long buckets so far; column blocks done

// 2. per-block histograms: hist[b][k]
__global__ void msm_hist_kernel(const uint32_t *__restrict__ digits, const seg_desc *__restrict__ segs,
                                const blk_desc *__restrict__ blks, uint32_t K, uint32_t *__restrict__ hist,
                                uint32_t *__restrict__ ctl)
{
    extern __shared__ uint32_t sh[];
    if (blockIdx.x == 0 && threadIdx.x < CTL_WORDS) ctl[threadIdx.x] = 0;
    const blk_desc bd = blks[blockIdx.x];
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) sh[k] = 0;
    __syncthreads();
    const uint32_t *d = digits + segs[bd.seg].digit_off;
    for (uint32_t i = bd.lo + threadIdx.x; i < bd.hi; i += blockDim.x) {
        uint32_t v = d[i];
        if (v != kZeroDigit) atomicAdd(&sh[v & (K - 1)], 1u);
    }
    __syncthreads();
    uint32_t *out = hist + (size_t)blockIdx.x * K;
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) out[k] = sh[k];
}

// 3. per global key g = seg * K + k: exclusive prefix over the segment's
//    blocks (in place in hist) and the total into counts[g], rounded up to a
//    multiple of pad + 1 (a power of two; the places past the total hold
//    kNoPoint).  The sum of a key without entries is infinity (all zero) here;
//    the accumulation writes all others.  With few keys (starts given, blocks
//    of 1024 threads), the last block to finish also scans the counts: one
//    launch in place of four and two copies, 12 us of the 2^10-point MSM's
//    200.
static constexpr uint32_t kScanHere = 16 * 1024;  // keys at most

__global__ void __launch_bounds__(1024)
    msm_colscan_kernel(uint32_t *__restrict__ hist, const seg_desc *__restrict__ segs, uint32_t K, uint32_t G,
                       uint32_t pad, uint32_t *counts, xyzz_t *__restrict__ buckets, uint32_t *__restrict__ starts,
                       uint32_t *ctl)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < G) {
        const seg_desc sd = segs[g / K];
        const uint32_t k = g % K;
        uint32_t run = 0;
        uint32_t *col = hist + (size_t)sd.blk0 * K + k;
        uint32_t w = 0;
        // batches of 16 independent loads keep the column walk off the latency path
        for (; w + 16 <= sd.nblk; w += 16) {
            uint32_t v[16];
#pragma unroll
            for (int u = 0; u < 16; u++) v[u] = col[(size_t)(w + u) * K];
#pragma unroll
            for (int u = 0; u < 16; u++) {
                col[(size_t)(w + u) * K] = run;
                run += v[u];
            }
        }
        for (; w < sd.nblk; w++) {
            uint32_t v = col[(size_t)w * K];
            col[(size_t)w * K] = run;
            run += v;
        }
        counts[g] = (run + pad) & ~pad;
        if (!run) buckets[g] = xyzz_t::inf();
    }
    if (!starts) return;
    __shared__ uint32_t part[16 * 32];
    __shared__ bool last;
    __threadfence();  // this thread's count before the block's arrival
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&ctl[CTL_DONE], 1u) + 1 == gridDim.x;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // strip j holds keys 1024 j ..: a warp's scan, the warps' totals, the strips'
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t v[16], incl[16];
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const uint32_t i = j * 1024u + threadIdx.x;
        v[j] = i < G ? __ldcg(counts + i) : 0u;
    }
#pragma unroll
    for (int j = 0; j < 16; j++) {
        incl[j] = v[j];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, incl[j], off);
            if (lane >= (uint32_t)off) incl[j] += x;
        }
        if (lane == 31) part[j * 32 + warp] = incl[j];
    }
    __syncthreads();
    if (warp == 0) {
        // lane l: the 16 totals 16 l .. 16 l + 15, in key order
        uint32_t sum = 0, own[16];
#pragma unroll
        for (int j = 0; j < 16; j++) {
            own[j] = part[lane * 16 + j];
            sum += own[j];
        }
        uint32_t run = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, run, off);
            if (lane >= (uint32_t)off) run += x;
        }
        if (lane == 31) starts[G] = run;
        run -= sum;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            part[lane * 16 + j] = run;
            run += own[j];
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const uint32_t i = j * 1024u + threadIdx.x;
        if (i < G) starts[i] = part[j * 32 + warp] + incl[j] - v[j];
    }
}

// 4. exclusive scan of counts[0..G) into starts[0..G], starts[G] = total:
//    tile sums, a one-block scan of the tile sums, then the tiles themselves
static constexpr uint32_t kScanTileU32 = 4096;

__global__ void u32_tile_sum_kernel(const uint32_t *__restrict__ in, uint32_t n, uint32_t *__restrict__ sums)
{
    __shared__ uint32_t sh[256];
    uint32_t base = blockIdx.x * kScanTileU32;
    uint32_t s = 0;
    for (uint32_t i = base + threadIdx.x; i < min(base + kScanTileU32, n); i += 256) s += in[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t off = 128; off; off >>= 1) {
        if (threadIdx.x < off) sh[threadIdx.x] += sh[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = sh[0];
}

// exclusive scan in place of up to 1024 * 64 values with one block
__global__ void u32_small_scan_kernel(uint32_t *__restrict__ v, uint32_t n)
{
    __shared__ uint32_t part[1024];
    const uint32_t T = blockDim.x;
    const uint32_t per = (n + T - 1) / T;
    const uint32_t lo = threadIdx.x * per, hi = min(lo + per, n);
    uint32_t s = 0;
    for (uint32_t i = lo; i < hi; i++) s += v[i];
    part[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t off = 1; off < T; off <<= 1) {
        uint32_t x = threadIdx.x >= off ? part[threadIdx.x - off] : 0;
        __syncthreads();
        part[threadIdx.x] += x;
        __syncthreads();
    }
    uint32_t run = threadIdx.x ? part[threadIdx.x - 1] : 0;
    for (uint32_t i = lo; i < hi; i++) {
        uint32_t x = v[i];
        v[i] = run;
        run += x;
    }
}

// out[i] = tile prefix + exclusive prefix within the tile
__global__ void u32_tile_scan_kernel(const uint32_t *__restrict__ in, uint32_t n, const uint32_t *__restrict__ tile_pre,
                                     uint32_t *__restrict__ out)
{
    __shared__ uint32_t part[256];
    const uint32_t base = blockIdx.x * kScanTileU32;
    const uint32_t per = kScanTileU32 / 256;
    const uint32_t lo = base + threadIdx.x * per;
    uint32_t s = 0;
    for (uint32_t i = lo; i < min(lo + per, n); i++) s += in[i];
    part[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t off = 1; off < 256; off <<= 1) {
        uint32_t x = threadIdx.x >= off ? part[threadIdx.x - off] : 0;
        __syncthreads();
        part[threadIdx.x] += x;
        __syncthreads();
    }
    uint32_t run = tile_pre[blockIdx.x] + (threadIdx.x ? part[threadIdx.x - 1] : 0);
    for (uint32_t i = lo; i < min(lo + per, n); i++) {
        out[i] = run;
        run += in[i];
    }
}

// 5. scatter into bucket order: sorted[pos] = point_ref | sign << 31
__global__ void msm_scatter_kernel(const uint32_t *__restrict__ digits, const seg_desc *__restrict__ segs,
                                   const blk_desc *__restrict__ blks, uint32_t K, uint64_t stride,
                                   const uint32_t *__restrict__ hist, const uint32_t *__restrict__ starts,
                                   uint32_t *__restrict__ sorted)
{
    extern __shared__ uint32_t cursor[];
    const blk_desc bd = blks[blockIdx.x];
    const seg_desc sd = segs[bd.seg];
    const uint32_t *h = hist + (size_t)blockIdx.x * K;
    const uint32_t *st = starts + (size_t)bd.seg * K;
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) cursor[k] = st[k] + h[k];
    __syncthreads();
    const uint32_t *d = digits + sd.digit_off;
    for (uint32_t i = bd.lo + threadIdx.x; i < bd.hi; i += blockDim.x) {
        uint32_t v = d[i];
        if (v == kZeroDigit) continue;
        uint32_t pos = atomicAdd(&cursor[v & (K - 1)], 1u);
        uint64_t ref = sd.point_base + (uint64_t)(i / sd.n) * stride + (i % sd.n);
        sorted[pos] = (uint32_t)ref | (v & 0x80000000u);
    }
}

// 5b. affine rounds.  Adding two affine points takes one inversion, 2 products
//     and 1 squaring, and Montgomery's trick shares one inversion among many
//     additions for 3 products each: 5 products and a squaring against the 8
//     and 2 of a mixed addition into XYZZ.  A round adds the entries 2i and
//     2i + 1 of the bucket-ordered list and leaves a list of half the length:
//     the buckets' starts are multiples of 2^rounds (kNoPoint fills them up),
//     so no pair crosses a bucket.  A block's tile is 128 x per_thread pairs:
//     each thread multiplies up its denominators, keeping the running products
//     in `prefix`, the block's 128 totals go up a product tree, one warp
//     inverts the root, the inverses come down, and each thread walks back
//     through its pairs.
//
//     What bounds it: the multiply-add pipe, 82 % busy between inversions
//     (about 8000 of its cycles a warp and pair, 6800 of them products), with
//     four blocks an SM.  The first round of a 2^20-point MSM (8.4 M pairs)
//     takes 2.2 ms, 0.27 ns a pair, against 0.33 ns a mixed addition.
//     Measured and not kept: an inversion per warp instead of per block (no
//     barriers, but four times the inversions' instructions: 0.6 ms more at
//     2^20), tiles of different lengths so that an SM's blocks invert at
//     different times (60 us more a round), 5 or 6 blocks an SM (spills).  The
//     points come through shared memory by asynchronous copies that go
//     through L1 (a 96-byte point is three sectors, each fetched by two 16-byte
//     copies): two pairs ahead on the way up, one on the way back, 2 % better
//     than plain loads; past L1 they were 8 % worse.
static constexpr uint32_t kNoPoint = 0xffffffffu;

__device__ __forceinline__ void store_words8(void *p, const uint32_t *w)
{
    asm volatile("st.global.v8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "l"(p)
                 : "memory");
}

// the products of a pair, inlined: the two loops hold six copies in all
// (45 KB), and the moves around a call cost more than fetching them
__device__ __forceinline__ fp_t mul_here(const fp_t &a, const fp_t &b)
{
    fp_t r;
#if defined(__CUDA_ARCH__)
    fp_mul_rows(r.v, a.v, b.v);
#endif
    return r;
}

__device__ __forceinline__ fp_t sqr_here(const fp_t &a)
{
    fp_t r;
#if defined(__CUDA_ARCH__)
    fp_sqr_rows(r.v, a.v);
#endif
    return r;
}

// a thread's 16-byte slots in shared memory, one a 128-thread row
struct pair_stage {
    uint4 *slot;  // the thread's place in row 0
    __device__ __forceinline__ void copy(uint32_t row, const void *src, uint32_t count) const
    {
#pragma unroll
        for (uint32_t c = 0; c < count; c++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(slot + (row + c) * kPairThreads)),
                         "l"((const uint4 *)src + c)
                         : "memory");
    }
    __device__ __forceinline__ void copy_strided(uint32_t row, const uint4 *src) const
    {
#pragma unroll
        for (uint32_t c = 0; c < 3; c++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(slot + (row + c) * kPairThreads)),
                         "l"(src + c * kPairThreads)
                         : "memory");
    }
    static __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
    template <int N>
    static __device__ __forceinline__ void wait()
    {
        asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
    }
    __device__ __forceinline__ fp_t value(uint32_t row) const
    {
        fp_t v;
        uint4 *d = reinterpret_cast<uint4 *>(&v);
#pragma unroll
        for (int c = 0; c < 3; c++) d[c] = slot[(row + c) * kPairThreads];
        return v;
    }
};

// a list's pair i: signed references into the bases, or the points themselves
template <bool REFS>
struct pair_refs {
    uint2 r;
    __device__ __forceinline__ void load(const uint32_t *refs, uint64_t i, bool in)
    {
        if (REFS) r = in ? reinterpret_cast<const uint2 *>(refs)[i] : make_uint2(kNoPoint, kNoPoint);
    }
    __device__ __forceinline__ bool none(int side) const { return REFS && (side ? r.y : r.x) == kNoPoint; }
    __device__ __forceinline__ bool neg(int side) const { return REFS && (side ? r.y : r.x) >> 31; }
    __device__ __forceinline__ const affine_t *point(const affine_t *points, uint64_t i, int side) const
    {
        if (!REFS) return points + 2 * i + side;
        return points + (none(side) ? 0u : (side ? r.y : r.x) & 0x7fffffffu);
    }
    __device__ __forceinline__ fp_t y(const affine_t *points, uint64_t i, int side) const
    {
        const fp_t v = point(points, i, side)->y;
        return neg(side) ? -v : v;
    }
};

enum { PAIR_ADD, PAIR_FIRST, PAIR_SECOND, PAIR_DOUBLE, PAIR_INF };

// how the pair's points are added, and the denominator of the slope (one
// where there is none); the point at infinity is all zero, so the second
// coordinates are read only where a first one is zero or both are equal
template <bool REFS>
__device__ __forceinline__ int pair_kind(const pair_refs<REFS> &ref, const affine_t *points, uint64_t i,
                                         const fp_t &xa, const fp_t &xb, fp_t &den)
{
    den = xb - xa;
    int kind = PAIR_ADD;
    if (ref.none(1) || (xb.is_zero() && ref.y(points, i, 1).is_zero())) {
        kind = PAIR_FIRST;
    } else if (ref.none(0) || (xa.is_zero() && ref.y(points, i, 0).is_zero())) {
        kind = PAIR_SECOND;
    } else if (den.is_zero()) {
        const fp_t ya = ref.y(points, i, 0);
        kind = ya == ref.y(points, i, 1) && !ya.is_zero() ? PAIR_DOUBLE : PAIR_INF;
        den = ya.dbl();
    }
    if (kind != PAIR_ADD && kind != PAIR_DOUBLE) den = fp_t::one();
    return kind;
}

template <bool REFS>
__global__ void __launch_bounds__(kPairThreads, kPairBlocks)
    msm_affine_pairs_kernel(const uint32_t *__restrict__ refs, const affine_t *__restrict__ points,
                            affine_t *__restrict__ out, const uint32_t *__restrict__ entries, uint32_t lo,
                            uint32_t hi, int round, uint32_t most_per_thread, uint4 *__restrict__ prefix)
{
    __shared__ fp_t node[2 * kPairThreads];  // product tree: root 1, leaves 128 ..
    __shared__ uint4 stage_mem[15 * kPairThreads];
    const uint32_t tid = threadIdx.x;
    const pair_stage stage{stage_mem + tid};
    // of the list's entries lo .. hi - 1 those that there are
    const uint32_t end = *entries;
    const uint64_t pairs = (min(end, hi) - min(end, lo)) >> round;
    // the host knows a bound of the pairs only: of scalars that are zero for the
    // most part (2^20 of them, one in ten not: 1.98 -> 1.34 ms) the tiles are
    // shorter, so that every block has one
    const uint32_t per_thread = min(most_per_thread, pairs_per_thread((uint32_t)pairs, gridDim.x));
    const uint64_t tile = (uint64_t)kPairThreads * per_thread;
    uint4 *pre = prefix + (uint64_t)blockIdx.x * per_thread * 3 * kPairThreads + tid;
    for (uint64_t base = blockIdx.x * tile + tid; base - tid < pairs; base += gridDim.x * tile) {
        const int turns =
            (int)min((uint64_t)per_thread, (pairs - (base - tid) + kPairThreads - 1) / kPairThreads);
        auto at = [&](int k) { return base + (uint64_t)(uint32_t)k * kPairThreads; };
        auto in = [&](int k) { return k >= 0 && k < turns && at(k) < pairs; };

        // up: the running product before each pair, x coordinates two ahead
        // (rows 0..5 and 6..11)
        pair_refs<REFS> r0, r1, r2;
        r0.load(refs, at(0), in(0));
        r1.load(refs, at(1), in(1));
        r2.load(refs, at(2), in(2));
        auto fetch_x = [&](const pair_refs<REFS> &r, int k) {
            if (in(k)) {
                const uint32_t row = k & 1 ? 6 : 0;
                stage.copy(row, r.point(points, at(k), 0), 3);
                stage.copy(row + 3, r.point(points, at(k), 1), 3);
            }
            stage.commit();
        };
        fetch_x(r0, 0);
        fetch_x(r1, 1);
        fp_t run = fp_t::one();
        for (int k = 0; k < turns; k++) {
            const uint4 *w = reinterpret_cast<const uint4 *>(&run);
#pragma unroll
            for (int c = 0; c < 3; c++) pre[(k * 3 + c) * kPairThreads] = w[c];
            stage.wait<1>();
            fp_t den = fp_t::one();
            if (in(k)) {
                const uint32_t row = k & 1 ? 6 : 0;
                pair_kind<REFS>(r0, points, at(k), stage.value(row), stage.value(row + 3), den);
            }
            r0 = r1, r1 = r2;
            fetch_x(r1, k + 2);
            r2.load(refs, at(k + 3), in(k + 3));
            run = mul_here(run, den);
        }
        __threadfence();  // the prefixes are read back by asynchronous copies

        // down: all of a pair but its sign, one ahead (a 0..5, b 6..11, its
        // prefix 12..14)
        auto fetch = [&](const pair_refs<REFS> &r, int k) {
            if (in(k)) {
                stage.copy(0, r.point(points, at(k), 0), 6);
                stage.copy(6, r.point(points, at(k), 1), 6);
                stage.copy_strided(12, pre + k * 3 * kPairThreads);
            }
            stage.commit();
        };
        stage.wait<0>();
        r0.load(refs, at(turns - 1), in(turns - 1));
        r1.load(refs, at(turns - 2), in(turns - 2));
        fetch(r0, turns - 1);

        __syncthreads();  // the previous tile's tree is read
        node[kPairThreads + tid] = run;
        __syncthreads();
        if (tid < 64) node[64 + tid] = node[128 + 2 * tid] * node[129 + 2 * tid];
        __syncthreads();
        fp_t inv;
        if (tid < 32) {
            for (uint32_t n = 32; n > 0; n >>= 1) {
                if (tid < n) inv = node[2 * (n + tid)] * node[2 * (n + tid) + 1];
                if (tid < n) node[n + tid] = inv;
                __syncwarp();
            }
            inv = inverse_warp<FpCfg>(node + 1);
            __syncwarp();
            if (tid == 0) node[1] = inv;
            __syncwarp();
            // a child's inverse: its parent's times its sibling
            for (uint32_t n = 2; n <= 32; n <<= 1) {
                if (tid < n) inv = node[(n + tid) >> 1] * node[(n + tid) ^ 1];
                __syncwarp();
                if (tid < n) node[n + tid] = inv;
                __syncwarp();
            }
        }
        __syncthreads();
        if (tid < 64) inv = node[(64 + tid) >> 1] * node[(64 + tid) ^ 1];
        __syncthreads();
        if (tid < 64) node[64 + tid] = inv;
        __syncthreads();
        inv = node[(128 + tid) >> 1] * node[(128 + tid) ^ 1];

        for (int k = turns; k-- > 0;) {
            stage.wait<0>();
            const uint64_t i = at(k);
            fp_t xa = fp_t::zero(), num = xa, ya = xa, di = xa;
            int kind = PAIR_INF;
            if (in(k)) {
                di = mul_here(inv, stage.value(12));
                xa = stage.value(0);
                const fp_t xb = stage.value(6);
                fp_t den;
                kind = pair_kind<REFS>(r0, points, i, xa, xb, den);
                inv = mul_here(inv, den);
                ya = stage.value(3);
                if (r0.neg(0)) ya = -ya;
                num = stage.value(9);
                if (r0.neg(1)) num = -num;
            }
            affine_t r;
            if (kind == PAIR_SECOND) {
                r.x = stage.value(6), r.y = num;
            } else if (kind == PAIR_FIRST && !r0.none(0)) {
                r.x = xa, r.y = ya;
            } else {
                r = affine_t::inf();
            }
            if (kind == PAIR_ADD) {
                num = num - ya;
                r.x = stage.value(6);
            } else if (kind == PAIR_DOUBLE) {
                num = sqr_here(xa);
                num = num.dbl() + num;
                r.x = xa;
            }
            r0 = r1;
            fetch(r0, k - 1);
            r1.load(refs, at(k - 2), in(k - 2));
            if (kind == PAIR_ADD || kind == PAIR_DOUBLE) {
                const fp_t s = mul_here(num, di);
                r.x = sqr_here(s) - xa - r.x;
                r.y = mul_here(s, xa - r.x) - ya;
            }
            if (i < pairs) {
                const uint32_t *o = reinterpret_cast<const uint32_t *>(&r);
#pragma unroll
                for (int c = 0; c < 3; c++) store_words8(reinterpret_cast<uint32_t *>(out + i) + 8 * c, o + 8 * c);
            }
        }
        stage.wait<0>();
    }
}

// starts of the lists after the affine rounds
__global__ void msm_shift_starts_kernel(const uint32_t *__restrict__ starts, uint32_t n, int rounds,
                                        uint32_t *__restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = starts[i] >> rounds;
}

// 6. accumulate L sorted entries per thread.  Instantiated for several
//    (block size, min blocks per SM) pairs: the register cap trades
//    occupancy against spills, and the plan picks one.
//    With REFS the entries are references into the bases, without it (after
//    affine rounds) the points themselves.
template <int BLOCK, int MINB, bool REFS = true>
__global__ void __launch_bounds__(BLOCK, MINB) msm_accumulate_kernel(
    const uint32_t *__restrict__ sorted, const uint32_t *__restrict__ starts, uint32_t G, uint32_t L,
    size_t nchunks, const affine_t *__restrict__ points, xyzz_t *__restrict__ buckets,
    xyzz_t *__restrict__ head, xyzz_t *__restrict__ tail, uint32_t *__restrict__ open_bucket)
{
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nchunks) return;
    const uint32_t T = starts[G];
    const uint64_t lo = (uint64_t)t * L;
    if (lo >= T) return;
    const uint64_t hi = min((uint64_t)T, lo + L);
    // largest g with starts[g] <= lo; starts[G] = T > lo
    uint32_t a = 0, b = G;
    while (b - a > 1) {
        uint32_t mid = (a + b) >> 1;
        if (starts[mid] <= lo) a = mid;
        else b = mid;
    }
    uint32_t g = a;
    uint32_t gend = starts[g + 1];
    bool started_here = starts[g] >= lo;
    bool open = false;
    xyzz_t acc = xyzz_t::inf();
    for (uint64_t pos = lo; pos < hi; pos++) {
        if (REFS) {
            uint32_t ref = sorted[pos];
            affine_t p = load_affine(points, ref & 0x7fffffffu);
            acc.add_affine(p, (ref >> 31) != 0);
        } else {
            acc.add_affine(load_affine(points, (uint32_t)pos), false);
        }
        open = true;
        if (pos + 1 == gend) {
            if (started_here) buckets[g] = acc;
            else head[t] = acc;
            acc = xyzz_t::inf();
            open = false;
            started_here = true;
            g++;
            while (g < G && starts[g + 1] == starts[g]) g++;
            gend = g < G ? starts[g + 1] : T;
        }
    }
    if (open) {
        tail[t] = acc;
        if (open_bucket && started_here) open_bucket[t] = g;
    }
}

// 6'. The same with two lanes a chunk, for batches too small to fill the GPU
//     with a thread a chunk: the 10 products of a mixed addition are 5 levels of
//     two that do not depend on each other, so an addition takes half as long
//     and its products cost the same.  Of the running point the even lane has
//     X (and a copy of Y) and ZZ, the odd one Y (and X) and ZZZ; of an entry the
//     even lane reads x, the odd one y.  A warp's lanes go through all L steps
//     together, so that the exchanges have all of them; what does not hold for
//     a pair (no entry left, nothing summed yet) is selected away.
__device__ __forceinline__ fp_t pair_swap(const fp_t &a)
{
    fp_t r;
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = __shfl_xor_sync(0xffffffffu, a.v[i], 1);
    return r;
}

__device__ __forceinline__ fp_t pair_pick(bool odd, const fp_t &o, const fp_t &e)
{
    fp_t r;
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = odd ? o.v[i] : e.v[i];
    return r;
}

static constexpr uint32_t kPairChunks = 64, kPairSm = 3;  // a block's chunks, an SM's blocks

__global__ void __launch_bounds__(2 * kPairChunks, kPairSm) msm_accumulate_pair_kernel(
    const uint32_t *__restrict__ sorted, const uint32_t *__restrict__ starts, uint32_t G, uint32_t L,
    size_t nchunks, const affine_t *__restrict__ points, xyzz_t *__restrict__ buckets,
    xyzz_t *__restrict__ head, xyzz_t *__restrict__ tail, uint32_t *__restrict__ open_bucket)
{
    const size_t t = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 2;
    const bool odd = threadIdx.x & 1u;
    const uint32_t T = starts[G];
    uint64_t lo = (uint64_t)t * L, hi = lo + L;
    if (t >= nchunks || lo >= T) lo = hi = 0;
    hi = min((uint64_t)T, hi);
    uint32_t g = 0, gend = 0;
    bool started_here = false;
    if (lo < hi) {
        // largest g with starts[g] <= lo; starts[G] = T > lo
        uint32_t b = G;
        while (b - g > 1) {
            const uint32_t mid = (g + b) >> 1;
            if (starts[mid] <= lo) g = mid;
            else b = mid;
        }
        gend = starts[g + 1];
        started_here = starts[g] >= lo;
    }
    auto load = [&](uint64_t pos) {
        fp_t q = fp_t::zero();
        if (pos >= hi) return q;
        const uint32_t ref = sorted[pos];
        const uint4 *src = reinterpret_cast<const uint4 *>(points + (ref & 0x7fffffffu)) + (odd ? 3 : 0);
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const uint4 w = __ldg(src + i);
            q.v[4 * i] = w.x, q.v[4 * i + 1] = w.y, q.v[4 * i + 2] = w.z, q.v[4 * i + 3] = w.w;
        }
        if (odd && (ref >> 31)) q = -q;
        return q;
    };
    // the lane's coordinate, the other lane's, and its denominator (ZZ or ZZZ)
    fp_t own = fp_t::zero(), other = fp_t::zero(), den = fp_t::zero();
    bool empty = true, open = false;
    auto store = [&](xyzz_t *to) {
        fp_t *f = reinterpret_cast<fp_t *>(to) + (odd ? 1 : 0);
        f[0] = empty ? fp_t::zero() : own;
        f[2] = empty ? fp_t::zero() : den;
    };
    fp_t next = load(lo);
    for (uint32_t i = 0; i < L; i++) {
        const uint64_t pos = lo + i;
        const fp_t q = next;
        next = load(pos + 1);
        const bool valid = pos < hi, zero = q.is_zero();
        // every lane of the warp takes part in an exchange: none stands behind
        // a condition of its own
        const bool zero2 = __shfl_xor_sync(0xffffffffu, (int)zero, 1);
        const bool take = valid && !(zero && zero2);  // a base at infinity adds nothing
        const fp_t q2 = pair_swap(q);
        if (__any_sync(0xffffffffu, take && !empty)) {
            const fp_t d = q * den - own;  // P | R
            const bool dz = d.is_zero(), dz2 = __shfl_xor_sync(0xffffffffu, (int)dz, 1);
            const fp_t e = d.sqr(), f = pair_swap(e);                               // PP | RR and the other
            const fp_t h = pair_pick(odd, other, d) * pair_pick(odd, f, e);         // P PP | X PP
            const fp_t h2 = pair_swap(h);
            const fp_t ppp = pair_pick(odd, h2, h), xpp = pair_pick(odd, h, h2);
            const fp_t x3 = pair_pick(odd, e, f) - ppp - xpp.dbl();
            const fp_t k = pair_pick(odd, d, other) * pair_pick(odd, xpp - x3, ppp);  // Y PPP | R (X PP - X3)
            const fp_t k2 = pair_swap(k);
            const fp_t y3 = pair_pick(odd, k, k2) - pair_pick(odd, k2, k);
            const fp_t den3 = den * pair_pick(odd, ppp, e);
            const bool same_x = odd ? dz2 : dz, same_y = odd ? dz : dz2;
            if (take && !empty) {
                if (!same_x) {
                    own = pair_pick(odd, y3, x3);
                    other = pair_pick(odd, x3, y3);
                    den = den3;
                } else if (same_y) {
                    const xyzz_t v = xyzz_t::dbl_affine(pair_pick(odd, q2, q), pair_pick(odd, q, q2));
                    own = pair_pick(odd, v.y, v.x);
                    other = pair_pick(odd, v.x, v.y);
                    den = pair_pick(odd, v.zzz, v.zz);
                    empty = v.zz.is_zero();
                } else {
                    empty = true;
                }
            } else if (take) {
                own = q, other = q2, den = fp_t::one();
                empty = false;
            }
        } else if (take) {
            own = q, other = q2, den = fp_t::one();
            empty = false;
        }
        if (valid) {
            open = true;
            if (pos + 1 == gend) {
                store(started_here ? buckets + g : head + t);
                empty = true;
                open = false;
                started_here = true;
                g++;
                while (g < G && starts[g + 1] == starts[g]) g++;
                gend = g < G ? starts[g + 1] : T;
            }
        }
        __syncwarp();
    }
    if (open) {
        store(tail + t);
        if (open_bucket && started_here && !odd) open_bucket[t] = g;
    }
}

// 7. buckets spanning several chunks.  A bucket spanning a few
//    chunks is summed by its own thread; longer ones (skewed digits: structured
//    scalars, the carry out of scalars below 2^64) are appended to `longs` for
//    msm_fixup_long_kernel.  One thread a bucket, or, where buckets are shorter
//    than chunks and most span none, one a chunk, so that the lanes that add
//    lie closer together.  Measured, 64 MSMs of 2^10 .. 2^18 points with 2^15
//    buckets each 1.60 -> 0.47 ms (chunks of 8 waves at most among it), 20 of
//    2^10 .. 2^13 0.77 -> 0.10 ms (long buckets out of the threads' hands
//    among it: one thread's 30 additions took 0.45 ms).
static constexpr uint32_t kNoBucket = 0xffffffffu;

__global__ void msm_fixup_kernel(const uint32_t *__restrict__ starts, const uint32_t *__restrict__ open_bucket,
                                 uint32_t n, uint32_t L, uint32_t short_span,
                                 const xyzz_t *__restrict__ head, const xyzz_t *__restrict__ tail,
                                 xyzz_t *__restrict__ buckets, uint32_t *__restrict__ longs,
                                 uint32_t *__restrict__ nlong)
{
    uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    // a thread a chunk: the bucket that starts in it and runs on past its end
    if (open_bucket) g = open_bucket[g];
    if (g == kNoBucket) return;
    uint32_t s = starts[g], e = starts[g + 1];
    if (s == e) return;
    uint32_t cs = s / L, ce = (e - 1) / L;
    if (cs == ce) return;
    if (ce - cs > short_span) {
        longs[atomicAdd(nlong, 1u)] = g;
        return;
    }
    xyzz_t acc = tail[cs];
    for (uint32_t c = cs + 1; c < ce; c++) acc.GB_ADD_LAT(tail[c]);
    acc.GB_ADD_LAT(head[ce]);
    buckets[g] = acc;
}

// ---------------------------------------------------------------------------
// Cooperative point arithmetic for the latency-bound reduction.  The bucket
// reduction is a few chains of dependent XYZZ operations per segment, run on
// few warps, so its time is the latency of one operation times the chain
// length.  Here a group of 4 lanes runs one chain: the products of a point
// operation that do not depend on each other are computed by different lanes
// at the same time, with the operands and results in the group's
// shared-memory slots.  An addition is then 4 product levels deep (instead of
// 14 products in sequence) and a doubling 3 (instead of 10); with 8 lanes it is
// as deep, and half of them idle (4 x 2^16 points, fix-up and reduction with 8
// lanes 289 us, with 4 245).  Every decision (infinity, equal or opposite points) reads shared
// values after a group barrier, so the lanes always take the same path.
static constexpr uint32_t kCoopLanes = 4;
static constexpr uint32_t kCoopGroups = 32;  // groups per 128-thread block
// buckets up to which groups do the fix-up, and up to which they do so also
// where chunks are longer than buckets
static constexpr uint32_t kCoopFixupMaxBuckets = 1u << 16, kCoopFixupSmall = 1u << 14;
// slots of a group: SUM, OPD (operand; 4 each: X, Y, ZZ, ZZZ), then 12
// temporaries; an odd number, so that a warp's groups lie in different banks
enum { CO_SUM = 0, CO_OPD = 4, CO_TMP = 8, CO_SLOTS = 21 };

struct coop_t {
    fp_t *s;        // the group's slots
    uint32_t lane;  // 0..3
    uint32_t mask;  // the group's lanes in the warp
    __device__ coop_t(fp_t *mem)
        : s(mem + (size_t)(threadIdx.x / kCoopLanes) * CO_SLOTS), lane(threadIdx.x % kCoopLanes),
          mask(0xfu << (threadIdx.x & 28u))
    {
    }
    __device__ void sync() const { __syncwarp(mask); }
};

__device__ __forceinline__ void coop_set_inf(const coop_t &c, int a)
{
    if (c.lane == 0) {
        const xyzz_t z = xyzz_t::inf();
        c.s[a] = z.x, c.s[a + 1] = z.y, c.s[a + 2] = z.zz, c.s[a + 3] = z.zzz;
    }
    c.sync();
}

// a point (4 field elements, one a lane), read and written 16 bytes at a time
__device__ __forceinline__ fp_t load16(const void *p)
{
    const uint4 *f = reinterpret_cast<const uint4 *>(p);
    fp_t r;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const uint4 w = f[i];
        r.v[4 * i] = w.x, r.v[4 * i + 1] = w.y, r.v[4 * i + 2] = w.z, r.v[4 * i + 3] = w.w;
    }
    return r;
}

__device__ __forceinline__ void store16(void *p, const fp_t &v)
{
    uint4 *t = reinterpret_cast<uint4 *>(p);
#pragma unroll
    for (int i = 0; i < 3; i++) t[i] = make_uint4(v.v[4 * i], v.v[4 * i + 1], v.v[4 * i + 2], v.v[4 * i + 3]);
}

__device__ __forceinline__ fp_t coop_get(const coop_t &c, const void *p) { return load16((const fp_t *)p + c.lane); }
__device__ __forceinline__ void coop_put(const coop_t &c, void *p, const fp_t &v) { store16((fp_t *)p + c.lane, v); }

// 4 slots from src to dst
__device__ __forceinline__ void coop_copy(const coop_t &c, fp_t *dst, const fp_t *src)
{
    const fp_t v = coop_get(c, src);
    c.sync();
    coop_put(c, dst, v);
    c.sync();
}

__device__ __forceinline__ void coop_load(const coop_t &c, int a, const xyzz_t *g)
{
    coop_put(c, c.s + a, coop_get(c, g));
    c.sync();
}

__device__ __forceinline__ void coop_store(const coop_t &c, int a, xyzz_t *g) { coop_put(c, g, coop_get(c, c.s + a)); }

// One level of products: lane l < n computes s[xi[l]] * s[yi[l]] into
// s[oi[l]].  All lanes run the same call with their own operands, so the
// products of a level run side by side (a product per lane per branch would
// run them one after another).  Operands are read before any result is
// written.
//
// The slot indices of lane l sit in bits 5l .. 5l + 4 of x, y and o.
__device__ __forceinline__ uint32_t coop_pack(std::initializer_list<int> v)
{
    uint32_t r = 0, sh = 0;
    for (int i : v) r |= (uint32_t)i << sh, sh += 5;
    return r;
}

__device__ __forceinline__ void coop_level(const coop_t &c, uint32_t n, uint32_t x, uint32_t y, uint32_t o)
{
    const uint32_t sh = 5u * (c.lane < n ? c.lane : 0u);
    const fp_t a = load16(c.s + ((x >> sh) & 31u)), b = load16(c.s + ((y >> sh) & 31u));
    const fp_t r = a * b;
    c.sync();
    if (c.lane < n) store16(c.s + ((o >> sh) & 31u), r);
    c.sync();
}

// The same with squares: lane l < n computes s[xi[l]]^2 into s[oi[l]] (the
// squaring takes 234 multiply-adds where the product takes 300)
__device__ __forceinline__ void coop_level_sqr(const coop_t &c, uint32_t n, uint32_t x, uint32_t o)
{
    const uint32_t sh = 5u * (c.lane < n ? c.lane : 0u);
    const fp_t r = load16(c.s + ((x >> sh) & 31u)).sqr();
    c.sync();
    if (c.lane < n) store16(c.s + ((o >> sh) & 31u), r);
    c.sync();
}

// a = 2 a (dbl-2008-s-1, the products of xyzz_t::dbl in three levels)
__device__ void coop_dbl(const coop_t &c, int a)
{
    fp_t *s = c.s;
    if (s[a + 2].is_zero()) return;
    enum { U = CO_TMP, V, XX, M, W, S, MM, D, T0, T1 };
    {
        const fp_t u = s[a + 1].dbl();
        if (u.is_zero()) {
            coop_set_inf(c, a);
            return;
        }
        c.sync();
        if (c.lane == 0) s[U] = u;
        c.sync();
    }
    {
        coop_level_sqr(c, 2, coop_pack({U, a}), coop_pack({V, XX}));  // V = U^2, XX = X^2
    }
    if (c.lane == 0) s[M] = s[XX].dbl() + s[XX];
    c.sync();
    {
        // W = U V, S = X V, ZZ3 = V ZZ, MM = M^2
        coop_level(c, 4, coop_pack({U, a, V, M}), coop_pack({V, V, a + 2, M}), coop_pack({W, S, a + 2, MM}));
    }
    const fp_t X3 = s[MM] - s[S].dbl();
    if (c.lane == 0) s[D] = s[S] - X3;
    c.sync();
    {
        // M (S - X3), W Y, ZZZ3 = W ZZZ
        coop_level(c, 3, coop_pack({M, W, W}), coop_pack({D, a + 1, a + 3}), coop_pack({T0, T1, a + 3}));
    }
    if (c.lane == 0) {
        s[a] = X3;
        s[a + 1] = s[T0] - s[T1];
    }
    c.sync();
}

// a += q (add-2008-s, the products of xyzz_t::add in four levels); q's
// slots are left unchanged
__device__ void coop_add(const coop_t &c, int a, int q)
{
    fp_t *s = c.s;
    if (s[q + 2].is_zero()) return;
    if (s[a + 2].is_zero()) {
        coop_copy(c, s + a, s + q);
        return;
    }
    enum { U1 = CO_TMP, U2, S1, S2, Z12, W12, P, R, PP, RR, PPP, QQ };
    {
        // U1 = X1 ZZ2, U2 = X2 ZZ1, S1 = Y1 ZZZ2, S2 = Y2 ZZZ1
        coop_level(c, 4, coop_pack({a, q, a + 1, q + 1}), coop_pack({q + 2, a + 2, q + 3, a + 3}),
                   coop_pack({U1, U2, S1, S2}));
    }
    {
        const fp_t p = load16(s + U2) - load16(s + U1);
        const fp_t r = load16(s + S2) - load16(s + S1);
        if (p.is_zero()) {
            if (r.is_zero()) coop_dbl(c, a);
            else coop_set_inf(c, a);
            return;
        }
        c.sync();
        if (c.lane == 0) store16(s + P, p);
        if (c.lane == 1) store16(s + R, r);
        c.sync();
    }
    {
        // PP = P^2, RR = R^2, ZZ1 ZZ2, ZZZ1 ZZZ2
        coop_level(c, 4, coop_pack({P, R, a + 2, a + 3}), coop_pack({P, R, q + 2, q + 3}),
                   coop_pack({PP, RR, Z12, W12}));
    }
    {
        // PPP = P PP, Q = U1 PP, ZZ3 = ZZ1 ZZ2 PP
        coop_level(c, 3, coop_pack({P, U1, Z12}), coop_pack({PP, PP, PP}), coop_pack({PPP, QQ, a + 2}));
    }
    const fp_t qq = load16(s + QQ);
    const fp_t X3 = load16(s + RR) - load16(s + PPP) - qq.dbl();
    if (c.lane == 0) store16(s + U2, qq - X3);  // U2 is free from here on
    c.sync();
    {
        // R (Q - X3) -> S2, S1 PPP -> U1, ZZZ3 = ZZZ1 ZZZ2 PPP
        coop_level(c, 3, coop_pack({R, S1, W12}), coop_pack({U2, PPP, PPP}), coop_pack({S2, U1, a + 3}));
    }
    if (c.lane == 0) {
        store16(s + a, X3);
        store16(s + a + 1, load16(s + S2) - load16(s + U1));
    }
    c.sync();
}

// `groups` groups side by side (a power of two; `part` is a group's place among
// them) add their SUM slots into the first one's; every thread of the block
// takes part
__device__ void coop_tree(const coop_t &c, uint32_t part, uint32_t groups)
{
    for (uint32_t off = groups / 2; off > 0; off >>= 1) {
        __syncthreads();
        if (part < off) {
            coop_copy(c, c.s + CO_OPD, c.s + off * CO_SLOTS + CO_SUM);
            coop_add(c, CO_SUM, CO_OPD);
        }
    }
}

// 7'. msm_fixup_kernel with 2^log_parts groups of lanes a bucket: the partials
//     of a bucket are shared out to its groups, whose sums meet in a tree.  The
//     time is the longest bucket's chain of 5 us an addition.  A group takes as
//     many products as a thread (an addition's 14 and 2 idle ones), so it also
//     does up to 2^16 buckets (4 x 2^16 points 111 -> 88 us, 2^16 points 118 ->
//     82); several groups a bucket where there are few (2^10 points 51 -> 32
//     us with 4, 2^12 53 -> 41 with 2).
__global__ void __launch_bounds__(128) msm_fixup_coop_kernel(const uint32_t *__restrict__ starts, uint32_t G,
                                                             uint32_t L, uint32_t log_parts,
                                                             const xyzz_t *__restrict__ head,
                                                             const xyzz_t *__restrict__ tail,
                                                             xyzz_t *__restrict__ buckets,
                                                             uint32_t *__restrict__ longs,
                                                             uint32_t *__restrict__ nlong)
{
    __shared__ __align__(16) fp_t sh[kCoopGroups * CO_SLOTS];
    const uint32_t grp = threadIdx.x / kCoopLanes;
    const coop_t c(sh);
    const uint32_t parts = 1u << log_parts, g = (blockIdx.x * kCoopGroups + grp) >> log_parts, part = grp & (parts - 1);
    // a bucket's groups, side by side in a warp, go together everywhere
    if (g >= G) return;
    const uint32_t s = starts[g], e = starts[g + 1];
    if (s == e) return;
    const uint32_t cs = s / L, ce = (e - 1) / L;
    if (cs == ce) return;
    if (ce - cs > kShortSpan) {
        if (c.lane == 0 && part == 0) longs[atomicAdd(nlong, 1u)] = g;
        return;
    }
    if (cs + part <= ce) coop_load(c, CO_SUM, cs + part == ce ? head + ce : tail + cs + part);
    else coop_set_inf(c, CO_SUM);
    for (uint32_t k = cs + part + parts; k <= ce; k += parts) {
        c.sync();
        coop_load(c, CO_OPD, k == ce ? head + k : tail + k);
        coop_add(c, CO_SUM, CO_OPD);
    }
    const uint32_t lanes = parts * kCoopLanes;
    const uint32_t bucket_mask = (lanes == 32 ? 0xffffffffu : (1u << lanes) - 1) << (threadIdx.x & 31u & ~(lanes - 1));
    for (uint32_t off = parts / 2; off > 0; off >>= 1) {
        __syncwarp(bucket_mask);
        if (part < off) {
            coop_copy(c, c.s + CO_OPD, c.s + off * CO_SLOTS + CO_SUM);
            coop_add(c, CO_SUM, CO_OPD);
        }
    }
    if (part == 0) coop_store(c, CO_SUM, buckets + g);
}

// 7b. long buckets, one block each (grid-stride over the list): up to
//     kLongDirect partials are shared out to the block's 64 groups and the
//     groups' sums added in a tree (about 10 additions of 5 us); of more,
//     every thread first sums a strided share (14 us an addition, but 256 at
//     once), and the groups add the 256 shares.
static constexpr uint32_t kLongGroups = 64, kLongDirect = 512;
static constexpr size_t kLongSmem = kLongGroups * CO_SLOTS * sizeof(fp_t) + kLongGroups * kCoopLanes * sizeof(xyzz_t);

__global__ void __launch_bounds__(kLongGroups *kCoopLanes)
    msm_fixup_long_kernel(const uint32_t *__restrict__ starts, uint32_t L, const xyzz_t *__restrict__ head,
                          const xyzz_t *__restrict__ tail, const uint32_t *__restrict__ longs,
                          const uint32_t *__restrict__ nlong, xyzz_t *__restrict__ buckets)
{
    extern __shared__ __align__(16) unsigned char long_mem[];
    fp_t *mem = reinterpret_cast<fp_t *>(long_mem);
    xyzz_t *share = reinterpret_cast<xyzz_t *>(mem + kLongGroups * CO_SLOTS);
    const uint32_t grp = threadIdx.x / kCoopLanes;
    const coop_t c(mem);
    const uint32_t count = *nlong;
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        const uint32_t g = longs[i];
        // partials: tail[cs], tail[cs+1 .. ce-1], head[ce]
        const uint32_t cs = starts[g] / L, ce = (starts[g + 1] - 1) / L;
        const bool direct = ce - cs < kLongDirect;
        if (!direct) {
            xyzz_t acc = xyzz_t::inf();
            for (uint32_t k = cs + threadIdx.x; k <= ce; k += blockDim.x) acc.add(k == ce ? head[k] : tail[k]);
            share[threadIdx.x] = acc;
        }
        __syncthreads();
        const uint32_t n = direct ? ce - cs + 1 : kLongGroups * kCoopLanes;
        coop_set_inf(c, CO_SUM);
        for (uint32_t k = grp; k < n; k += kLongGroups) {
            c.sync();
            coop_load(c, CO_OPD, !direct ? share + k : cs + k == ce ? head + ce : tail + cs + k);
            coop_add(c, CO_SUM, CO_OPD);
        }
        coop_tree(c, grp, kLongGroups);
        if (grp == 0) coop_store(c, CO_SUM, buckets + g);
        __syncthreads();
    }
}

// 8'. The reduction of a single MSM or a small batch, whose time is the depth
//     of its chain of dependent additions: no running sums and no
//     multiplication by an offset.  A segment's K = rows x cols buckets, bucket
//     k at row k / cols and column k mod cols, have
//         sum (k + 1) B_k = cols sum_i i R_i + sum_j (j + 1) C_j
//     with the sums R_i of the rows and C_j of the columns: 2 K additions in
//     trees, as many as running sums take.  Each weighted sum of lines is
//     split by the bits of the weights, T_b = sum of the lines whose weight has
//     bit b, so that sum_b 2^b T_b over both is log2 K + 1 doublings and as
//     many additions, done by the host for a few segments and by one group a
//     segment beyond.  Measured against running sums over sub-segments, each
//     with its offset's double-and-add: one MSM of 2^12 buckets 0.172 -> 0.066
//     ms, of 2^15 0.299 -> 0.128, three of 2^15 0.53 -> 0.211 (with the host's
//     share, 15 us an MSM, outside these).  What bounds it: about 20 dependent
//     additions of 5 us.
struct line_shape {
    uint32_t lr, lc;  // log2 of rows and columns
    __host__ __device__ uint32_t lines() const { return (1u << lr) + (1u << lc); }
    __host__ __device__ uint32_t bits() const { return lr + lc + 1; }
};

// 8a'. partial line sums, 2^lm buckets a thread: a segment's 2 K / 2^lm
//      partials are the rows' [row][cols / 2^lm], then the columns'
//      [column][rows / 2^lm]
__global__ void __launch_bounds__(128) msm_line_partial_kernel(const xyzz_t *__restrict__ buckets, line_shape sh,
                                                               uint32_t lm, uint64_t total,
                                                               xyzz_t *__restrict__ partial)
{
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const uint32_t lk = sh.lr + sh.lc, half = 1u << (lk - lm), m = 1u << lm;
    const uint64_t seg = t >> (lk + 1 - lm);
    const uint32_t u = (uint32_t)t & (2 * half - 1);
    const xyzz_t *B = buckets + (seg << lk);
    uint32_t first, step, to;
    if (u < half) {
        const uint32_t row = u >> (sh.lc - lm), q = u & ((1u << (sh.lc - lm)) - 1);
        first = (row << sh.lc) + q, step = 1u << (sh.lc - lm), to = u;
    } else {
        const uint32_t col = (u - half) & ((1u << sh.lc) - 1), q = (u - half) >> sh.lc;
        first = (q << sh.lc) + col, step = 1u << (lk - lm), to = half + (col << (sh.lr - lm)) + q;
    }
    xyzz_t acc = B[first];
    for (uint32_t e = 1; e < m; e++) acc.add(B[first + e * step]);
    partial[seg * 2 * half + to] = acc;
}

// 8b'. whole line sums, 2^log_groups groups of lanes a line and a block's 32
//      groups on as many lines, from the partials (lm > 0) or the buckets (lm =
//      0).  Few lines take a block each; of many lines, which the number of
//      resident blocks bounds, short ones share a block (see sum_groups).
__global__ void __launch_bounds__(128) msm_line_sum_kernel(const xyzz_t *__restrict__ src, line_shape sh, uint32_t lm,
                                                           uint32_t log_groups, uint32_t total,
                                                           xyzz_t *__restrict__ lines)
{
    __shared__ __align__(16) fp_t mem[kCoopGroups * CO_SLOTS];
    const coop_t c(mem);
    const uint32_t grp = threadIdx.x / kCoopLanes, groups = 1u << log_groups, part = grp & (groups - 1);
    const uint32_t at = (blockIdx.x * kCoopGroups + grp) >> log_groups;
    const uint32_t lk = sh.lr + sh.lc, rows = 1u << sh.lr;
    const uint32_t seg = at / sh.lines(), line = at % sh.lines();
    const bool row = line < rows;
    const uint32_t n = at < total ? 1u << ((row ? sh.lc : sh.lr) - lm) : 0u;
    const xyzz_t *p = src + ((uint64_t)seg << (lm ? lk + 1 - lm : lk));
    uint32_t step = 1;
    if (row) p += (uint64_t)line * n;
    else if (lm) p += ((uint64_t)1 << (lk - lm)) + (uint64_t)(line - rows) * n;
    else p += line - rows, step = 1u << sh.lc;
    coop_set_inf(c, CO_SUM);
    for (uint32_t e = part; e < n; e += groups) {
        c.sync();
        coop_load(c, CO_OPD, p + (uint64_t)e * step);
        coop_add(c, CO_SUM, CO_OPD);
    }
    coop_tree(c, part, groups);
    if (part == 0 && n) coop_store(c, CO_SUM, lines + at);
}

// 8c'. the sums by weight bit, 2^log_groups groups a bit: rows weigh i (bits 0
//      .. lr - 1, in places 2^lc and up of the result), columns j + 1 (bits 0 ..
//      lc)
__global__ void __launch_bounds__(128) msm_bit_sum_kernel(const xyzz_t *__restrict__ lines, line_shape sh,
                                                          uint32_t log_groups, uint32_t total,
                                                          xyzz_t *__restrict__ bits)
{
    __shared__ __align__(16) fp_t mem[kCoopGroups * CO_SLOTS];
    const coop_t c(mem);
    const uint32_t grp = threadIdx.x / kCoopLanes, groups = 1u << log_groups, part = grp & (groups - 1);
    const uint32_t at = (blockIdx.x * kCoopGroups + grp) >> log_groups;
    const uint32_t seg = at / sh.bits(), place = at % sh.bits(), rows = 1u << sh.lr;
    const bool row = place < sh.lr;
    const uint32_t b = row ? place : place - sh.lr, lw = row ? sh.lr : sh.lc;
    const xyzz_t *p = lines + (uint64_t)seg * sh.lines() + (row ? 0 : rows);
    // weights below 2^lw with bit b, or 2^lc itself for the columns' last bit
    const uint32_t n = at >= total ? 0u : b < lw ? 1u << (lw - 1) : 1u;
    coop_set_inf(c, CO_SUM);
    for (uint32_t e = part; e < n; e += groups) {
        const uint32_t w = b < lw ? (e >> b) << (b + 1) | 1u << b | (e & ((1u << b) - 1)) : 1u << b;
        c.sync();
        coop_load(c, CO_OPD, p + (row ? w : w - 1));
        coop_add(c, CO_SUM, CO_OPD);
    }
    coop_tree(c, part, groups);
    if (part == 0 && n) coop_store(c, CO_SUM, bits + at);
}

// 8d'. the bit sums of a segment to one point, a block a segment: a group
//      doubles a bit's sum up to its place, and the groups' points meet in a
//      tree (at most 15 doublings and 4 additions in a row, where Horner's rule
//      by one group takes as many doublings and 16 additions: a plain MSM of
//      2^16 points, 24 segments of 2^10 buckets, reduction 205 -> 168 us)
static constexpr uint32_t kCombineGroups = 16;

__global__ void __launch_bounds__(kCombineGroups *kCoopLanes) msm_bit_combine_kernel(const xyzz_t *__restrict__ bits,
                                                                                    line_shape sh,
                                                                                    xyzz_t *__restrict__ seg_sum)
{
    __shared__ __align__(16) fp_t mem[kCombineGroups * CO_SLOTS];
    const uint32_t grp = threadIdx.x / kCoopLanes;
    const coop_t c(mem);
    const xyzz_t *p = bits + (uint64_t)blockIdx.x * sh.bits();
    if (grp < sh.bits()) {
        coop_load(c, CO_SUM, p + grp);
        const uint32_t place = grp < sh.lr ? sh.lc + grp : grp - sh.lr;
        for (uint32_t k = 0; k < place; k++) coop_dbl(c, CO_SUM);
    } else {
        coop_set_inf(c, CO_SUM);
    }
    coop_tree(c, grp, kCombineGroups);
    if (grp == 0) coop_store(c, CO_SUM, seg_sum + blockIdx.x);
}

// 8e. plain MSMs beyond a few: combine an MSM's window segments by Horner's
//     rule, a group an MSM ((windows - 1) * c doublings)
__global__ void __launch_bounds__(128) msm_combine_coop_kernel(const xyzz_t *__restrict__ seg_sum, uint32_t nitems,
                                                               uint32_t segs_per_item, int c,
                                                               xyzz_t *__restrict__ out)
{
    __shared__ __align__(16) fp_t sh[kCoopGroups * CO_SLOTS];
    const uint32_t grp = threadIdx.x / kCoopLanes;
    const coop_t cp(sh);
    const uint32_t m = blockIdx.x * kCoopGroups + grp;
    if (m >= nitems) return;  // whole groups leave together; no block barrier follows
    const xyzz_t *ss = seg_sum + (size_t)m * segs_per_item;
    coop_set_inf(cp, CO_SUM);
    for (int w = (int)segs_per_item - 1; w >= 0; w--) {
        if (w != (int)segs_per_item - 1)
            for (int k = 0; k < window_bits(c, w); k++) coop_dbl(cp, CO_SUM);
        coop_load(cp, CO_OPD, ss + w);
        coop_add(cp, CO_SUM, CO_OPD);
    }
    cp.sync();
    coop_store(cp, CO_SUM, out + m);
}

// precompute: table[j * n + i] = 2^(c*j) P_i
__global__ void msm_precompute_kernel(affine_t *table, size_t n, int c, int nwin)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    affine_t p = table[i];
    xyzz_t acc = xyzz_t::from_affine(p);
    for (int j = 1; j < nwin; j++) {
        for (int k = 0; k < window_bits(c, j - 1); k++) acc = acc.dbl();
        table[(size_t)j * n + i] = acc.to_affine();
    }
}

// scrambled scalars: out[i] = in[i] + mask[i mod mask_len]
__global__ void add_mask_kernel(fr_t *__restrict__ out, const fr_t *__restrict__ in, const fr_t *__restrict__ mask,
                                size_t mask_len, size_t len)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < len) out[i] = in[i] + mask[i % mask_len];
}

// ---------------------------------------------------------------------------
// host engine
// ---------------------------------------------------------------------------

static void set_smem_attrs()
{
    static device_once once;
    once.run(current_device(), [] {
        const size_t bytes = ((size_t)1 << (kMaxWindowBits - 1)) * 4;
        allow_dynamic_smem(msm_hist_kernel, bytes);
        allow_dynamic_smem(msm_scatter_kernel, bytes);
        allow_dynamic_smem(msm_fixup_long_kernel, kLongSmem);
    });
}

// Exclusive scan of n u32 counts into out[0..n], out[n] = total (device).
static void u32_exclusive_scan(const uint32_t *in, uint32_t n, uint32_t *out, cudaStream_t s)
{
    uint32_t tiles = (n + kScanTileU32 - 1) / kScanTileU32;
    if (tiles > 1024 * 64) throw cuda_error((int)cudaErrorInvalidValue, "MSM bucket count too large");
    dev_buf<uint32_t> sums(tiles + 1, s);
    u32_tile_sum_kernel<<<tiles, 256, 0, s>>>(in, n, sums);
    GB_CHECK_LAUNCH();
    // total = sum of tile sums: scan tiles+1 values whose last is 0
    GB_CUDA_OK(cudaMemsetAsync(sums.get() + tiles, 0, sizeof(uint32_t), s));
    u32_small_scan_kernel<<<1, 1024, 0, s>>>(sums, tiles + 1);
    GB_CHECK_LAUNCH();
    // sums[tiles] now holds the grand total; pass it through device memory
    u32_tile_scan_kernel<<<tiles, 256, 0, s>>>(in, n, sums, out);
    GB_CHECK_LAUNCH();
    GB_CUDA_OK(cudaMemcpyAsync(out + n, sums.get() + tiles, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
}

// Entries per accumulation thread: about half a bucket (8..64), then set so
// that the chunks fill whole waves of resident accumulation blocks (a 2^16
// MSM's 65536 chunks of 16 fill 84 % of one wave on 152 SMs; chunks of 14
// fill 96 %; a 2^20 MSM's 3.4 waves of 64 become 3 of 72).
static uint32_t chunk_length(uint64_t digits, double avg, uint32_t G, int variant, int sms)
{
    uint32_t L = (uint32_t)std::max(8.0, std::min(64.0, avg * 0.5));
    static device_once once;
    static int per_sm[kMaxDevices][3];
    const int v = variant < 0 || variant > 2 ? 1 : variant, dev = current_device();
    once.run(dev, [&] {
        int b[3];
        GB_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b[0], msm_accumulate_kernel<256, 1>, 256, 0));
        GB_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b[1], msm_accumulate_kernel<256, 2>, 256, 0));
        GB_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b[2], msm_accumulate_kernel<128, 3>, 128, 0));
        for (int k = 0; k < 3; k++) per_sm[dev][k] = std::max(1, b[k]) * (k == 2 ? 128 : 256);
    });
    const uint64_t wave = (uint64_t)sms * (uint64_t)per_sm[dev][v];  // chunks resident at once
    // short buckets, large batches: chunks long enough for 8 waves, as every
    // chunk's edge costs a fix-up
    if (wave) L = std::max<uint32_t>(L, (uint32_t)std::min<uint64_t>(64, digits / (8 * wave)));
    if (!wave || !digits) return L;
    // whole waves, rounded down (longer chunks: shorter fix-up chains) when
    // there are several, up when there is less than one
    const uint64_t waves = std::max<uint64_t>(1, digits / ((uint64_t)L * wave));
    const uint64_t L2 = (digits + waves * wave - 1) / (waves * wave);
    if (L2 >= 8 && L2 <= 2 * (uint64_t)L) return (uint32_t)L2;
    if (L2 >= 8) return L;
    // Less than one wave of 8-digit chunks (small MSMs, where two lanes a chunk
    // are not chosen): the accumulation takes about L dependent additions per
    // thread and the fix-up about avg / L (the chunks a bucket spans; groups of
    // lanes up to kCoopFixupMaxBuckets buckets, single threads, ~1.6x slower,
    // beyond), so L ~ sqrt(avg x their latency ratio); and at least 3 digits
    // per resident chunk slot, where the additions start to queue on the
    // multiply-add pipe.
    const double ratio = G <= kCoopFixupMaxBuckets ? 0.8 : 1.3;
    const uint64_t by_latency = (uint64_t)std::lround(std::sqrt(avg * ratio));
    const uint64_t by_load = (3 * digits + wave - 1) / wave;
    return (uint32_t)std::min<uint64_t>(L, std::max<uint64_t>(4, std::max(by_latency, by_load)));
}

// Entries per pair of lanes: the accumulation takes about L dependent
// additions of 5 us and the fix-up avg / L, so L ~ sqrt(avg); and the chunks
// fill whole waves of resident ones, one wave unless that takes more than twice
// that (measured, call in us for L = 3, 4, 5, 6, 8: 2^10 points, 11 entries a
// bucket, 176* 181 186 190 197; 2^12, 20 entries, 220 220 210* 214 224; 2 x
// 2^12 268 259 268 249* 264).
static uint32_t pair_chunk_length(uint64_t digits, double avg, uint32_t G, int sms)
{
    const uint64_t wave = (uint64_t)sms * kPairSm * kPairChunks;
    // a few buckets of hundreds of entries (a window of 8 or 9 bits asked for)
    // have a block each to join their chunks, many at once: 2^12 points in 128
    // buckets 0.37 -> 0.27 ms with 16 in place of 33
    const double by_latency = std::min(G <= 256 ? 16.0 : 64.0, std::max(3.0, std::sqrt(avg * 1.1)));
    uint64_t L = 1;
    for (uint64_t waves = 1;; waves++) {
        L = (digits + waves * wave - 1) / (waves * wave);
        if ((double)L <= 2 * by_latency) break;
    }
    return (uint32_t)std::max<uint64_t>(L, (uint64_t)by_latency);
}

// What the device leaves of each MSM and the host finishes once it is copied:
// one point; the bit sums of its buckets (a context's MSM); or its window
// sums (a plain MSM).  The last two are one chain of dependent doublings and
// additions, which a host core runs 7 times faster than a group of GPU lanes
// (about 25 us for 16 bit sums, 0.15 to 0.2 ms for 20 windows, against 0.13
// and 1.1 ms); the GPU runs them for batches of more than a few MSMs (plain,
// 2^16 points, ms finished by the host and by the GPU: 5 3.82 4.00, 6 4.50
// 4.53, 7 5.25 5.14).
static constexpr uint32_t kHostTailBits = 8, kHostTailWindows = 6;  // MSMs at most

struct msm_tail {
    enum { POINT, BITS, WINDOWS } kind = POINT;
    uint32_t points = 1;  // of an MSM
    int c = 0;
    line_shape shape{0, 0};
    jacobian_t finish(const xyzz_t *p) const;
};

jacobian_t msm_tail::finish(const xyzz_t *dev) const
{
    using namespace hostfp;
    static_assert(sizeof(xyzz64) == sizeof(xyzz_t), "one memory image");
    const xyzz64 *p = reinterpret_cast<const xyzz64 *>(dev);
    xyzz64 acc = infinity();
    if (kind == POINT) {
        acc = p[0];
    } else if (kind == WINDOWS) {
        for (int w = (int)points - 1; w >= 0; w--) {
            if (w != (int)points - 1)
                for (int k = 0; k < window_bits(c, w); k++) acc = dbl(acc);
            acc = add(acc, p[w]);
        }
    } else {
        const int lr = (int)shape.lr, lc = (int)shape.lc;
        for (int b = lr + lc; b >= 0; b--) {
            acc = dbl(acc);
            if (b >= lc && b < lr + lc) acc = add(acc, p[b - lc]);
            if (b <= lc) acc = add(acc, p[lr + b]);
        }
    }
    // (X ZZ^2, Y ZZZ^2, ZZZ) is a Jacobian form of the point
    xyzz64 r{kOne, kOne, acc.zzz, acc.zzz};
    if (!is_zero(acc.zz)) {
        r.x = mont_mul(acc.x, mont_mul(acc.zz, acc.zz));
        r.y = mont_mul(acc.y, mont_mul(acc.zzz, acc.zzz));
    } else {
        r.zz = acc.zz;
    }
    jacobian_t j;
    memcpy(&j, &r, sizeof(j));  // x, y and z in place of zz
    return j;
}

// The host half of a batch: its descriptors and launch sizes.
struct batch_plan {
    bool pair = false, fix_coop = false;  // two lanes a chunk; groups of lanes in the fix-up
    uint32_t log_parts = 0;               // log2 of the groups a bucket in it
    int c = 0, nwin = 0, variant = 1;
    bool precomputed = false, fix_by_chunk = false;
    size_t stride = 0;
    uint32_t nitems = 0, K = 0, segs_per_item = 0, nseg = 0, G = 0, nblocks = 0, L = 0, short_span = kShortSpan;
    line_shape shape{0, 0};
    msm_tail tail;
    int rounds = 0;          // affine rounds before the accumulation
    uint64_t entries = 0;    // bound of the bucket-ordered list, padding included
    uint64_t scratch = 0;    // bytes of the affine rounds' lists and prefixes
    uint64_t points_total = 0, digits_total = 0, nchunks = 0;
    std::vector<item_desc> idesc;
    std::vector<seg_desc> sdesc;
    std::vector<blk_desc> bdesc;
};

// The plan of `nitems` items, a group of a batch of batch_items (all of them,
// mostly); most_scratch bounds the affine rounds' scratch.
static batch_plan plan_batch(const msm_item *items, uint32_t nitems, size_t batch_items, int c, bool precomputed,
                             size_t stride, uint64_t most_scratch)
{
    batch_plan P;
    P.nitems = nitems;
    const int nwin = windows_for(c);
    const uint32_t K = 1u << (c - 1);
    const uint32_t segs_per_item = precomputed ? 1u : (uint32_t)nwin;
    const uint32_t nseg = nitems * segs_per_item;
    const uint64_t G64 = (uint64_t)nseg * K;
    if (G64 >= 0x7fffffffull) throw cuda_error((int)cudaErrorInvalidValue, "MSM batch too large");
    const uint32_t G = (uint32_t)G64;

    // items, segments, sort blocks
    std::vector<item_desc> idesc(nitems);
    std::vector<seg_desc> sdesc(nseg);
    uint64_t points_total = 0, digits_total = 0;
    typical_bucket bucket;
    for (uint32_t m = 0; m < nitems; m++) {
        const msm_item &it = items[m];
        if (it.n >= kMaxDigits / (uint64_t)nwin) throw cuda_error((int)cudaErrorInvalidValue, "MSM too large");
        idesc[m] = item_desc{it.scalars, points_total, digits_total, (uint32_t)it.n};
        for (uint32_t j = 0; j < segs_per_item; j++) {
            seg_desc &sd = sdesc[m * segs_per_item + j];
            sd.digit_off = digits_total + (precomputed ? 0 : (uint64_t)j * it.n);
            sd.len = (uint32_t)(precomputed ? it.n * nwin : it.n);
            sd.n = (uint32_t)std::max<size_t>(it.n, 1);
            sd.point_base = it.point_base;
        }
        bucket.add(it.n);
        points_total += it.n;
        digits_total += (uint64_t)it.n * nwin;
    }
    if (points_total + stride * (uint64_t)nwin >= 0x80000000ull && precomputed)
        throw cuda_error((int)cudaErrorInvalidValue, "MSM table too large for 31-bit point references");
    // ~4 sort blocks per SM pair over the whole batch, 4096..65536 digits
    // each, and at least K (2K from 2^23 digits): every block writes and the
    // column scan and scatter read a K-entry histogram, so blocks far
    // shorter than K move more histogram than digits (measured on GB300: the
    // sort of a 2^18-point MSM 0.192 -> 0.098 ms, of three 2^16-point MSMs
    // 0.183 -> 0.093 ms, of a 2^20-point MSM 0.387 -> 0.311 ms)
    const uint64_t per_min = std::max<uint64_t>(4096, (uint64_t)K << (digits_total >= (1u << 23) ? 1 : 0));
    uint64_t per = std::max<uint64_t>(per_min, std::min<uint64_t>(65536, (digits_total + 607) / 608));
    std::vector<blk_desc> bdesc;
    for (uint32_t sidx = 0; sidx < nseg; sidx++) {
        seg_desc &sd = sdesc[sidx];
        sd.blk0 = (uint32_t)bdesc.size();
        uint32_t nb = (uint32_t)std::max<uint64_t>(1, (sd.len + per - 1) / per);
        uint32_t chunk = (sd.len + nb - 1) / std::max<uint32_t>(nb, 1);
        for (uint32_t b = 0; b < nb; b++) {
            uint32_t lo = b * chunk, hi = std::min(sd.len, lo + chunk);
            bdesc.push_back(blk_desc{sidx, lo, std::max(lo, hi)});
        }
        sd.nblk = nb;
    }
    const uint32_t nblocks = (uint32_t)bdesc.size();
    const double avg = (double)digits_total / (double)G;
    const int variant = default_acc_variant();
    const int sms = sm_count();
    const uint64_t slots = (uint64_t)sms * kPairBlocks;
    const int rounds = affine_rounds(digits_total, avg, G, slots, most_scratch);
    const uint64_t entries = padded_entries(digits_total, G, rounds);
    // a batch of less than 6 entries a resident thread: two lanes a chunk
    // (measured, accumulation in us with a thread and with two lanes a chunk:
    // 2^10 points 63 -> 25, 2^12 64 -> 44, 2 x 2^12 107 -> 72, 4 x 2^12 151 ->
    // 129, 2^14 189 -> 149; 2 x 2^14, 8 entries a thread, 243 and 243, and 2^16
    // 432 and 450)
    const bool pair = variant == 1 && !rounds && digits_total < 6 * (uint64_t)sms * 512;
    const double typical = bucket.entries(c, precomputed) / (1 << rounds);
    const uint32_t L = pair ? pair_chunk_length(digits_total, typical, G, sms)
                            : chunk_length(entries >> rounds, typical, G, variant, sms);
    const uint64_t nchunks = std::max<uint64_t>(1, ((entries >> rounds) + L - 1) / L);

    P.pair = pair;
    P.c = c;
    P.nwin = nwin;
    P.variant = variant;
    P.precomputed = precomputed;
    P.stride = stride;
    P.K = K;
    P.segs_per_item = segs_per_item;
    P.nseg = nseg;
    P.G = G;
    P.nblocks = nblocks;
    P.L = L;
    P.shape.lr = (uint32_t)(c - 1) / 2;
    P.shape.lc = (uint32_t)(c - 1) - P.shape.lr;
    // the steps left to the host: see msm_tail
    P.tail.c = c;
    if (precomputed && batch_items <= kHostTailBits) {
        P.tail.kind = msm_tail::BITS;
        P.tail.shape = P.shape;
        P.tail.points = P.shape.bits();
    } else if (!precomputed && batch_items <= kHostTailWindows) {
        P.tail.kind = msm_tail::WINDOWS;
        P.tail.points = segs_per_item;
    }
    P.points_total = points_total;
    P.digits_total = digits_total;
    P.nchunks = nchunks;
    P.fix_by_chunk = G > kCoopFixupSmall && avg / (1 << rounds) < L;
    P.fix_coop = !P.fix_by_chunk && G <= kCoopFixupMaxBuckets;
    P.log_parts = G <= 2048 ? 2 : G <= 8192 ? 1 : 0;
    P.short_span = short_span(avg / (1 << rounds), typical, L);
    P.rounds = rounds;
    P.entries = entries;
    P.scratch = rounds_scratch(entries, rounds, slots);
    P.idesc = std::move(idesc);
    P.sdesc = std::move(sdesc);
    P.bdesc = std::move(bdesc);
    return P;
}

// Buffers of the affine rounds, allocated before a batch's first launch, so
// that a device without room for them fails before any work is queued.
struct round_buffers {
    dev_buf<uint4> prefix;
    dev_buf<affine_t> list_a, list_b, result;  // result: of all slices
    round_buffers(const batch_plan &P, cudaStream_t s)
    {
        if (!P.rounds) return;
        const uint64_t slots = (uint64_t)sm_count() * kPairBlocks, slice = slice_entries(P.entries);
        prefix = dev_buf<uint4>(slots * pairs_per_thread(slice / 2, slots) * 3 * kPairThreads, s);
        if (sliced(P.entries)) result = dev_buf<affine_t>((P.entries >> P.rounds) + 1, s);
        if (!result || P.rounds > 1) list_a = dev_buf<affine_t>(slice / 2 + 1, s);
        if (P.rounds > 1) list_b = dev_buf<affine_t>(slice / 4 + 1, s);
    }
};

// The affine rounds: the bucket-ordered references through P.rounds pairwise
// additions, to a list of points a 2^rounds-th as long.
static const affine_t *run_affine_rounds(const batch_plan &P, const uint32_t *sorted, const uint32_t *starts,
                                         const affine_t *points, const round_buffers &buf, cudaStream_t s)
{
    const uint64_t slots = (uint64_t)sm_count() * kPairBlocks, slice = slice_entries(P.entries);
    const affine_t *in = nullptr;
    for (uint64_t lo = 0; lo < P.entries; lo += slice) {
        const uint64_t hi = std::min(P.entries, lo + slice);
        in = points;
        for (int r = 1; r <= P.rounds; r++) {
            affine_t *out = buf.result && r == P.rounds ? buf.result.get() + (lo >> r)
                            : r & 1                     ? buf.list_a.get()
                                                        : buf.list_b.get();
            const uint64_t pairs = (hi - lo) >> r;
            const uint32_t per = std::min(pairs_per_thread(pairs, slots), pairs_per_thread(slice / 2, slots));
            const uint64_t tiles = (pairs + (uint64_t)per * kPairThreads - 1) / ((uint64_t)per * kPairThreads);
            const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min(slots, tiles));
            if (r == 1)
                msm_affine_pairs_kernel<true><<<grid, kPairThreads, 0, s>>>(
                    sorted + lo, in, out, starts + P.G, (uint32_t)lo, (uint32_t)hi, r, per, buf.prefix);
            else
                msm_affine_pairs_kernel<false><<<grid, kPairThreads, 0, s>>>(
                    nullptr, in, out, starts + P.G, (uint32_t)lo, (uint32_t)hi, r, per, buf.prefix);
            GB_CHECK_LAUNCH();
            in = out;
        }
    }
    return buf.result ? buf.result.get() : in;
}

// The device half: every launch of the batch, its scratch allocated and
// freed in stream order on s, the descriptors already in device memory.
// Queues device work only (no host synchronisation, no copy from host
// memory), so a CUDA graph can capture it.
static void run_planned(const batch_plan &P, const item_desc *d_items, const seg_desc *d_segs,
                        const blk_desc *d_blks, const affine_t *points, xyzz_t *d_out, cudaStream_t s)
{
    const int c = P.c, variant = P.variant;
    const bool precomputed = P.precomputed;
    const size_t stride = P.stride;
    const uint32_t nitems = P.nitems, K = P.K, segs_per_item = P.segs_per_item, nseg = P.nseg, G = P.G;
    const uint32_t nblocks = P.nblocks, L = P.L;
    const uint64_t points_total = P.points_total, digits_total = P.digits_total, nchunks = P.nchunks;
    const round_buffers round_buf(P, s);
    dev_buf<uint32_t> digits(std::max<uint64_t>(digits_total, 1), s), sorted(std::max<uint64_t>(P.entries, 1), s);
    dev_buf<uint32_t> hist((size_t)nblocks * K, s), counts(G, s), starts((size_t)G + 1, s), ctl(CTL_WORDS, s);
    dev_buf<xyzz_t> buckets(G, s), head(nchunks, s), tail(nchunks, s);
    dev_buf<uint32_t> open_bucket(P.fix_by_chunk ? nchunks : 0, s);

    int tok_all = timed_begin(s);
    int tok_sort = timed_begin(s);
    if (points_total) {
        launch_recode(d_items, nitems, points_total, c, digits, s);
    }
    const size_t smem = (size_t)K * 4;
    msm_hist_kernel<<<nblocks, 1024, smem, s>>>(digits, d_segs, d_blks, K, hist, ctl);
    GB_CHECK_LAUNCH();
    const bool scan_here = G <= kScanHere;
    const uint32_t col_threads = scan_here ? 1024 : 256;
    msm_colscan_kernel<<<blocks_for(G, col_threads), col_threads, 0, s>>>(
        hist, d_segs, K, G, (1u << P.rounds) - 1, counts, buckets, scan_here ? starts.get() : nullptr, ctl);
    GB_CHECK_LAUNCH();
    if (P.rounds) GB_CUDA_OK(cudaMemsetAsync(sorted.get(), 0xff, P.entries * sizeof(uint32_t), s));  // kNoPoint
    if (!scan_here) u32_exclusive_scan(counts, G, starts, s);
    msm_scatter_kernel<<<nblocks, 1024, smem, s>>>(digits, d_segs, d_blks, K, precomputed ? stride : 0, hist,
                                                   starts, sorted);
    GB_CHECK_LAUNCH();
    timed_end(tok_sort, s, GB_SLOT_MSM_SORT);
    int tok = timed_begin(s);
    if (P.fix_by_chunk) GB_CUDA_OK(cudaMemsetAsync(open_bucket.get(), 0xff, nchunks * sizeof(uint32_t), s));
    dev_buf<uint32_t> shifted;
    const uint32_t *bounds = starts;
    if (P.rounds) {
        const affine_t *list = run_affine_rounds(P, sorted, starts, points, round_buf, s);
        shifted = dev_buf<uint32_t>((size_t)G + 1, s);
        msm_shift_starts_kernel<<<blocks_for(G + 1, 256), 256, 0, s>>>(starts, G + 1, P.rounds, shifted);
        GB_CHECK_LAUNCH();
        bounds = shifted;
        msm_accumulate_kernel<256, 2, false><<<(unsigned)((nchunks + 255) / 256), 256, 0, s>>>(
            nullptr, bounds, G, L, nchunks, list, buckets, head, tail, open_bucket);
    } else if (P.pair) {
        msm_accumulate_pair_kernel<<<(unsigned)((nchunks + kPairChunks - 1) / kPairChunks), 2 * kPairChunks, 0, s>>>(
            sorted, starts, G, L, nchunks, points, buckets, head, tail, open_bucket);
    } else if (variant == 1) {
        msm_accumulate_kernel<256, 2><<<(unsigned)((nchunks + 255) / 256), 256, 0, s>>>(
            sorted, starts, G, L, nchunks, points, buckets, head, tail, open_bucket);
    } else if (variant == 2) {
        msm_accumulate_kernel<128, 3><<<(unsigned)((nchunks + 127) / 128), 128, 0, s>>>(
            sorted, starts, G, L, nchunks, points, buckets, head, tail, open_bucket);
    } else {
        msm_accumulate_kernel<256, 1><<<(unsigned)((nchunks + 255) / 256), 256, 0, s>>>(
            sorted, starts, G, L, nchunks, points, buckets, head, tail, open_bucket);
    }
    GB_CHECK_LAUNCH();
    timed_end(tok, s, GB_SLOT_MSM_ACCUMULATE);
    int tok_fix = timed_begin(s);
    {
        dev_buf<uint32_t> longs(G, s);
        uint32_t *nlong = ctl.get() + CTL_LONGS;
        if (P.fix_coop) {
            const uint32_t groups = G << P.log_parts;
            msm_fixup_coop_kernel<<<(groups + kCoopGroups - 1) / kCoopGroups, 128, 0, s>>>(
                bounds, G, L, P.log_parts, head, tail, buckets, longs, nlong);
        } else {
            const uint32_t n = P.fix_by_chunk ? (uint32_t)nchunks : G;
            msm_fixup_kernel<<<blocks_for(n, 128), 128, 0, s>>>(bounds, open_bucket, n, L, P.short_span, head, tail,
                                                                buckets, longs, nlong);
        }
        GB_CHECK_LAUNCH();
        msm_fixup_long_kernel<<<sm_count() * 2, kLongGroups * kCoopLanes, kLongSmem, s>>>(bounds, L, head, tail, longs,
                                                                                          nlong, buckets);
        GB_CHECK_LAUNCH();
    }
    timed_end(tok_fix, s, GB_SLOT_MSM_FIXUP);
    int tok_red = timed_begin(s);
    // an MSM's one point goes to d_out, its segments' sums elsewhere first
    dev_buf<xyzz_t> sums;
    xyzz_t *seg_sum = d_out;
    if (segs_per_item > 1 && P.tail.kind == msm_tail::POINT) {
        sums = dev_buf<xyzz_t>(nseg, s);
        seg_sum = sums;
    }
    {
        const line_shape sh = P.shape;
        const uint64_t total = (uint64_t)nseg * K;
        // 2^lm buckets a thread adds before the lines' blocks take over: none up
        // to 2^20 buckets, where chains are what costs (one-thread additions
        // take 14 us each, a group's 5), and 16 beyond, where a thread's 14
        // products an addition beat a group's 16 slots (measured, us for lm =
        // 0, 1, 2, 3, 4: 4096 buckets 66* 87 110 162 271, 2^15 128* 136 140 191
        // 300, 4 x 2^15 272* 310 284 271 334, 8 x 2^15 428* 505 487 461 442, 12
        // x 2^15 669* 792 751 730 844; 64 x 2^15 ms 2.89 3.53 3.21 3.04 2.88*);
        // but no more than a column has (8 with windows of 8 bits).
        const uint32_t lm = total <= 1u << 20 ? 0 : std::min(4u, sh.lr);
        dev_buf<xyzz_t> partial, lines((size_t)nseg * sh.lines(), s), bits;
        const xyzz_t *src = buckets;
        if (lm) {
            const uint64_t n = total * 2 >> lm;
            partial = dev_buf<xyzz_t>(n, s);
            msm_line_partial_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(buckets, sh, lm, n, partial);
            GB_CHECK_LAUNCH();
            src = partial;
        }
        const uint32_t nlines = sh.lines() * nseg, lg = sum_groups(nlines, 1u << (sh.lc - lm), sm_count());
        msm_line_sum_kernel<<<blocks_for((size_t)nlines << lg, kCoopGroups), 128, 0, s>>>(src, sh, lm, lg, nlines,
                                                                                           lines);
        GB_CHECK_LAUNCH();
        xyzz_t *bit_sum = d_out;
        if (P.tail.kind != msm_tail::BITS) {
            bits = dev_buf<xyzz_t>((size_t)nseg * sh.bits(), s);
            bit_sum = bits;
        }
        const uint32_t nbits = sh.bits() * nseg, bg = sum_groups(nbits, 1u << (sh.lc - 1), sm_count());
        msm_bit_sum_kernel<<<blocks_for((size_t)nbits << bg, kCoopGroups), 128, 0, s>>>(lines, sh, bg, nbits,
                                                                                         bit_sum);
        GB_CHECK_LAUNCH();
        if (P.tail.kind != msm_tail::BITS) {
            msm_bit_combine_kernel<<<nseg, kCombineGroups * kCoopLanes, 0, s>>>(bits, sh, seg_sum);
            GB_CHECK_LAUNCH();
        }
    }
    if (segs_per_item > 1 && P.tail.kind == msm_tail::POINT) {
        msm_combine_coop_kernel<<<(nitems + kCoopGroups - 1) / kCoopGroups, 128, 0, s>>>(seg_sum, nitems,
                                                                                          segs_per_item, c, d_out);
        GB_CHECK_LAUNCH();
    }
    timed_end(tok_red, s, GB_SLOT_MSM_REDUCE);
    timed_end(tok_all, s, GB_SLOT_MSM_TOTAL);
}

// CUDA-graph replay of a batch's launch sequence.  A batch whose shape
// (window, sizes, chunking, launch geometry) and bases pointer come a
// second time on the same stream is captured as a graph, replayed from then
// on: the graph reads its descriptors from device buffers of its own, refreshed by
// one copy each before the launch, and writes its results to a buffer of
// its own, copied to the caller's after it.  Its scratch is allocated and
// freed by the graph's memory nodes.  A proof or a server sends the same
// batch shapes round after round, so the host enqueues 4 operations instead
// of about 25, and the device runs the sequence without per-launch gaps.
struct graph_key {
    int device = 0;
    cudaStream_t stream = nullptr;
    const affine_t *points = nullptr;
    int c = 0, variant = 0;
    bool precomputed = false, fix_by_chunk = false;
    int tail = 0;
    size_t stride = 0;
    uint32_t nitems = 0, K = 0, segs_per_item = 0, nseg = 0, G = 0, nblocks = 0, L = 0, short_span = 0;
    int rounds = 0;
    uint64_t points_total = 0, digits_total = 0, nchunks = 0;
    auto tie() const
    {
        return std::tie(device, stream, points, c, variant, precomputed, fix_by_chunk, tail, stride, nitems, K,
                        segs_per_item, nseg, G, nblocks, L, short_span, rounds, points_total, digits_total, nchunks);
    }
    bool operator<(const graph_key &o) const { return tie() < o.tie(); }
};

// A captured graph and its buffers, freed on its stream when the last user
// lets go of it (an executable graph still running is freed when it
// completes; the buffers go back in stream order behind it).
struct graph_entry {
    cudaStream_t stream = nullptr;
    cudaGraphExec_t exec = nullptr;
    item_desc *d_items = nullptr;
    seg_desc *d_segs = nullptr;
    blk_desc *d_blks = nullptr;
    xyzz_t *d_out = nullptr;
    uint64_t last_use = 0;
    std::mutex mu;  // descriptor upload, launch and result copy stay together
    ~graph_entry()
    {
        if (exec) cudaGraphExecDestroy(exec);
        dev_free(d_items, stream);
        dev_free(d_segs, stream);
        dev_free(d_blks, stream);
        dev_free(d_out, stream);
    }
};

// The cache lives until the process exits (never destroyed: its entries
// would otherwise call into a CUDA runtime that is already shutting down).
static std::mutex g_graph_mu;
static auto &g_graphs = *new std::map<graph_key, std::shared_ptr<graph_entry>>();
static auto &g_graph_failed = *new std::set<graph_key>();
// shapes seen once: a shape is captured the second time it comes, so that
// one-off shapes (a server's changing group sizes) cost no capture
static auto &g_graph_seen = *new std::set<graph_key>();
static uint64_t g_graph_clock = 0;
static std::atomic<unsigned long long> g_graph_launches{0}, g_graph_captures{0};
static constexpr size_t kMaxGraphs = 256;
// on unless GB_MSM_GRAPHS=0 or gb_msm_graphs_enable(0)
static std::atomic<int> g_graphs_on{-1};

static bool graphs_enabled()
{
    int on = g_graphs_on.load(std::memory_order_relaxed);
    if (on < 0) {
        const char *e = getenv("GB_MSM_GRAPHS");
        on = (e && e[0] == '0') ? 0 : 1;
        g_graphs_on.store(on, std::memory_order_relaxed);
    }
    return on && !profiling_enabled();
}

// Runs the planned batch through a cached graph; false when this shape
// cannot be captured, or the device has no memory for the graph's scratch (the
// caller then launches it directly).
static bool run_planned_graph(const batch_plan &P, const affine_t *points, xyzz_t *d_out, cudaStream_t s)
{
    if (P.scratch > kGraphScratch) return false;
    graph_key key;
    key.device = current_device();
    key.stream = s;
    key.points = points;
    key.c = P.c, key.variant = P.variant, key.precomputed = P.precomputed, key.fix_by_chunk = P.fix_by_chunk;
    key.stride = P.stride, key.nitems = P.nitems, key.K = P.K, key.segs_per_item = P.segs_per_item;
    key.nseg = P.nseg, key.G = P.G, key.nblocks = P.nblocks, key.L = P.L, key.short_span = P.short_span;
    key.points_total = P.points_total, key.digits_total = P.digits_total, key.nchunks = P.nchunks;
    key.rounds = P.rounds, key.tail = P.tail.kind;

    // a stream the caller is capturing gets the launches themselves
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    GB_CUDA_OK(cudaStreamIsCapturing(s, &capturing));
    if (capturing != cudaStreamCaptureStatusNone) return false;
    std::shared_ptr<graph_entry> e;
    {
        std::lock_guard<std::mutex> lk(g_graph_mu);
        if (g_graph_failed.count(key)) return false;
        auto it = g_graphs.find(key);
        if (it != g_graphs.end()) e = it->second;
        else if (g_graph_seen.insert(key).second) {
            if (g_graph_seen.size() > 4 * kMaxGraphs) g_graph_seen.clear();
            return false;
        } else {
            // captured under the cache lock: one capture at a time, and no
            // other thread uses this key until it is in the cache
            e = std::make_shared<graph_entry>();
            e->stream = s;
            e->d_items = (item_desc *)dev_alloc(P.nitems * sizeof(item_desc), s);
            e->d_segs = (seg_desc *)dev_alloc(P.nseg * sizeof(seg_desc), s);
            e->d_blks = (blk_desc *)dev_alloc(P.nblocks * sizeof(blk_desc), s);
            e->d_out = (xyzz_t *)dev_alloc((size_t)P.nitems * P.tail.points * sizeof(xyzz_t), s);
            cudaGraph_t g = nullptr;
            if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
                (void)cudaGetLastError();
                g_graph_failed.insert(key);
                return false;
            }
            bool launched = true;
            try {
                run_planned(P, e->d_items, e->d_segs, e->d_blks, points, e->d_out, s);
            } catch (...) {
                launched = false;
            }
            const cudaError_t ec = cudaStreamEndCapture(s, &g);
            cudaError_t ei = cudaErrorUnknown;
            if (launched && ec == cudaSuccess && g) ei = cudaGraphInstantiate(&e->exec, g, 0);
            if (g) cudaGraphDestroy(g);
            if (ei != cudaSuccess) {
                (void)cudaGetLastError();
                e->exec = nullptr;
                g_graph_failed.insert(key);
                return false;
            }
            g_graph_captures++;
            if (g_graphs.size() >= kMaxGraphs) {
                auto lru = g_graphs.begin();
                for (auto j = g_graphs.begin(); j != g_graphs.end(); ++j)
                    if (j->second->last_use < lru->second->last_use) lru = j;
                g_graphs.erase(lru);
            }
            g_graphs.emplace(key, e);
        }
        e->last_use = ++g_graph_clock;
    }
    // the previous launch of this graph is on the same stream: the copies
    // into its descriptor buffers are ordered after it
    std::lock_guard<std::mutex> lk(e->mu);
    h2d(e->d_items, P.idesc.data(), P.nitems * sizeof(item_desc), s);
    h2d(e->d_segs, P.sdesc.data(), P.nseg * sizeof(seg_desc), s);
    h2d(e->d_blks, P.bdesc.data(), P.nblocks * sizeof(blk_desc), s);
    // a graph's scratch is allocated when it is launched
    const cudaError_t el = alloc_refused(P.scratch) ? cudaErrorMemoryAllocation : cudaGraphLaunch(e->exec, s);
    if (el == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();
        std::lock_guard<std::mutex> lg(g_graph_mu);
        auto it = g_graphs.find(key);
        if (it != g_graphs.end() && it->second == e) g_graphs.erase(it);
        g_graph_seen.erase(key);
        return false;
    }
    GB_CUDA_OK(el);
    GB_CUDA_OK(cudaMemcpyAsync(d_out, e->d_out, (size_t)P.nitems * P.tail.points * sizeof(xyzz_t),
                               cudaMemcpyDeviceToDevice, s));
    g_graph_launches++;
    return true;
}

// A batch's results: tail.points XYZZ points per MSM, in device memory of the
// stream the batch ran on.
struct batch_result {
    msm_tail tail;
    dev_buf<xyzz_t> points;
};

// A planned batch, or group of one, queued on s; d_out: its tail.points points
// per MSM.
static void launch_planned(const batch_plan &P, const affine_t *points, xyzz_t *d_out, cudaStream_t s, bool use_graph)
{
    if (use_graph && graphs_enabled() && run_planned_graph(P, points, d_out, s)) return;
    dev_buf<item_desc> d_items(P.nitems, s);
    dev_buf<seg_desc> d_segs(P.nseg, s);
    dev_buf<blk_desc> d_blks(P.nblocks, s);
    h2d(d_items, P.idesc.data(), P.nitems * sizeof(item_desc), s);
    h2d(d_segs, P.sdesc.data(), P.nseg * sizeof(seg_desc), s);
    h2d(d_blks, P.bdesc.data(), P.nblocks * sizeof(blk_desc), s);
    run_planned(P, d_items, d_segs, d_blks, points, d_out, s);
}

// Run a batch of MSMs, in groups if it is very large.  precomputed: `points`
// is a table of nwin rows of `stride` bases (row j = 2^(c*j) P); plain:
// `points` holds the bases.  use_graph: the bases pointer is stable across
// calls (a context's), so the batch may replay a captured graph.  A device
// without room for the affine rounds' scratch runs the batch without rounds,
// as it takes a ninth of the memory then.
static batch_result msm_run_batch(const std::vector<msm_item> &items, int c, bool precomputed, const affine_t *points,
                                  size_t stride, cudaStream_t s, bool use_graph = false)
{
    set_smem_attrs();
    batch_result r;
    for (size_t g = 0, m = 0; g < items.size(); g += m) {
        m = group_items(g, items.size(), [&](size_t i) { return items[i].n; }, c, precomputed);
        auto plan = [&](uint64_t most_scratch) {
            return plan_batch(items.data() + g, (uint32_t)m, items.size(), c, precomputed, stride, most_scratch);
        };
        const batch_plan P = plan(kRoundsScratch);
        if (!g) {
            r.tail = P.tail;
            r.points = dev_buf<xyzz_t>(items.size() * P.tail.points, s);
        }
        xyzz_t *out = r.points.get() + g * P.tail.points;
        try {
            launch_planned(P, points, out, s, use_graph);
        } catch (const cuda_error &e) {
            if (e.code() != (int)cudaErrorMemoryAllocation || !P.rounds) throw;
            launch_planned(plan(0), points, out, s, false);
        }
    }
    return r;
}

}  // namespace gb

// ---------------------------------------------------------------------------
// context + C ABI
// ---------------------------------------------------------------------------

namespace gb {

struct msm_context_t {
    int device = 0;
    size_t npoints = 0;
    RawMsmConfig config{};
    int c = 0;
    int nwin = 0;
    affine_t *table = nullptr;  // [nwin][npoints]: 2^(c*j) P_i
    cudaStream_t owner = nullptr;
    // read-only once created: calls from different lanes run concurrently,
    // each with its own stream-ordered scratch
};

static RawMsmConfig default_config(size_t npoints)
{
    uint32_t k = 0;
    size_t cap = npoints > 1 ? npoints - 1 : 0;
    while (cap) { k++; cap >>= 1; }
    RawMsmConfig c{k, 100000, 32768, 0, 3, 2, 1, 4, 0, 3};
    return c;
}

// Same acceptance rules as the reference (bls12_381_g1_msm.cu:90-110), with
// the window range widened to what this engine supports (0 = automatic).
static bool valid_config(const RawMsmConfig &c)
{
    return c.domain_k <= 31 && c.min_msm_scalars >= 1 && c.unfiltered_min_scalars >= 1 &&
           (c.window_bits == 0 || (c.window_bits >= 8 && c.window_bits <= 18)) &&
           c.sort_grid_divisor >= 1 && c.sort_grid_divisor <= 8 && c.sort_window_lanes >= 1 &&
           c.sort_window_lanes <= 4 &&
           (c.integration_blocks == 1 || c.integration_blocks == 2 || c.integration_blocks == 4 ||
            c.integration_blocks == 8 || c.integration_blocks == 16) &&
           c.batch_lanes >= 1 && c.batch_lanes <= 16 && c.reuse_event <= 1 && c.device_reduce <= 3;
}

static int plan_window(size_t n, bool precomputed, uint32_t requested)
{
    if (requested) return std::min<int>((int)requested, kMaxWindowBits);
    return choose_window(n, precomputed);
}

// Plain MSMs of host bases + host scalars [nmsms][n] (nothing resident):
// one batch through the engine.
// Autotuner for the plain path: the key is the size class of the largest
// item, the batch-size class and the sparsity of a sample of the scalars
// (zero scalars, scalars below 2^64: both empty the high windows); a new key
// times the cost model's window and a few others on this batch.
__global__ void scalar_sample_kernel(const fr_t *__restrict__ scalars, size_t n, unsigned *counts)
{
    unsigned zero = 0, small = 0;
    for (size_t i = threadIdx.x; i < n; i += blockDim.x) {
        fr_t c = scalars[i].from_mont();
        bool hi_zero = true;
#pragma unroll
        for (int k = 2; k < 8; k++) hi_zero &= c.v[k] == 0;
        if (hi_zero) {
            if (c.v[0] == 0 && c.v[1] == 0) zero++;
            else small++;
        }
    }
    atomicAdd(&counts[0], zero);
    atomicAdd(&counts[1], small);
}

static int tuned_window(const std::vector<msm_item> &items, const affine_t *points, size_t stride, cudaStream_t s)
{
    size_t n_max = 0, total = 0;
    for (const msm_item &it : items) {
        n_max = std::max(n_max, it.n);
        total += it.n;
    }
    int c = choose_window(n_max, false);
    if (!autotune_enabled() || n_max < 256) return c;
    const msm_item &first = *std::max_element(items.begin(), items.end(),
                                              [](const msm_item &a, const msm_item &b) { return a.n < b.n; });
    const size_t sample = std::min<size_t>(first.n, 4096);
    dev_buf<unsigned> counts(2, s);
    GB_CUDA_OK(cudaMemsetAsync(counts.get(), 0, 2 * sizeof(unsigned), s));
    scalar_sample_kernel<<<1, 256, 0, s>>>(first.scalars, sample, counts);
    GB_CHECK_LAUNCH();
    unsigned h[2] = {0, 0};
    d2h(h, counts, sizeof(h), s);
    lane_sync(s);
    auto cls = [&](unsigned v) { return v * 20 < sample ? 0 : (v * 10 < sample * 3 ? 1 : 2); };
    int lg = 0;
    while (((size_t)1 << (lg + 1)) <= n_max) lg++;
    const size_t nitems = items.size();
    const int bclass = nitems == 1 ? 0 : nitems <= 8 ? 1 : nitems <= 64 ? 2 : 3;
    const std::string key = "msm:2^" + std::to_string(lg) + ":b" + std::to_string(bclass) + ":z" +
                            std::to_string(cls(h[0])) + ":s" + std::to_string(cls(h[1]));
    if (autotune_lookup(key, &c)) return c;
    float best = 1e30f;
    const int model = c;
    for (int cand : {model, 8, 10, 13, 16}) {
        if (cand == model && best < 1e30f) continue;  // timed first
        if (cand > kMaxWindowBits || ((size_t)1 << (cand - 1)) > 8 * total) continue;
        float ms = time_on_stream(s, [&] { msm_run_batch(items, cand, false, points, stride, s); });
        if (ms < best) {
            best = ms;
            c = cand;
        }
    }
    autotune_store(key, c);
    return c;
}

// A plain batch over bases in device memory, results to the host.
static void plain_run_items(jacobian_t *out, const affine_t *d_points, const std::vector<msm_item> &items,
                            cudaStream_t s)
{
    const batch_result r = msm_run_batch(items, tuned_window(items, d_points, 0, s), false, d_points, 0, s);
    std::vector<xyzz_t> staging(items.size() * r.tail.points);
    d2h(staging.data(), r.points, staging.size() * sizeof(xyzz_t), s);
    lane_sync(s);
    for (size_t i = 0; i < items.size(); i++) out[i] = r.tail.finish(staging.data() + i * r.tail.points);
    timed_collect();
}

static void msm_host_plain(jacobian_t *out, const affine_t *points, const fr_t *scalars, size_t n, size_t nmsms)
{
    cudaStream_t s = lane_stream();
    dev_buf<affine_t> d_points(n, s);
    dev_buf<fr_t> d_scalars(n * nmsms, s);
    h2d(d_points, points, n * sizeof(affine_t), s);
    h2d(d_scalars, scalars, n * nmsms * sizeof(fr_t), s);
    std::vector<msm_item> items;
    for (size_t m = 0; m < nmsms; m++) items.push_back(msm_item{d_scalars.get() + m * n, n, 0});
    plain_run_items(out, d_points, items, s);
}

// Page-locked staging buffers of the asynchronous MSM calls, reused: a
// cudaFreeHost would synchronise the device, so buffers are kept until exit.
static std::mutex g_pinned_mu;
static std::multimap<size_t, xyzz_t *> g_pinned_free;

static xyzz_t *pinned_take(size_t n, size_t *cap)
{
    n = std::max<size_t>(n, 64);
    {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        auto it = g_pinned_free.lower_bound(n);
        if (it != g_pinned_free.end()) {
            *cap = it->first;
            xyzz_t *p = it->second;
            g_pinned_free.erase(it);
            return p;
        }
    }
    xyzz_t *p = nullptr;
    GB_CUDA_OK(cudaHostAlloc((void **)&p, n * sizeof(xyzz_t), cudaHostAllocPortable));
    *cap = n;
    return p;
}

static void pinned_give(xyzz_t *p, size_t cap)
{
    if (!p) return;
    std::lock_guard<std::mutex> lk(g_pinned_mu);
    g_pinned_free.emplace(cap, p);
}

// A context batch's results on their way to the host: the page-locked buffer
// they land in, and per part (the items with the precomputed table, then the
// others) what is left to do and the items' places in the batch.
struct pending_points {
    xyzz_t *staging = nullptr;
    size_t cap = 0;
    struct part {
        msm_tail tail;
        std::vector<size_t> order;
    };
    std::vector<part> parts;
    pending_points() = default;
    pending_points(const pending_points &) = delete;
    pending_points &operator=(const pending_points &) = delete;
    ~pending_points() { pinned_give(staging, cap); }
    // once the copies have landed
    void finish(jacobian_t *out) const
    {
        const xyzz_t *p = staging;
        for (const part &q : parts)
            for (size_t i : q.order) {
                out[i] = q.tail.finish(p);
                p += q.tail.points;
            }
    }
};

// A batch against the context, queued on stream s.  Large items use the
// precomputed table; small ones run as one plain batch over table row 0 (the
// bases themselves) with a window sized for them.  The results are copied to
// page-locked memory on s.
static void context_enqueue_items(msm_context_t *ctx, pending_points &pending, const std::vector<msm_item> &items,
                                  cudaStream_t s)
{
    std::vector<msm_item> sub[2];
    std::vector<size_t> idx[2];
    const size_t K = (size_t)1 << (ctx->c - 1);
    size_t between = 0, points = 0;  // items between the two ratios
    for (const msm_item &it : items)
        if (it.n * kTableMinRatio >= K && it.n * kTableRatio < K) between++, points += it.n;
    const size_t ratio = between && between > table_items(K, points / between) ? kTableRatio : kTableMinRatio;
    for (size_t i = 0; i < items.size(); i++) {
        const bool big = items[i].n * ratio >= K || items.size() == 1;
        sub[!big].push_back(items[i]);
        idx[!big].push_back(i);
    }
    batch_result r[2];
    if (!sub[0].empty()) r[0] = msm_run_batch(sub[0], ctx->c, true, ctx->table, ctx->npoints, s, true);
    if (!sub[1].empty())
        r[1] = msm_run_batch(sub[1], tuned_window(sub[1], ctx->table, 0, s), false, ctx->table, 0, s, true);
    const size_t n0 = sub[0].size() * r[0].tail.points, n1 = sub[1].size() * r[1].tail.points;
    pending.staging = pinned_take(n0 + n1, &pending.cap);
    d2h(pending.staging, r[0].points, n0 * sizeof(xyzz_t), s);
    d2h(pending.staging + n0, r[1].points, n1 * sizeof(xyzz_t), s);
    for (int k = 0; k < 2; k++) pending.parts.push_back({r[k].tail, std::move(idx[k])});
}

// The same, results to the host when it returns.
static void context_run_items(msm_context_t *ctx, jacobian_t *out_host, const std::vector<msm_item> &items,
                              cudaStream_t s)
{
    pending_points pending;
    context_enqueue_items(ctx, pending, items, s);
    lane_sync(s);
    pending.finish(out_host);
    timed_collect();
}

// An MSM batch in flight: its completion event and its results.
struct msm_ticket_t {
    int device = 0;
    uint32_t lane = 0;
    cudaEvent_t done = nullptr;
    pending_points pending;
};

static void ticket_release(msm_ticket_t *t)
{
    if (!t) return;
    if (t->done) cudaEventDestroy(t->done);
    delete t;
}

// The device address of page-locked host memory (mapped into the unified
// address space, so kernels read it over the host link), or null for
// pageable or device memory.
static const fr_t *pinned_device_view(const fr_t *p)
{
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    if (a.type != cudaMemoryTypeHost || !a.devicePointer) return nullptr;
    return reinterpret_cast<const fr_t *>(a.devicePointer);
}

static void context_run_device(msm_context_t *ctx, jacobian_t *out_host, const fr_t *d_scalars, size_t npoints,
                               size_t nmsms, cudaStream_t s)
{
    std::vector<msm_item> items;
    for (size_t m = 0; m < nmsms; m++) items.push_back(msm_item{d_scalars + m * npoints, npoints, 0});
    context_run_items(ctx, out_host, items, s);
}

}  // namespace gb

using namespace gb;

extern "C" {

// bls12_381_g1_msm.cu:6164-6200
RustError midnight_sppark_bls12_381_g1_msm(RawG1Projective *out_raw, const RawG1Affine *points_raw, const RawFr *scalars_raw, size_t len)
{
    jacobian_t *out = reinterpret_cast<jacobian_t *>(out_raw);
    const affine_t *points = reinterpret_cast<const affine_t *>(points_raw);
    const fr_t *scalars = reinterpret_cast<const fr_t *>(scalars_raw);
    GB_ENTRY_BEGIN
    if (!out || (len && (!points || !scalars)))
        return make_error((int)cudaErrorInvalidValue, "invalid BLS12-381 G1 MSM arguments");
    msm_host_plain(out, points, scalars, len, 1);
    return ok();
    GB_ENTRY_END
}

// One MSM over bases and scalars already in device memory (the caller's
// pointers, e.g. a resident SRS and a polynomial): the plain engine with
// windows combined by Horner's rule, no precomputed table, so it needs n x
// 96 bytes of bases instead of a context's nwin x n x 96.  No reference
// counterpart: the reference's resident MSMs all go through a context.
RustError gb_g1_msm_device(RawG1Projective *out_raw, const RawG1Affine *d_points_raw, const RawFr *d_scalars_raw,
                           size_t n)
{
    jacobian_t *out = reinterpret_cast<jacobian_t *>(out_raw);
    const affine_t *d_points = reinterpret_cast<const affine_t *>(d_points_raw);
    const fr_t *d_scalars = reinterpret_cast<const fr_t *>(d_scalars_raw);
    GB_ENTRY_BEGIN
    if (!out || (n && (!d_points || !d_scalars)))
        return make_error((int)cudaErrorInvalidValue, "invalid device MSM arguments");
    cudaStream_t s = lane_stream();
    plain_run_items(out, d_points, {msm_item{d_scalars, n, 0}}, s);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:6202-6245; scalars laid out [nmsms][npoints]
RustError midnight_sppark_bls12_381_g1_msm_batch(RawG1Projective *out_raw, const RawG1Affine *points_raw, const RawFr *scalars_raw, size_t npoints, size_t nmsms)
{
    jacobian_t *out = reinterpret_cast<jacobian_t *>(out_raw);
    const affine_t *points = reinterpret_cast<const affine_t *>(points_raw);
    const fr_t *scalars = reinterpret_cast<const fr_t *>(scalars_raw);
    GB_ENTRY_BEGIN
    if (nmsms == 0) return ok();
    if (!out || (npoints && (!points || !scalars)))
        return make_error((int)cudaErrorInvalidValue, "invalid BLS12-381 G1 MSM batch arguments");
    msm_host_plain(out, points, scalars, npoints, nmsms);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:6247-6267: uploads the bases once and precomputes the
// per-window shifted copies used by every later context call.
RustError midnight_sppark_bls12_381_g1_msm_context_create_with_config(void **out, const RawG1Affine *points_raw, size_t npoints, RawMsmConfig config)
{
    const affine_t *points = reinterpret_cast<const affine_t *>(points_raw);
    if (!out) return make_error((int)cudaErrorInvalidValue, "null context output");
    *out = nullptr;
    if (!valid_config(config)) return make_error((int)cudaErrorInvalidValue, "invalid BLS12-381 MSM config");
    if (npoints && !points) return make_error((int)cudaErrorInvalidValue, "null MSM bases");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    auto *ctx = new msm_context_t();
    ctx->device = current_device();
    ctx->npoints = npoints;
    ctx->config = config;
    ctx->owner = s;
    ctx->c = plan_window(npoints, true, config.window_bits);
    ctx->nwin = windows_for(ctx->c);
    try {
        size_t total = npoints * (size_t)ctx->nwin;
        if (total) {
            ctx->table = (affine_t *)dev_malloc(total * sizeof(affine_t));
            h2d(ctx->table, points, npoints * sizeof(affine_t), s);
            msm_precompute_kernel<<<blocks_for(npoints, 128), 128, 0, s>>>(ctx->table, npoints, ctx->c,
                                                                           ctx->nwin);
            GB_CHECK_LAUNCH();
        }
        lane_sync(s);
    } catch (...) {
        if (ctx->table) cudaFree(ctx->table);
        delete ctx;
        throw;
    }
    *out = ctx;
    return ok();
    GB_ENTRY_END
}

RustError midnight_sppark_bls12_381_g1_msm_context_create(void **out, const RawG1Affine *points_raw, size_t npoints)
{
    return midnight_sppark_bls12_381_g1_msm_context_create_with_config(out, points_raw, npoints,
                                                                       default_config(npoints));
}

// Device bytes a context holds: its table of nwin x npoints affine points
// (the bases shifted by each window).  No reference counterpart.
size_t gb_g1_msm_context_device_bytes(const void *context)
{
    auto *ctx = reinterpret_cast<const msm_context_t *>(context);
    return ctx ? ctx->npoints * (size_t)ctx->nwin * sizeof(affine_t) : 0;
}

void midnight_sppark_bls12_381_g1_msm_context_free(void *context)
{
    auto *ctx = reinterpret_cast<msm_context_t *>(context);
    if (!ctx) return;
    cudaStreamSynchronize(ctx->owner);
    if (ctx->table) cudaFree(ctx->table);
    delete ctx;
}

// bls12_381_g1_msm.cu:6288-6308: host scalars against resident bases
RustError midnight_sppark_bls12_381_g1_msm_context_batch(RawG1Projective *out_raw, void *context, const RawFr *scalars_raw, size_t npoints, size_t nmsms)
{
    jacobian_t *out = reinterpret_cast<jacobian_t *>(out_raw);
    const fr_t *scalars = reinterpret_cast<const fr_t *>(scalars_raw);
    if (!context) return make_error(-1, "null BLS12-381 G1 MSM context");
    GB_ENTRY_BEGIN
    auto *ctx = reinterpret_cast<msm_context_t *>(context);
    if (nmsms == 0) return ok();
    if (!out || (npoints && !scalars)) return make_error((int)cudaErrorInvalidValue, "invalid MSM batch arguments");
    if (npoints > ctx->npoints) return make_error((int)cudaErrorInvalidValue, "more scalars than context bases");
    cudaStream_t s = lane_stream();
    // page-locked host scalars are read in place by the recode kernel over
    // the host link, with no staging copy; pageable ones are staged
    if (const fr_t *view = pinned_device_view(scalars)) {
        count_transfer(true, npoints * nmsms * sizeof(fr_t));
        context_run_device(ctx, out, view, npoints, nmsms, s);
        return ok();
    }
    dev_buf<fr_t> d_scalars(npoints * nmsms, s);
    h2d(d_scalars, scalars, npoints * nmsms * sizeof(fr_t), s);
    context_run_device(ctx, out, d_scalars, npoints, nmsms, s);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:6310-6344: resident scalars (device vector)
RustError midnight_sppark_bls12_381_g1_msm_context_device_batch(RawG1Projective *out_raw, void *context, const void *device_vec, size_t scalar_offset, size_t npoints, size_t nmsms)
{
    jacobian_t *out = reinterpret_cast<jacobian_t *>(out_raw);
    if (!context || !device_vec || (nmsms != 0 && !out))
        return make_error(-1, "invalid resident BLS12-381 G1 MSM arguments");
    GB_ENTRY_BEGIN
    auto *ctx = reinterpret_cast<msm_context_t *>(context);
    auto *dv = reinterpret_cast<const fr_device_vec *>(device_vec);
    if (npoints != 0 && nmsms > (SIZE_MAX - scalar_offset) / npoints)
        return make_error((int)cudaErrorInvalidValue, "resident MSM range overflow");
    if (scalar_offset + npoints * nmsms > dv->len)
        return make_error((int)cudaErrorInvalidValue, "resident MSM range exceeds device vector");
    if (npoints > ctx->npoints) return make_error((int)cudaErrorInvalidValue, "more scalars than context bases");
    if (nmsms == 0) return ok();
    cudaStream_t s = lane_stream();
    device_vec_wait(dv, s);
    context_run_device(ctx, out, dv->values + scalar_offset, npoints, nmsms, s);
    return ok();
    GB_ENTRY_END
}

// The resident batch of midnight_sppark_bls12_381_g1_msm_context_device_batch,
// queued on the calling lane and returned at once: *ticket is completed by
// gb_msm_ticket_wait, which waits for the batch and writes its points.  The
// host can queue further work on the lane meanwhile (work that does not
// need the points), so the device is not left idle while the host waits for
// them.  No reference counterpart (the reference's calls return the points).
RustError gb_g1_msm_context_device_batch_async(void **ticket, void *context, const void *device_vec,
                                               size_t scalar_offset, size_t npoints, size_t nmsms)
{
    if (!ticket) return make_error((int)cudaErrorInvalidValue, "null MSM ticket output");
    *ticket = nullptr;
    if (!context || !device_vec) return make_error(-1, "invalid resident BLS12-381 G1 MSM arguments");
    GB_ENTRY_BEGIN
    auto *ctx = reinterpret_cast<msm_context_t *>(context);
    auto *dv = reinterpret_cast<const fr_device_vec *>(device_vec);
    if (npoints != 0 && nmsms > (SIZE_MAX - scalar_offset) / npoints)
        return make_error((int)cudaErrorInvalidValue, "resident MSM range overflow");
    if (scalar_offset + npoints * nmsms > dv->len)
        return make_error((int)cudaErrorInvalidValue, "resident MSM range exceeds device vector");
    if (npoints > ctx->npoints) return make_error((int)cudaErrorInvalidValue, "more scalars than context bases");
    cudaStream_t s = lane_stream();
    auto *t = new msm_ticket_t();
    try {
        t->device = current_device();
        t->lane = current_lane();
        GB_CUDA_OK(cudaEventCreateWithFlags(&t->done, cudaEventDisableTiming));
        if (nmsms) {
            device_vec_wait(dv, s);
            std::vector<msm_item> items;
            for (size_t m = 0; m < nmsms; m++)
                items.push_back(msm_item{dv->values + scalar_offset + m * npoints, npoints, 0});
            context_enqueue_items(ctx, t->pending, items, s);
        }
        GB_CUDA_OK(cudaEventRecord(t->done, s));
    } catch (...) {
        ticket_release(t);
        throw;
    }
    *ticket = t;
    return ok();
    GB_ENTRY_END
}

// Graph replay of context batches on (1) or off (0); the counters give the
// graphs captured and the batches replayed since the process started.
RustError gb_msm_graphs_enable(int on)
{
    gb::g_graphs_on.store(on ? 1 : 0, std::memory_order_relaxed);
    return ok();
}

RustError gb_msm_graph_stats(unsigned long long *captures, unsigned long long *launches)
{
    if (!captures || !launches) return make_error((int)cudaErrorInvalidValue, "null graph counter output");
    *captures = gb::g_graph_captures.load();
    *launches = gb::g_graph_launches.load();
    return ok();
}

// Waits for the batch of `ticket`, writes its points to out (nmsms of them,
// in batch order; out may be null to discard them) and releases the ticket,
// which must not be used again.  A wait that ran out in the lane's NTT work
// since its previous synchronisation is reported here, as by the lane's
// synchronising calls.
RustError gb_msm_ticket_wait(void *ticket, RawG1Projective *out_raw)
{
    auto *t = reinterpret_cast<msm_ticket_t *>(ticket);
    if (!t) return make_error((int)cudaErrorInvalidValue, "null MSM ticket");
    jacobian_t *out = reinterpret_cast<jacobian_t *>(out_raw);
    GB_ENTRY_BEGIN
    const cudaError_t e = cudaEventSynchronize(t->done);
    if (e != cudaSuccess) {
        ticket_release(t);
        return make_error((int)e, cudaGetErrorString(e));
    }
    int prev_dev = 0;
    GB_CUDA_OK(cudaGetDevice(&prev_dev));
    const uint32_t prev_lane = current_lane();
    try {
        if (prev_dev != t->device) GB_CUDA_OK(cudaSetDevice(t->device));
        set_lane(t->lane);
        lane_check();
    } catch (...) {
        set_lane(prev_lane);
        cudaSetDevice(prev_dev);
        ticket_release(t);
        throw;
    }
    set_lane(prev_lane);
    if (prev_dev != t->device) GB_CUDA_OK(cudaSetDevice(prev_dev));
    if (out) t->pending.finish(out);
    ticket_release(t);
    timed_collect();
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:6346-6377: ragged slices of one device vector
RustError midnight_sppark_bls12_381_g1_msm_context_device_ragged(RawG1Projective *out_raw, void *context, const void *device_vec, const RawMsmSlice *slices, size_t count)
{
    jacobian_t *out = reinterpret_cast<jacobian_t *>(out_raw);
    if (!context || !device_vec || (count != 0 && (!out || !slices)))
        return make_error(-1, "invalid ragged resident BLS12-381 G1 MSM arguments");
    if (count == 0) return ok();
    GB_ENTRY_BEGIN
    auto *ctx = reinterpret_cast<msm_context_t *>(context);
    auto *dv = reinterpret_cast<const fr_device_vec *>(device_vec);
    for (size_t i = 0; i < count; i++) {
        const RawMsmSlice &sl = slices[i];
        if (sl.scalar_offset > dv->len || sl.len > dv->len - sl.scalar_offset)
            return make_error((int)cudaErrorInvalidValue, "ragged MSM slice exceeds device vector");
        if (sl.point_offset > ctx->npoints || sl.len > ctx->npoints - sl.point_offset)
            return make_error((int)cudaErrorInvalidValue, "ragged MSM slice exceeds context bases");
    }
    cudaStream_t s = lane_stream();
    device_vec_wait(dv, s);
    std::vector<msm_item> items;
    for (size_t i = 0; i < count; i++)
        items.push_back(msm_item{dv->values + slices[i].scalar_offset, slices[i].len, slices[i].point_offset});
    context_run_items(ctx, out, items, s);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:6379-6404 (test hooks): a delay for the next
// scrambled batches' mask producer on this thread; the masked scalars are
// zeroed and the stream held back before the mask is added, so that an MSM
// that did not wait for them would read zeros
static thread_local uint32_t t_mask_delay_ms = 0;

void midnight_sppark_test_mask_delay(uint32_t delay_ms)
{
    t_mask_delay_ms = delay_ms;
}

// bls12_381_g1_msm.cu:6426-6486: MSM of (scalars + mask) for each batch
// entry; the caller subtracts its precomputed MSM(mask, bases)
// (midnight-sppark-msm/src/lib.rs:3302-3354).
RustError midnight_sppark_bls12_381_g1_msm_context_device_scrambled_batch(RawG1Projective *out_raw, void *context,
                                                                          const void *device_vec,
                                                                          size_t scalar_offset, size_t npoints,
                                                                          size_t nmsms, const void *mask_device_vec)
{
    jacobian_t *out = reinterpret_cast<jacobian_t *>(out_raw);
    if (!context || !device_vec || !mask_device_vec || (nmsms != 0 && !out))
        return make_error(-1, "invalid scrambled resident BLS12-381 G1 MSM arguments");
    GB_ENTRY_BEGIN
    auto *ctx = reinterpret_cast<msm_context_t *>(context);
    auto *dv = reinterpret_cast<const fr_device_vec *>(device_vec);
    auto *mv = reinterpret_cast<const fr_device_vec *>(mask_device_vec);
    if (mv->len != npoints) return make_error((int)cudaErrorInvalidValue, "resident MSM scramble mask length mismatch");
    if (npoints != 0 && nmsms > (SIZE_MAX - scalar_offset) / npoints)
        return make_error((int)cudaErrorInvalidValue, "scrambled resident MSM range overflow");
    const size_t count = npoints * nmsms;
    if (scalar_offset + count > dv->len)
        return make_error((int)cudaErrorInvalidValue, "scrambled resident MSM range exceeds device vector");
    if (npoints > ctx->npoints) return make_error((int)cudaErrorInvalidValue, "more scalars than context bases");
    if (count == 0) return ok();
    cudaStream_t s = lane_stream();
    device_vec_wait(dv, s);
    device_vec_wait(mv, s);
    dev_buf<fr_t> masked(count, s);
    if (t_mask_delay_ms) {
        GB_CUDA_OK(cudaMemsetAsync(masked.get(), 0, count * sizeof(fr_t), s));
        lane_sync(s);
        stream_host_delay(s, t_mask_delay_ms);
    }
    add_mask_kernel<<<blocks_for(count, 256), 256, 0, s>>>(masked, dv->values + scalar_offset, mv->values, npoints,
                                                           count);
    GB_CHECK_LAUNCH();
    context_run_device(ctx, out, masked, npoints, nmsms, s);
    return ok();
    GB_ENTRY_END
}

}  // extern "C"
