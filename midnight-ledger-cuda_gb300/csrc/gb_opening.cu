// KZG opening helpers on the device: batched polynomial evaluation at a
// point (midnight-sppark-msm/src/bls12_381_g1_msm.cu:3985-4031,
// midnight_sppark_bls12_381_fr_device_eval_polys) and the Kate quotient
// (f(X) - f(z)) / (X - z) of every polynomial of a batch (the division the
// reference's multi-open computes with its kate scan, .cu:1923-1959).
//
// Evaluation and division are Horner's rule in blocks: every thread runs it
// over a few coefficients, and the threads' values meet in log steps with the
// powers z^(2^s), which are squarings.  No power of z is tabulated and 1 / z
// is not needed.  With tables and a suffix sum, a quotient of 2^12 coefficients
// was ten launches of 80 us together; now it is two.  A proof of 2^12 rows
// takes 3.32 ms instead of 3.94 with that, one of 2^16 rows 9.96.
#include <algorithm>
#include <vector>

#include "gb_vec.cuh"

namespace gb {

static constexpr int kEvalThreads = 256;  // 2^8

// The loops around products stay loops (unroll 1): these kernels run for
// microseconds from a cold instruction cache, and a product is 5 KB of code
// (40 polynomials of 2^12 coefficients: 37 us unrolled, 26 as loops).

// the value of the lane `off` further up in a full warp
__device__ __forceinline__ fr_t lane_down(const fr_t &a, unsigned off)
{
    fr_t r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_down_sync(0xffffffffu, a.v[i], off);
    return r;
}

// an evaluation: len coefficients at polys, at points[row]
struct eval_pair {
    const fr_t *polys;
    uint32_t row;
};

// One slice of T * per coefficients (T = 2^LOG_T threads, per a multiple of 4)
// of one polynomial a block: out[p * slices + slice] = its value at y =
// points[row]^(2^squarings).  Thread t runs Horner's rule in y^T over the
// coefficients t, t + T, .. of the slice, then the threads are folded by
// y^(T/2), .. y.  With T = 256 and per = 16 a chain of 16 + per dependent products
// bounds it, so the coefficients are read 4 ahead and one warp has the powers
// ready (40 polynomials of 2^12 coefficients 48 -> 26 us, of 2^16 87 -> 45).  T =
// 32 is for many or short polynomials, which are bound by the products that do
// not depend on their length: no warp is idle in the folds.  Given flat,
// polynomial p lies at flat + p * len; without pairs all are evaluated at the
// first point.  With `ready` the points come with their powers y^(2^s), s = 0 ..
// LOG_T.
template <int LOG_T>
__global__ void __launch_bounds__(1 << LOG_T) eval_slices_kernel(const eval_pair *__restrict__ pairs,
                                                                 const fr_t *__restrict__ flat, size_t len,
                                                                 const fr_t *__restrict__ points, bool ready,
                                                                 int squarings, int per, uint32_t slices,
                                                                 fr_t *__restrict__ out)
{
    constexpr size_t T = 1 << LOG_T;
    __shared__ fr_t sh[T], pw[LOG_T + 1];  // pw[s] = y^(2^s)
    const size_t p = blockIdx.y, lo = (size_t)blockIdx.x * per * T, t = threadIdx.x;
    const eval_pair e = pairs ? pairs[p] : eval_pair{nullptr, 0};
    const fr_t *c = (flat ? flat + p * len : e.polys) + lo + t;
    const size_t left = lo + t < len ? len - (lo + t) : 0, row = min(len - lo, T);  // row: threads with coefficients
    auto load = [&](fr_t *v, int k) {  // coefficients k .. k + 3 of the thread
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = (size_t)(k + u) * T < left ? c[(size_t)(k + u) * T] : fr_t::zero();
    };
    fr_t now[4], next[4];
    load(now, per - 4);
    if (ready) {
        if (t <= LOG_T) pw[t] = points[e.row * (LOG_T + 1) + t];
    } else if (t < 32) {
        fr_t y = points[e.row];
#pragma unroll 1
        for (int k = 0; k < squarings; k++) y = y.sqr();
#pragma unroll 1
        for (int k = 0; k <= LOG_T && (len - lo > T || ((size_t)1 << k) < row); k++) {
            if (t == 0) pw[k] = y;
            if (k < LOG_T) y = y.sqr();
        }
    }
    __syncthreads();
    const fr_t y = pw[LOG_T];
    fr_t acc = fr_t::zero();
    bool any = false;  // conditions on these rows are the same for the block
    for (int k = per - 4; k >= 0; k -= 4) {
        if (k) load(next, k - 4);
#pragma unroll
        for (int u = 3; u >= 0; u--) {
            if (lo + (size_t)(k + u) * T >= len) continue;
            if (any) acc = acc * y;
            acc = acc + now[u];
            any = true;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) now[u] = next[u];
    }
    sh[t] = acc;
#pragma unroll 1
    for (int k = LOG_T - 1; k >= 5; k--) {
        __syncthreads();
        if (t < (1u << k)) sh[t] = sh[t] + sh[t + (1u << k)] * pw[k];
    }
    if (t >= 32) return;
    acc = sh[t];
#pragma unroll 1
    for (int k = 4; k >= 0; k--)
        if ((1u << k) < row) acc = acc + lane_down(acc, 1u << k) * pw[k];
    if (t == 0) out[p * slices + blockIdx.x] = acc;
}

// Values of `total` polynomials of len coefficients into d_out: pair p's at its
// point, or, without pairs (null), those in a row at `flat` at points[0]; on the
// host: npoints points.  The slices' values are the coefficients of a polynomial
// in point^slice, evaluated the same way.
static void eval_pairs(fr_t *d_out, const std::vector<eval_pair> *pairs, const fr_t *flat, size_t total,
                       const RawFr *points, size_t npoints, size_t len, cudaStream_t s)
{
    const size_t chunk = 65535;  // grid.y limit
    if (!total) return;
    if (npoints > 65535 && len <= ((size_t)1 << 24))
        throw cuda_error((int)cudaErrorInvalidValue, "too many evaluation points");
    // A warp a polynomial for short ones and for many (measured, us with 256
    // threads and with a warp: 1000 polynomials of 256 coefficients 84 35, 20000
    // 1146 186, 40 of 512 35 36, of 1024 35 45; 600 of 2048 72 70, 1000 of 4096 146
    // 133)
    const bool warps = len <= 512 || (len <= 4096 && total >= 456) || (len <= 6144 && total >= 1000);
    // points of many polynomials each: their powers made here, once
    const bool ready = warps && npoints * 16 <= total;
    dev_buf<fr_t> d_points(npoints * (ready ? 6 : 1), s);
    if (ready) {
        std::vector<fr_t> powers(npoints * 6);
        for (size_t q = 0; q < npoints; q++) {
            powers[6 * q] = from_raw(points[q]);
            for (int k = 1; k < 6; k++) powers[6 * q + k] = powers[6 * q + k - 1].sqr();
        }
        h2d(d_points, powers.data(), powers.size() * sizeof(fr_t), s);
    } else {
        h2d(d_points, points, npoints * sizeof(fr_t), s);
    }
    dev_buf<eval_pair> d_pairs(pairs ? total : 0, s);
    if (pairs) h2d(d_pairs, pairs->data(), total * sizeof(eval_pair), s);
    dev_buf<fr_t> values;
    // Coefficients a thread: up to 64 where that leaves two waves of blocks, or
    // covers the polynomial and there are many, which spares the products of the
    // squarings and folds (2000 polynomials of 8192 coefficients 650 -> 407 us);
    // else 16, to be short
    auto blocks = [&](int log) { return total * ((len + ((size_t)kEvalThreads << log) - 1) >> (8 + log)); };
    int log_per = 4;
    while (log_per < 6 && len > (size_t)kEvalThreads << log_per &&
           (blocks(log_per + 1) >= 608 || (total >= 304 && len <= (size_t)kEvalThreads << 6)))
        log_per++;
    for (int squarings = 0;; squarings += 8 + log_per) {
        const size_t slice = warps ? len : (size_t)kEvalThreads << log_per;
        const uint32_t slices = (uint32_t)((len + slice - 1) / slice);
        dev_buf<fr_t> next(slices > 1 ? total * slices : 0, s);
        fr_t *out = slices > 1 ? next.get() : d_out;
        for (size_t b = 0; b < total; b += chunk) {
            const eval_pair *dp = pairs ? d_pairs.get() + b : nullptr;
            const fr_t *df = flat ? flat + b * len : nullptr;
            const dim3 grid(slices, (unsigned)std::min(chunk, total - b));
            if (warps)
                eval_slices_kernel<5><<<grid, 32, 0, s>>>(dp, df, len, d_points, ready, 0,
                                                          (int)((len + 127) / 128 * 4), 1, out + b);
            else
                eval_slices_kernel<8><<<grid, kEvalThreads, 0, s>>>(dp, df, len, d_points, false, squarings,
                                                                    1 << log_per, slices, out + b * slices);
            GB_CHECK_LAUNCH();
        }
        if (slices == 1) return;
        len = slices;
        values = std::move(next);
        flat = values;
    }
}

static void eval_polys(fr_t *d_out, const fr_t *polys, size_t len, size_t count, const RawFr &z, cudaStream_t s)
{
    eval_pairs(d_out, nullptr, polys, count, &z, 1, len, s);
}

// Kate quotient.  With the coefficients taken from the top, a_t =
// f_(len-1-t), Horner's values H_t = a_t + z H_(t-1) are the quotient:
// q_(len-2-t) = H_t, and q_(len-1) = 0.  A tile is 256 threads of PER
// coefficients; a first launch leaves every tile's last H, as if the tile were
// the first one, a second launch adds what the tiles before bring and writes q.
// grid.y divisions in a launch, each with its own polynomial and point.
struct kate_item {
    const fr_t *f;
    fr_t *q;
    const fr_t *z;  // z^(2^s) for s < kKatePowers
};
static constexpr int kKatePowers = 48;
static constexpr int kKateLog = 8;  // log2 of the threads
static constexpr int kKateThreads = 1 << kKateLog;

// Horner's rule over a thread's coefficients from v on
template <int LOG_PER>
__device__ __forceinline__ fr_t kate_thread(const fr_t *f, size_t len, size_t base, const fr_t &z, fr_t v)
{
#pragma unroll
    for (int e = 0; e < 1 << LOG_PER; e++) {
        v = v * z;
        if (base + e < len) v = v + f[len - 1 - (base + e)];
    }
    return v;
}

template <int LOG_PER>
__global__ void __launch_bounds__(kKateThreads) kate_tile_kernel(const kate_item *__restrict__ items, size_t len,
                                                                 fr_t *__restrict__ totals)
{
    __shared__ fr_t sh[kKateThreads];
    const unsigned t = threadIdx.x;
    const kate_item it = items[blockIdx.y];
    const size_t base = ((size_t)blockIdx.x * kKateThreads + t) << LOG_PER;
    sh[t] = kate_thread<LOG_PER>(it.f, len, base, it.z[0], fr_t::zero());
    for (int k = 0; k < kKateLog; k++) {
        const unsigned off = 1u << k;
        __syncthreads();
        if ((t & (2 * off - 1)) == 2 * off - 1) sh[t] = sh[t] + sh[t - off] * it.z[LOG_PER + k];
    }
    if (t == kKateThreads - 1) totals[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = sh[t];
}

// inclusive scan of the recurrence over a block: thread t's value is left as
// sum_u z^(2^log_step u) sh[t - u]
__device__ __forceinline__ void kate_block_scan(fr_t *sh, const fr_t *z, int log_step)
{
    const unsigned t = threadIdx.x;
    for (int k = 0; k < kKateLog; k++) {
        const unsigned off = 1u << k;
        __syncthreads();
        const fr_t other = t >= off ? sh[t - off] * z[log_step + k] : fr_t::zero();
        __syncthreads();
        if (t >= off) sh[t] = sh[t] + other;
    }
    __syncthreads();
}

// what the tiles before each one bring to it, in place of the totals; one
// block a division, 2^log_m tiles a thread
__global__ void __launch_bounds__(kKateThreads) kate_carry_kernel(const kate_item *__restrict__ items,
                                                                  fr_t *__restrict__ totals, size_t tiles,
                                                                  int log_tile, int log_m)
{
    __shared__ fr_t sh[kKateThreads];
    fr_t *T = totals + (size_t)blockIdx.x * tiles;
    const fr_t *z = items[blockIdx.x].z;
    const unsigned t = threadIdx.x;
    const size_t lo = (size_t)t << log_m, end = lo + ((size_t)1 << log_m);
    fr_t v = fr_t::zero();
    for (size_t b = lo; b < end; b++) {
        v = v * z[log_tile];
        if (b < tiles) v = v + T[b];
    }
    sh[t] = v;
    kate_block_scan(sh, z, log_tile + log_m);
    v = t ? sh[t - 1] : fr_t::zero();
    for (size_t b = lo; b < end && b < tiles; b++) {
        const fr_t own = T[b];
        T[b] = v;
        v = v * z[log_tile] + own;
    }
}

template <int LOG_PER>
__global__ void __launch_bounds__(kKateThreads) kate_apply_kernel(const kate_item *__restrict__ items, size_t len,
                                                                  const fr_t *__restrict__ totals, bool carried)
{
    __shared__ fr_t sh[kKateThreads];
    const unsigned t = threadIdx.x, b = blockIdx.x;
    const kate_item it = items[blockIdx.y];
    const fr_t *T = totals + (size_t)blockIdx.y * gridDim.x;
    const size_t base = ((size_t)b * kKateThreads + t) << LOG_PER;
    fr_t carry = fr_t::zero();
    if (carried) {
        carry = T[b];
    } else if (b) {
        // the at most 255 tiles before: sum_u z^(tile u) T[b - 1 - u]
        sh[t] = t < b ? T[b - 1 - t] : fr_t::zero();
        for (int k = kKateLog - 1; k >= 0; k--) {
            __syncthreads();
            if (t < (1u << k)) sh[t] = sh[t] + sh[t + (1u << k)] * it.z[kKateLog + LOG_PER + k];
        }
        __syncthreads();
        carry = sh[0];
        __syncthreads();
    }
    sh[t] = kate_thread<LOG_PER>(it.f, len, base, it.z[0], t ? fr_t::zero() : carry);
    kate_block_scan(sh, it.z, LOG_PER);
    fr_t h = t ? sh[t - 1] : carry;  // Horner's value before the thread's coefficients
#pragma unroll
    for (int e = 0; e < 1 << LOG_PER; e++) {
        const size_t i = base + e;
        if (i >= len) break;
        h = h * it.z[0] + it.f[len - 1 - i];
        if (i + 1 < len) it.q[len - 2 - i] = h;
        else it.q[len - 1] = fr_t::zero();
    }
}

static std::vector<fr_t> kate_powers(const fr_t *points, size_t n)
{
    std::vector<fr_t> z(n * kKatePowers);
    for (size_t p = 0; p < n; p++) {
        z[p * kKatePowers] = points[p];
        for (int k = 1; k < kKatePowers; k++) z[p * kKatePowers + k] = z[p * kKatePowers + k - 1].sqr();
    }
    return z;
}

template <int LOG_PER>
static void kate_divide_tiled(const kate_item *d_items, size_t count, size_t len, cudaStream_t s)
{
    constexpr int log_tile = kKateLog + LOG_PER;
    const size_t tiles = (len + ((size_t)1 << log_tile) - 1) >> log_tile;
    int log_m = 0;
    while (((size_t)kKateThreads << log_m) < tiles) log_m++;
    if (tiles > 0x7fffffff || log_tile + log_m + kKateLog > kKatePowers)
        throw cuda_error((int)cudaErrorInvalidValue, "Kate division too long");
    constexpr size_t kMaxY = 65535;
    dev_buf<fr_t> totals(tiles * std::min(count, kMaxY), s);
    for (size_t p = 0; p < count; p += kMaxY, d_items += kMaxY) {
        const unsigned m = (unsigned)std::min(kMaxY, count - p);
        if (tiles > 1) {
            kate_tile_kernel<LOG_PER><<<dim3((unsigned)tiles, m), kKateThreads, 0, s>>>(d_items, len, totals);
            GB_CHECK_LAUNCH();
        }
        if (log_m) {
            kate_carry_kernel<<<m, kKateThreads, 0, s>>>(d_items, totals, tiles, log_tile, log_m);
            GB_CHECK_LAUNCH();
        }
        kate_apply_kernel<LOG_PER><<<dim3((unsigned)tiles, m), kKateThreads, 0, s>>>(d_items, len, totals, log_m > 0);
        GB_CHECK_LAUNCH();
    }
}

// divisions of polynomials of len coefficients; an item's q and f don't overlap
static void kate_divide_items(const kate_item *d_items, size_t count, size_t len, cudaStream_t s)
{
    if (!len || !count) return;
    // a coefficient a thread is the shortest chain and most products (the scan's
    // 12 a warp); more coefficients share the scan (measured, us a call with 1,
    // 2, 4, 8: 2^12 coefficients 40* 40 40 40, 3 x 2^14 52 45* 58 74, 2^16 51
    // 46* 58 74, 3 x 2^16 105 74* 82 74, 2^18 133 100 82 75*, 3 x 2^20 1060 655
    // 561 504*)
    const size_t total = len * count;
    if (total <= (size_t)1 << 14) kate_divide_tiled<0>(d_items, count, len, s);
    else if (total <= (size_t)3 << 16) kate_divide_tiled<1>(d_items, count, len, s);
    else kate_divide_tiled<3>(d_items, count, len, s);
}

// the quotients by X
__global__ void shift_down_kernel(const fr_t *__restrict__ f, size_t len, size_t total, fr_t *__restrict__ q)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < total) q[t] = t % len + 1 < len ? f[t + 1] : fr_t::zero();
}

// count polynomials in a row, divided by X - z; d_out and f don't overlap.  By
// X it is a copy (2^20 coefficients 40 us, by Horner's rule 221).
static void kate_divide(fr_t *d_out, const fr_t *f, size_t len, size_t count, const fr_t &z, cudaStream_t s)
{
    if (z.is_zero()) {
        shift_down_kernel<<<blocks_for(len * count, 256), 256, 0, s>>>(f, len, len * count, d_out);
        GB_CHECK_LAUNCH();
        return;
    }
    const std::vector<fr_t> powers = kate_powers(&z, 1);
    dev_buf<fr_t> d_powers(powers.size(), s);
    h2d(d_powers, powers.data(), powers.size() * sizeof(fr_t), s);
    std::vector<kate_item> items(count);
    for (size_t p = 0; p < count; p++) items[p] = kate_item{f + p * len, d_out + p * len, d_powers.get()};
    dev_buf<kate_item> d_items(count, s);
    h2d(d_items, items.data(), count * sizeof(kate_item), s);
    kate_divide_items(d_items, count, len, s);
}

// q[k][i] = sum over the items t of q k (q_offsets[k] <= t < q_offsets[k+1])
// of coeffs[t] * poly(item_polys[t])[i]; polynomials through a pointer table
__global__ void multiopen_q_kernel(fr_t *__restrict__ out, const fr_t *const *__restrict__ polys,
                                   const uint32_t *__restrict__ q_offsets, const uint32_t *__restrict__ item_polys,
                                   const fr_t *__restrict__ coeffs, size_t len, size_t q_count)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= len * q_count) return;
    const size_t k = t / len, i = t - k * len;
    fr_t acc = fr_t::zero();
    for (uint32_t it = q_offsets[k]; it < q_offsets[k + 1]; it++) acc = acc + polys[item_polys[it]][i] * coeffs[it];
    out[t] = acc;
}

// out[i] = sum_p k[p] * polys[p][i], polynomials through a pointer table
__global__ void lincomb_table_kernel(fr_t *__restrict__ out, const fr_t *const *__restrict__ polys,
                                     const fr_t *__restrict__ k, size_t len, size_t count)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= len) return;
    fr_t acc = fr_t::zero();
    for (size_t p = 0; p < count; p++) acc = acc + polys[p][i] * k[p];
    out[i] = acc;
}

// checks of the q description shared by both preparation entry points
static const char *check_q_layout(const uint32_t *q_offsets, size_t q_offsets_len, const uint32_t *q_poly_indices,
                                  size_t q_items_len, size_t poly_count, const uint32_t *query_poly_indices,
                                  const uint32_t *query_point_indices, size_t query_count, size_t point_count)
{
    const size_t q_count = q_offsets_len - 1;
    if (q_offsets[0] != 0 || q_offsets[q_count] != q_items_len) return "invalid multi-open q offsets";
    for (size_t k = 0; k < q_count; k++)
        if (q_offsets[k] > q_offsets[k + 1]) return "non-monotonic multi-open q offsets";
    for (size_t t = 0; t < q_items_len; t++)
        if (q_poly_indices[t] >= poly_count) return "multi-open q polynomial index out of range";
    for (size_t r = 0; r < query_count; r++)
        if (query_poly_indices[r] >= poly_count || query_point_indices[r] >= point_count)
            return "multi-open query index out of range";
    return nullptr;
}

// the q polynomials into d_q and the query evaluations into d_eval, the
// polynomials named by a host table of device pointers
static void multiopen_prepare_core(fr_t *d_q, fr_t *d_eval, const std::vector<const fr_t *> &polys, size_t len,
                                   const uint32_t *q_offsets, size_t q_offsets_len, const uint32_t *q_poly_indices,
                                   const RawFr *q_coefficients, size_t q_items_len, const RawFr *points,
                                   size_t point_count, const uint32_t *query_poly_indices,
                                   const uint32_t *query_point_indices, size_t query_count, cudaStream_t s)
{
    const size_t q_count = q_offsets_len - 1;
    dev_buf<const fr_t *> d_polys(polys.size(), s);
    dev_buf<uint32_t> d_offsets(q_offsets_len, s), d_items(q_items_len, s);
    dev_buf<fr_t> d_coeffs(q_items_len, s);
    h2d(d_polys, polys.data(), polys.size() * sizeof(const fr_t *), s);
    h2d(d_offsets, q_offsets, q_offsets_len * sizeof(uint32_t), s);
    h2d(d_items, q_poly_indices, q_items_len * sizeof(uint32_t), s);
    h2d(d_coeffs, q_coefficients, q_items_len * sizeof(fr_t), s);
    if (q_count) {
        multiopen_q_kernel<<<blocks_for(len * q_count, 256), 256, 0, s>>>(d_q, d_polys, d_offsets, d_items, d_coeffs,
                                                                           len, q_count);
        GB_CHECK_LAUNCH();
    }
    std::vector<eval_pair> pairs(query_count);
    for (size_t r = 0; r < query_count; r++) pairs[r] = eval_pair{polys[query_poly_indices[r]], query_point_indices[r]};
    eval_pairs(d_eval, &pairs, nullptr, query_count, points, point_count, len, s);
}

}  // namespace gb

using namespace gb;

extern "C" {

// bls12_381_g1_msm.cu:3985-4031: out[p] = sum_i polys[p][i] * point^i
RustError midnight_sppark_bls12_381_fr_device_eval_polys(RawFr *out_raw, const void *device_vec, size_t poly_len,
                                                         size_t poly_count, RawFr point_raw)
{
    if (!out_raw || !device_vec || poly_len == 0 || poly_count == 0 || poly_count > SIZE_MAX / poly_len)
        return make_error((int)cudaErrorInvalidValue, "invalid resident polynomial evaluation arguments");
    GB_ENTRY_BEGIN
    auto *v = reinterpret_cast<const fr_device_vec *>(device_vec);
    if (v->len != poly_len * poly_count)
        return make_error((int)cudaErrorInvalidValue, "resident polynomial evaluation shape mismatch");
    cudaStream_t s = lane_stream();
    device_vec_wait(v, s);
    dev_buf<fr_t> d(poly_count, s);
    eval_polys(d, v->values, poly_len, poly_count, point_raw, s);
    d2h(out_raw, d, poly_count * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

// Several evaluations in one call (no reference counterpart: the reference
// makes one midnight_sppark_bls12_381_fr_device_eval_polys call per point).
// Request r evaluates the counts[r] polynomials of poly_len coefficients held
// by vecs[r] at points[r]; out receives the values request by request.
RustError gb_fr_device_eval_many(RawFr *out_raw, const void *const *vecs, const size_t *counts,
                                 const RawFr *points_raw, size_t requests, size_t poly_len)
{
    if (!out_raw || !vecs || !counts || !points_raw || requests == 0 || poly_len == 0 || requests > 65535)
        return make_error((int)cudaErrorInvalidValue, "invalid batched evaluation arguments");
    GB_ENTRY_BEGIN
    std::vector<eval_pair> pairs;
    for (size_t r = 0; r < requests; r++) {
        auto *v = reinterpret_cast<const fr_device_vec *>(vecs[r]);
        if (!v || counts[r] == 0 || counts[r] > SIZE_MAX / poly_len || v->len != counts[r] * poly_len)
            return make_error((int)cudaErrorInvalidValue, "batched evaluation shape mismatch");
        for (size_t p = 0; p < counts[r]; p++) pairs.push_back(eval_pair{v->values + p * poly_len, (uint32_t)r});
    }
    cudaStream_t s = lane_stream();
    for (size_t r = 0; r < requests; r++) device_vec_wait(reinterpret_cast<const fr_device_vec *>(vecs[r]), s);
    const size_t total = pairs.size();
    dev_buf<fr_t> d_out(total, s);
    eval_pairs(d_out, &pairs, nullptr, total, points_raw, requests, poly_len, s);
    d2h(out_raw, d_out, total * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

// Kate quotients (f - f(z)) / (X - z) of poly_count resident polynomials of
// poly_len coefficients, into a new device vector of the same shape.
RustError gb_fr_device_kate_divide(void **out, const void *device_vec, size_t poly_len, size_t poly_count,
                                   RawFr point_raw)
{
    if (!out || !device_vec || poly_len == 0 || poly_count == 0 || poly_count > SIZE_MAX / poly_len)
        return make_error((int)cudaErrorInvalidValue, "invalid Kate division arguments");
    *out = nullptr;
    GB_ENTRY_BEGIN
    auto *v = reinterpret_cast<const fr_device_vec *>(device_vec);
    if (v->len != poly_len * poly_count)
        return make_error((int)cudaErrorInvalidValue, "Kate division shape mismatch");
    cudaStream_t s = lane_stream();
    device_vec_wait(v, s);
    fr_device_vec *r = device_vec_new(poly_len * poly_count, s);
    try {
        kate_divide(r->values, v->values, poly_len, poly_count, from_raw(point_raw), s);
        device_vec_mark_ready(r, s);
    } catch (...) {
        device_vec_delete(r);
        throw;
    }
    *out = r;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:3600-3721: host polynomials [poly_count][poly_len];
// q_out [q_count][poly_len] (q k = the sum of its items' coefficient times
// polynomial), eval_out[r] = polynomial query_poly_indices[r] at
// points[query_point_indices[r]]
RustError midnight_sppark_bls12_381_fr_multiopen_prepare(
    RawFr *q_out, RawFr *eval_out, const RawFr *polys, size_t poly_len, size_t poly_count, const uint32_t *q_offsets,
    size_t q_offsets_len, const uint32_t *q_poly_indices, const RawFr *q_coefficients, size_t q_items_len,
    const RawFr *points, size_t point_count, const uint32_t *query_poly_indices, const uint32_t *query_point_indices,
    size_t query_count)
{
    if (poly_len == 0 || poly_count == 0 || q_offsets_len < 2 || !q_out || !eval_out || !polys || !q_offsets ||
        !q_poly_indices || !q_coefficients || !points || point_count == 0 || !query_poly_indices ||
        !query_point_indices)
        return make_error((int)cudaErrorInvalidValue, "invalid multi-open preparation arguments");
    if (const char *bad = check_q_layout(q_offsets, q_offsets_len, q_poly_indices, q_items_len, poly_count,
                                         query_poly_indices, query_point_indices, query_count, point_count))
        return make_error((int)cudaErrorInvalidValue, bad);
    const size_t q_count = q_offsets_len - 1;
    if (poly_count > SIZE_MAX / poly_len || q_count > SIZE_MAX / poly_len || point_count > SIZE_MAX / poly_len)
        return make_error((int)cudaErrorInvalidValue, "multi-open preparation size overflow");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    dev_buf<fr_t> d_polys(poly_len * poly_count, s), d_q(poly_len * q_count, s), d_eval(query_count, s);
    h2d(d_polys, polys, poly_len * poly_count * sizeof(fr_t), s);
    std::vector<const fr_t *> table(poly_count);
    for (size_t p = 0; p < poly_count; p++) table[p] = d_polys.get() + p * poly_len;
    multiopen_prepare_core(d_q, d_eval, table, poly_len, q_offsets, q_offsets_len, q_poly_indices, q_coefficients,
                           q_items_len, points, point_count, query_poly_indices, query_point_indices, query_count, s);
    d2h(q_out, d_q, poly_len * q_count * sizeof(fr_t), s);
    d2h(eval_out, d_eval, query_count * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:3723-3871: the same over resident polynomials; poly
// reference p names polynomial index of source 0 (dynamic), 1 (fixed) or 2
// (extra), each a device vector of whole polynomials.  q_out (host) and
// q_device_out (a new device vector) are each optional, not both absent.
RustError midnight_sppark_bls12_381_fr_multiopen_prepare_device(
    RawFr *q_out, void **q_device_out, RawFr *eval_out, const void *dynamic_source, const void *fixed_source,
    const void *extra_source, size_t poly_len, const RawDevicePolyRef *poly_refs, size_t poly_count,
    const uint32_t *q_offsets, size_t q_offsets_len, const uint32_t *q_poly_indices, const RawFr *q_coefficients,
    size_t q_items_len, const RawFr *points, size_t point_count, const uint32_t *query_poly_indices,
    const uint32_t *query_point_indices, size_t query_count)
{
    if (poly_len == 0 || poly_count == 0 || q_offsets_len < 2 || (!q_out && !q_device_out) || !eval_out ||
        !dynamic_source || !fixed_source || !extra_source || !poly_refs || !q_offsets || !q_poly_indices ||
        !q_coefficients || !points || point_count == 0 || !query_poly_indices || !query_point_indices)
        return make_error((int)cudaErrorInvalidValue, "invalid resident multi-open arguments");
    if (q_device_out) *q_device_out = nullptr;
    const fr_device_vec *src[3] = {reinterpret_cast<const fr_device_vec *>(dynamic_source),
                                   reinterpret_cast<const fr_device_vec *>(fixed_source),
                                   reinterpret_cast<const fr_device_vec *>(extra_source)};
    std::vector<const fr_t *> table(poly_count);
    for (size_t p = 0; p < poly_count; p++) {
        const RawDevicePolyRef r = poly_refs[p];
        if (r.source > 2 || (size_t)r.index >= src[r.source]->len / poly_len)
            return make_error((int)cudaErrorInvalidValue, "resident polynomial reference out of range");
        table[p] = src[r.source]->values + (size_t)r.index * poly_len;
    }
    if (const char *bad = check_q_layout(q_offsets, q_offsets_len, q_poly_indices, q_items_len, poly_count,
                                         query_poly_indices, query_point_indices, query_count, point_count))
        return make_error((int)cudaErrorInvalidValue, bad);
    const size_t q_count = q_offsets_len - 1;
    if (q_count > SIZE_MAX / poly_len || point_count > SIZE_MAX / poly_len)
        return make_error((int)cudaErrorInvalidValue, "multi-open preparation size overflow");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    for (const fr_device_vec *v : src) device_vec_wait(v, s);
    fr_device_vec *q = device_vec_new(poly_len * q_count, s);
    try {
        dev_buf<fr_t> d_eval(query_count, s);
        multiopen_prepare_core(q->values, d_eval, table, poly_len, q_offsets, q_offsets_len, q_poly_indices,
                               q_coefficients, q_items_len, points, point_count, query_poly_indices,
                               query_point_indices, query_count, s);
        device_vec_mark_ready(q, s);
        if (q_out) d2h(q_out, q->values, poly_len * q_count * sizeof(fr_t), s);
        d2h(eval_out, d_eval, query_count * sizeof(fr_t), s);
        lane_sync(s);
    } catch (...) {
        device_vec_delete(q);
        throw;
    }
    if (q_device_out) *q_device_out = q;
    else device_vec_delete(q);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:3873-3983: f = sum_k scalars[k] * floor(q_k / prod_j
// (X - points[j])) over q k's points (point_offsets[k] <= j <
// point_offsets[k+1]), one Kate division per point; a new device vector of
// poly_len coefficients
RustError midnight_sppark_bls12_381_fr_multiopen_f_poly_device(void **out, const void *q_device_vec, size_t poly_len,
                                                               const uint32_t *point_offsets,
                                                               size_t point_offsets_len, const RawFr *points,
                                                               size_t point_count, const RawFr *combination_scalars,
                                                               size_t scalar_count)
{
    if (!out || !q_device_vec || poly_len < 2 || !point_offsets || point_offsets_len < 2 || !points ||
        !combination_scalars)
        return make_error((int)cudaErrorInvalidValue, "invalid resident f-polynomial arguments");
    *out = nullptr;
    const size_t q_count = point_offsets_len - 1;
    auto *qv = reinterpret_cast<const fr_device_vec *>(q_device_vec);
    if (q_count != scalar_count || q_count > SIZE_MAX / poly_len || qv->len != q_count * poly_len ||
        point_offsets[0] != 0 || point_offsets[q_count] != point_count)
        return make_error((int)cudaErrorInvalidValue, "resident f-polynomial shape mismatch");
    for (size_t k = 0; k < q_count; k++)
        if (point_offsets[k] > point_offsets[k + 1])
            return make_error((int)cudaErrorInvalidValue, "non-monotonic f-polynomial point offsets");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    device_vec_wait(qv, s);
    // round j divides every q that has more than j points by X - its j-th
    // one, into one half of work and the other in turn
    size_t rounds = 0;
    for (size_t k = 0; k < q_count; k++) rounds = std::max<size_t>(rounds, point_offsets[k + 1] - point_offsets[k]);
    dev_buf<fr_t> work(std::min<size_t>(rounds, 2) * q_count * poly_len, s);
    std::vector<fr_t> zs(point_count);
    for (size_t j = 0; j < point_count; j++) zs[j] = from_raw(points[j]);
    const std::vector<fr_t> powers = kate_powers(zs.data(), point_count);
    dev_buf<fr_t> d_powers(powers.size(), s);
    h2d(d_powers, powers.data(), powers.size() * sizeof(fr_t), s);
    std::vector<const fr_t *> table(q_count);
    for (size_t k = 0; k < q_count; k++) table[k] = qv->values + k * poly_len;
    std::vector<kate_item> items;
    std::vector<size_t> starts(1, 0);
    for (size_t j = 0; j < rounds; j++) {
        for (size_t k = 0; k < q_count; k++) {
            if (j >= point_offsets[k + 1] - point_offsets[k]) continue;
            fr_t *dst = work.get() + ((j & 1) * q_count + k) * poly_len;
            items.push_back(kate_item{table[k], dst, d_powers.get() + (point_offsets[k] + j) * kKatePowers});
            table[k] = dst;
        }
        starts.push_back(items.size());
    }
    dev_buf<kate_item> d_items(items.size(), s);
    h2d(d_items, items.data(), items.size() * sizeof(kate_item), s);
    for (size_t j = 0; j < rounds; j++)
        kate_divide_items(d_items.get() + starts[j], starts[j + 1] - starts[j], poly_len, s);
    dev_buf<const fr_t *> d_table(q_count, s);
    h2d(d_table, table.data(), q_count * sizeof(const fr_t *), s);
    dev_buf<fr_t> d_scalars(scalar_count, s);
    h2d(d_scalars, combination_scalars, scalar_count * sizeof(fr_t), s);
    fr_device_vec *v = device_vec_new(poly_len, s);
    try {
        lincomb_table_kernel<<<blocks_for(poly_len, 256), 256, 0, s>>>(v->values, d_table, d_scalars, poly_len,
                                                                       q_count);
        GB_CHECK_LAUNCH();
        device_vec_mark_ready(v, s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:4025-4118: pi = floor((sum_k scalars[k] q_k +
// scalars[q_count] f) / (X - point)), a new device vector of poly_len - 1
// coefficients (q_count = scalar_count - 1)
RustError midnight_sppark_bls12_381_fr_multiopen_pi_device(void **out, const void *q_device_vec,
                                                           const void *f_device_vec, size_t poly_len,
                                                           const RawFr *combination_scalars, size_t scalar_count,
                                                           RawFr point)
{
    if (!out || !q_device_vec || !f_device_vec || poly_len < 2 || !combination_scalars || scalar_count < 2)
        return make_error((int)cudaErrorInvalidValue, "invalid resident pi-polynomial arguments");
    *out = nullptr;
    const size_t q_count = scalar_count - 1;
    auto *qv = reinterpret_cast<const fr_device_vec *>(q_device_vec);
    auto *fv = reinterpret_cast<const fr_device_vec *>(f_device_vec);
    if (q_count > SIZE_MAX / poly_len || qv->len != q_count * poly_len || fv->len != poly_len)
        return make_error((int)cudaErrorInvalidValue, "resident pi-polynomial shape mismatch");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    device_vec_wait(qv, s);
    device_vec_wait(fv, s);
    std::vector<const fr_t *> table(scalar_count);
    for (size_t k = 0; k < q_count; k++) table[k] = qv->values + k * poly_len;
    table[q_count] = fv->values;
    dev_buf<const fr_t *> d_table(scalar_count, s);
    h2d(d_table, table.data(), scalar_count * sizeof(const fr_t *), s);
    dev_buf<fr_t> d_scalars(scalar_count, s), combined(poly_len, s), quotient(poly_len, s);
    h2d(d_scalars, combination_scalars, scalar_count * sizeof(fr_t), s);
    lincomb_table_kernel<<<blocks_for(poly_len, 256), 256, 0, s>>>(combined, d_table, d_scalars, poly_len,
                                                                   scalar_count);
    GB_CHECK_LAUNCH();
    // the quotient ignores the constant term, so subtracting the value at
    // the point (as the reference does first) changes nothing
    kate_divide(quotient, combined, poly_len, 1, from_raw(point), s);
    fr_device_vec *v = device_vec_new(poly_len - 1, s);
    try {
        GB_CUDA_OK(cudaMemcpyAsync(v->values, quotient.get(), (poly_len - 1) * sizeof(fr_t), cudaMemcpyDeviceToDevice,
                                   s));
        device_vec_mark_ready(v, s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

}  // extern "C"
