// Fr vector kernels: multiplicative prefix scan, Montgomery-trick batch
// inversion, permutation / lookup grand products, quotient limb split, linear
// combinations, canonical sort and the resident device-vector entry points of
// the C ABI (midnight-sppark-msm/src/bls12_381_g1_msm.cu:1188-1700 kernels,
// 2741-3442 device vectors, 3558-4634 vector ops and products).
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <vector>

#include "gb_inv_warp.cuh"
#include "gb_ntt.cuh"
#include "gb_vec.cuh"

namespace gb {

static constexpr int kScanThreads = 256;
static constexpr int kScanPer = 8;  // elements per thread
static constexpr size_t kScanTile = (size_t)kScanThreads * kScanPer;

// ------------------------------------------------------------ block scans

// Inclusive multiplicative scan of one value per thread across the block
// (Hillis-Steele over shared memory).  Returns the inclusive prefix.
__device__ fr_t block_scan_mul(fr_t v, fr_t *sh)
{
    sh[threadIdx.x] = v;
    __syncthreads();
    for (unsigned off = 1; off < blockDim.x; off <<= 1) {
        fr_t other = threadIdx.x >= off ? sh[threadIdx.x - off] : fr_t::one();
        __syncthreads();
        if (threadIdx.x >= off) sh[threadIdx.x] = sh[threadIdx.x] * other;
        __syncthreads();
    }
    return sh[threadIdx.x];
}

// ------------------------------------------------------------ prefix product

// phase 1: per tile product -> aux[tile]
__global__ void __launch_bounds__(kScanThreads) scan_tile_product_kernel(const fr_t *__restrict__ in, size_t n,
                                                                         fr_t *__restrict__ aux)
{
    __shared__ fr_t sh[kScanThreads];
    size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanPer;
    fr_t p = fr_t::one();
#pragma unroll
    for (int e = 0; e < kScanPer; e++)
        if (base + e < n) p = p * in[base + e];
    fr_t incl = block_scan_mul(p, sh);
    if (threadIdx.x == blockDim.x - 1) aux[blockIdx.x] = incl;
}

// phase 3: out[i] = carry_in(tile) * prefix within tile (inclusive)
__global__ void __launch_bounds__(kScanThreads) scan_tile_apply_kernel(const fr_t *__restrict__ in, size_t n,
                                                                       const fr_t *__restrict__ aux_incl,
                                                                       fr_t *out)
{
    __shared__ fr_t sh[kScanThreads];
    size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanPer;
    fr_t vals[kScanPer];
    fr_t p = fr_t::one();
#pragma unroll
    for (int e = 0; e < kScanPer; e++) {
        vals[e] = base + e < n ? in[base + e] : fr_t::one();
        p = p * vals[e];
    }
    fr_t incl = block_scan_mul(p, sh);
    __syncthreads();
    fr_t excl = threadIdx.x ? sh[threadIdx.x - 1] : fr_t::one();
    fr_t run = blockIdx.x ? aux_incl[blockIdx.x - 1] * excl : excl;
    (void)incl;
#pragma unroll
    for (int e = 0; e < kScanPer; e++) {
        run = run * vals[e];
        if (base + e < n) out[base + e] = run;
    }
}

// inclusive prefix product, out may alias in
void prefix_product(fr_t *out, const fr_t *in, size_t n, cudaStream_t s)
{
    if (!n) return;
    size_t tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles > 0x7fffffff) throw cuda_error(-1, "scan too large");
    dev_buf<fr_t> aux(tiles, s);
    scan_tile_product_kernel<<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, aux);
    GB_CHECK_LAUNCH();
    if (tiles > 1) prefix_product(aux, aux, tiles, s);
    scan_tile_apply_kernel<<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, aux, out);
    GB_CHECK_LAUNCH();
}

// ------------------------------------------------------------ batch inversion

// 1 / p for the nonzero p of each of the block's 256 threads: a product tree
// in shared memory (root 1, leaves 256 ..), the root inverted by one warp, the
// inverses coming down (a child's is its parent's times its sibling).
__device__ fr_t block_inverses(fr_t p, fr_t *node)
{
    const unsigned t = threadIdx.x;
    node[kScanThreads + t] = p;
    __syncthreads();
    for (unsigned n = kScanThreads / 2; n >= 32; n >>= 1) {
        if (t < n) node[n + t] = node[2 * (n + t)] * node[2 * (n + t) + 1];
        __syncthreads();
    }
    if (t < 32) {
        fr_t v;
        for (unsigned n = 16; n > 0; n >>= 1) {
            if (t < n) v = node[2 * (n + t)] * node[2 * (n + t) + 1];
            if (t < n) node[n + t] = v;
            __syncwarp();
        }
        v = inverse_warp<FrCfg>(node + 1);
        __syncwarp();
        if (t == 0) node[1] = v;
        __syncwarp();
        for (unsigned n = 2; n <= 32; n <<= 1) {
            if (t < n) v = node[(n + t) >> 1] * node[(n + t) ^ 1];
            __syncwarp();
            if (t < n) node[n + t] = v;
            __syncwarp();
        }
    }
    __syncthreads();
    for (unsigned n = 64; n < kScanThreads; n <<= 1) {
        fr_t v;
        if (t < n) v = node[(n + t) >> 1] * node[(n + t) ^ 1];
        __syncthreads();
        if (t < n) node[n + t] = v;
        __syncthreads();
    }
    return node[(kScanThreads + t) >> 1] * node[(kScanThreads + t) ^ 1];
}

// Montgomery's trick per tile of 256 x PER elements, one inversion a tile;
// zeros stay zero (the field inverse the reference applies maps 0 to 0).  out
// may alias in.  If `mul` is given, out[i] = mul[i] / in[i].
template <int PER>
__global__ void __launch_bounds__(kScanThreads) batch_invert_kernel(const fr_t *in, size_t n, const fr_t *mul,
                                                                    fr_t *out)
{
    __shared__ fr_t node[2 * kScanThreads];
    const size_t base = (size_t)blockIdx.x * (kScanThreads * PER) + threadIdx.x;
    fr_t x[PER], q[PER];
    fr_t p = fr_t::one();
#pragma unroll
    for (int e = 0; e < PER; e++) {
        const size_t i = base + (size_t)e * kScanThreads;
        x[e] = i < n ? in[i] : fr_t::zero();
        q[e] = p;  // product of this thread's earlier nonzero elements
        if (!x[e].is_zero()) p = p * x[e];
    }
    fr_t J = block_inverses(p, node);
#pragma unroll
    for (int e = PER - 1; e >= 0; e--) {
        const size_t i = base + (size_t)e * kScanThreads;
        if (i >= n) continue;
        fr_t r = fr_t::zero();
        if (!x[e].is_zero()) {
            r = J * q[e];
            J = J * x[e];
            if (mul) r = mul[i] * r;
        }
        out[i] = r;
    }
}

// Elements a thread: 4 until the tiles fill the GPU (a tile is one chain: its
// inversion, about 12 us, and 16 tree levels), then 8
static int tile_per(size_t n) { return n <= (size_t)1 << 18 ? 4 : 8; }

void batch_invert(fr_t *out, const fr_t *in, size_t n, const fr_t *mul, cudaStream_t s)
{
    if (!n) return;
    const int per = tile_per(n);
    const size_t tiles = (n + kScanThreads * per - 1) / (kScanThreads * per);
    if (per == 4) batch_invert_kernel<4><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, mul, out);
    else batch_invert_kernel<8><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, mul, out);
    GB_CHECK_LAUNCH();
}

__global__ void power_factors_kernel(fr_t *d, fr_t w, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) d[i] = i ? w : fr_t::one();
}

// Power tables up to 2^24 entries: w^i = T0[i & 255] * T1[(i >> 8) & 255] *
// T2[i >> 16], where T0[j] = w^j, T1[j] = w^(256 j), T2[j] = w^(65536 j); a
// block a table.  Every thread squares its way to its entry's bits (at most 32
// dependent products, 13 us; block scans took 24 us for the three tables).  The
// apply kernel spends two products per element.
__global__ void __launch_bounds__(256) power_tables_kernel(fr_t w, fr_t *__restrict__ tables)
{
    for (unsigned k = 0; k < 8 * blockIdx.x; k++) w = w.sqr();
    fr_t v = fr_t::one();
    for (unsigned b = 0; b < 8; b++) {
        if ((threadIdx.x >> b) & 1u) v = v * w;
        w = w.sqr();
    }
    tables[blockIdx.x * 256 + threadIdx.x] = v;
}

__global__ void power_apply_kernel(const fr_t *__restrict__ tables, size_t n, fr_t *__restrict__ d)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    fr_t v = tables[i & 255];
    if (i >> 8) v = v * tables[256 + ((i >> 8) & 255)];
    if (i >> 16) v = v * tables[512 + (i >> 16)];
    d[i] = v;
}

void omega_powers(fr_t *d, const fr_t &w, size_t n, cudaStream_t s)
{
    if (!n) return;
    if (n > ((size_t)1 << 24)) {
        power_factors_kernel<<<blocks_for(n, 256), 256, 0, s>>>(d, w, n);
        GB_CHECK_LAUNCH();
        prefix_product(d, d, n, s);
        return;
    }
    dev_buf<fr_t> tables(3 * 256, s);
    power_tables_kernel<<<n > 65536 ? 3 : n > 256 ? 2 : 1, 256, 0, s>>>(w, tables);
    GB_CHECK_LAUNCH();
    power_apply_kernel<<<blocks_for(n, 256), 256, 0, s>>>(tables, n, d);
    GB_CHECK_LAUNCH();
}

// ------------------------------------------------------------ products

// z[0] = init, z[i] = init * prefix[i-1]; init read from device memory
__global__ void shifted_apply_kernel(fr_t *__restrict__ out, const fr_t *__restrict__ prefix,
                                     const fr_t *__restrict__ init, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    fr_t a = *init;
    out[i] = i ? a * prefix[i - 1] : a;
}

// A grand product z is two launches: the fractions num / den of every row with
// their tiles' products, then each tile's share of z, which multiplies the
// tiles before it itself.  Neither numerators nor denominators touch memory, and
// the fractions stand where z goes, so there is no scratch but the tiles'
// products.
// Both are a few chains on few warps, bound by the latency of a product (0.45
// us) and of the tile's inversion (12 us, by a warp; 100 us by one thread).
// Measured, the permutation products of 3 columns of 2^16 rows 0.297 -> 0.100
// ms, of 2^10 0.22 -> 0.073 ms.

static __device__ __noinline__ fr_t fr_mul_called(fr_t a, fr_t b) { return a * b; }

// Permutation fraction of row i, set `set` (prover.rs:392-460):
// num = prod_j (v_j + delta^j w^i beta + gamma), den = prod_j (v_j + beta s_j + gamma).
// Column c is columns[c * len ..] or, with a pointer table, col_ptrs[c][..].
struct perm_fraction {
    const fr_t *columns;
    const fr_t *const *col_ptrs;
    const fr_t *perms, *delta_powers;
    fr_t beta, gamma;
    size_t len, column_count, chunk_len;
    fr_t w2[32];  // omega^(2^b)
    typedef fr_t state;  // beta w^i
    __device__ state begin(size_t i) const
    {
        fr_t v = beta;
        for (int b = 0; b < 32 && (i >> b); b++)
            if ((i >> b) & 1) v = fr_mul_called(v, w2[b]);
        if (i >> 32) v = fr_mul_called(v, fr_mul_called(w2[31], w2[31]).pow_u64(i >> 32));
        return v;
    }
    // kScanThreads = 2^8 rows on
    __device__ void next(state &v) const { v = fr_mul_called(v, w2[8]); }
    __device__ void at(size_t set, size_t i, const state &bw, fr_t &num, fr_t &den) const
    {
        const size_t c0 = set * chunk_len, c1 = min(c0 + chunk_len, column_count);
        num = fr_t::one(), den = fr_t::one();
        for (size_t c = c0; c < c1; c++) {
            const fr_t v = (col_ptrs ? col_ptrs[c][i] : columns[c * len + i]) + gamma;
            num = fr_mul_called(num, v + fr_mul_called(delta_powers[c], bw));
            den = fr_mul_called(den, v + fr_mul_called(beta, perms[c * len + i]));
        }
    }
};

// Lookup fraction (lookup/prover.rs:1075-1240):
// num = (A + beta)(S + gamma), den = (A' + beta)(S' + gamma)
struct lookup_fraction {
    const fr_t *ci, *ct, *pi, *pt;
    fr_t beta, gamma;
    size_t len;
    typedef int state;
    __device__ state begin(size_t) const { return 0; }
    __device__ void next(state &) const {}
    __device__ void at(size_t set, size_t i, const state &, fr_t &num, fr_t &den) const
    {
        const size_t f = set * len + i;
        num = fr_mul_called(ci[f] + beta, ct[f] + gamma);
        den = fr_mul_called(pi[f] + beta, pt[f] + gamma);
    }
};

// frac[set][i] = num / den (0 where den is 0) and tile_products[set][tile]
template <class F, int PER>
__global__ void __launch_bounds__(kScanThreads) fraction_kernel(const __grid_constant__ F f, size_t len, size_t set0,
                                                                fr_t *__restrict__ frac,
                                                                fr_t *__restrict__ tile_products)
{
    __shared__ fr_t node[2 * kScanThreads];
    const size_t base = (size_t)blockIdx.x * kScanThreads * PER + threadIdx.x, set = set0 + blockIdx.y;
    fr_t num[PER], den[PER], q[PER];
    fr_t p = fr_t::one();
    typename F::state st = f.begin(base);
#pragma unroll
    for (int e = 0; e < PER; e++) {
        const size_t i = base + (size_t)e * kScanThreads;
        num[e] = fr_t::one(), den[e] = fr_t::one();
        if (i < len) f.at(set, i, st, num[e], den[e]);
        if (e + 1 < PER) f.next(st);
        q[e] = p;
        if (!den[e].is_zero()) p = fr_mul_called(p, den[e]);
    }
    fr_t J = block_inverses(p, node), prod = fr_t::one();
#pragma unroll
    for (int e = PER - 1; e >= 0; e--) {
        const size_t i = base + (size_t)e * kScanThreads;
        fr_t r = fr_t::zero();
        if (!den[e].is_zero()) {
            r = fr_mul_called(num[e], fr_mul_called(J, q[e]));
            J = fr_mul_called(J, den[e]);
        }
        if (i < len) frac[set * len + i] = r;
        prod = fr_mul_called(prod, r);  // one past the end
    }
    __syncthreads();
    node[threadIdx.x] = prod;
    __syncthreads();
    for (unsigned off = kScanThreads / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) node[threadIdx.x] = node[threadIdx.x] * node[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) tile_products[set * gridDim.x + blockIdx.x] = node[0];
}

// z[i] = init * (product of the fractions before i) for i < len - bf, the
// blinds after; `tiles` are the tiles' products, or with `scanned` their
// inclusive prefix products.  z holds the fractions; a thread reads its own and
// writes z in their place.
template <int PER>
__global__ void __launch_bounds__(kScanThreads) grand_product_kernel(const fr_t *__restrict__ tiles, bool scanned,
                                                                     size_t len, size_t set0, const fr_t *init,
                                                                     const fr_t *__restrict__ blinds, size_t bf,
                                                                     fr_t *z)
{
    __shared__ fr_t sh[kScanThreads];
    const size_t set = set0 + blockIdx.y, b = blockIdx.x;
    tiles += set * gridDim.x;
    z += set * len;
    fr_t carry = init ? *init : fr_t::one();
    if (scanned) {
        if (b) carry = carry * tiles[b - 1];
    } else if (b) {
        fr_t p = fr_t::one();
        for (size_t t = threadIdx.x; t < b; t += kScanThreads) p = p * tiles[t];
        sh[threadIdx.x] = p;
        __syncthreads();
        for (unsigned off = kScanThreads / 2; off > 0; off >>= 1) {
            if (threadIdx.x < off && threadIdx.x + off < b) sh[threadIdx.x] = sh[threadIdx.x] * sh[threadIdx.x + off];
            __syncthreads();
        }
        carry = carry * sh[0];
        __syncthreads();
    }
    const size_t base = (b * kScanThreads + threadIdx.x) * PER;
    fr_t v[PER], p = fr_t::one();
#pragma unroll
    for (int e = 0; e < PER; e++) {
        v[e] = base + e < len ? z[base + e] : fr_t::one();
        p = p * v[e];
    }
    block_scan_mul(p, sh);
    __syncthreads();
    fr_t run = threadIdx.x ? carry * sh[threadIdx.x - 1] : carry;
#pragma unroll
    for (int e = 0; e < PER; e++) {
        const size_t i = base + e;
        if (i < len) z[i] = i < len - bf ? run : blinds[set * bf + i - (len - bf)];
        run = run * v[e];
    }
}

// z of `sets` products into out [sets][len]; chained: a set starts from the
// last unblinded value of the one before
template <int PER, class F>
static void grand_products_tiled(fr_t *out, const F &f, size_t len, size_t sets, bool chained, const fr_t *d_blinds,
                                 size_t bf, cudaStream_t s)
{
    const size_t tile = (size_t)kScanThreads * PER, tiles = (len + tile - 1) / tile;
    if (tiles > 0x7fffffff) throw cuda_error((int)cudaErrorInvalidValue, "grand product too large");
    dev_buf<fr_t> products(tiles * sets, s);
    constexpr size_t kMaxY = 65535;
    for (size_t k = 0; k < sets; k += kMaxY) {
        const dim3 grid((unsigned)tiles, (unsigned)std::min(kMaxY, sets - k));
        fraction_kernel<F, PER><<<grid, kScanThreads, 0, s>>>(f, len, k, out, products);
        GB_CHECK_LAUNCH();
    }
    // beyond 2^20 rows a tile's own walk over the tiles before it costs more
    // than a scan of their products
    const bool scanned = tiles > 1024;
    if (scanned)
        for (size_t k = 0; k < sets; k++) prefix_product(products + k * tiles, products + k * tiles, tiles, s);
    for (size_t k = 0; k < sets; k += chained ? 1 : kMaxY) {
        const dim3 grid((unsigned)tiles, chained ? 1u : (unsigned)std::min(kMaxY, sets - k));
        const fr_t *init = chained && k ? out + (k - 1) * len + (len - (bf + 1)) : nullptr;
        grand_product_kernel<PER><<<grid, kScanThreads, 0, s>>>(products, scanned, len, k, init, d_blinds, bf, out);
        GB_CHECK_LAUNCH();
    }
}

template <class F>
static void grand_products(fr_t *out, const F &f, size_t len, size_t sets, bool chained, const fr_t *d_blinds,
                           size_t bf, cudaStream_t s)
{
    if (!len || !sets) return;
    // rows a thread: a tile is one chain, so short products take short tiles.
    // Measured, us a call with 1, 2 and 4: 2^12 rows 78* 94 129, 2^15 82* 98
    // 137, 2^16 113 99* 137, 2^17 202 144 137*, 2^18 355 264 251*.
    if (len <= (size_t)1 << 15) grand_products_tiled<1>(out, f, len, sets, chained, d_blinds, bf, s);
    else if (len <= (size_t)1 << 16) grand_products_tiled<2>(out, f, len, sets, chained, d_blinds, bf, s);
    else grand_products_tiled<4>(out, f, len, sets, chained, d_blinds, bf, s);
}

void permutation_products(fr_t *out, const fr_t *d_columns, const fr_t *const *d_col_ptrs, const fr_t *d_perms,
                          size_t len, size_t column_count, size_t chunk_len, const fr_t &beta, const fr_t &gamma,
                          const fr_t &omega, const fr_t *d_delta, const fr_t *d_blinds, size_t bf, cudaStream_t s)
{
    perm_fraction f{d_columns, d_col_ptrs, d_perms, d_delta, beta, gamma, len, column_count, chunk_len, {}};
    f.w2[0] = omega;
    for (int b = 1; b < 32; b++) f.w2[b] = b <= 8 || (len >> b) ? f.w2[b - 1].sqr() : fr_t::one();
    grand_products(out, f, len, (column_count + chunk_len - 1) / chunk_len, true, d_blinds, bf, s);
}

void lookup_products(fr_t *out, const fr_t *ci, const fr_t *ct, const fr_t *pi, const fr_t *pt, size_t len,
                     size_t lookup_count, const fr_t &beta, const fr_t &gamma, const fr_t *d_blinds, size_t bf,
                     cudaStream_t s)
{
    const lookup_fraction f{ci, ct, pi, pt, beta, gamma, len};
    grand_products(out, f, len, lookup_count, false, d_blinds, bf, s);
}

// ------------------------------------------------------------ misc kernels

__global__ void lincomb_kernel(fr_t *__restrict__ out, const fr_t *__restrict__ polys, const fr_t *__restrict__ k,
                               size_t len, size_t count)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= len) return;
    fr_t acc = fr_t::zero();
    for (size_t p = 0; p < count; p++) acc = acc + polys[p * len + i] * k[p];
    out[i] = acc;
}

__global__ void quotient_pieces_kernel(fr_t *__restrict__ out, const fr_t *__restrict__ q, size_t poly_len,
                                       size_t pieces)
{
    size_t f = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= poly_len * pieces) return;
    size_t piece = f / poly_len, i = f % poly_len;
    out[f] = i == poly_len - 1 ? fr_t::zero() : q[piece * (poly_len - 1) + i];
}

__global__ void blind_quotient_pieces_kernel(fr_t *pieces, const fr_t *__restrict__ blinds, size_t poly_len,
                                             size_t count)
{
    // sequential over pieces: piece p's last slot and piece p+1's first slot
    if (threadIdx.x || blockIdx.x) return;
    for (size_t p = 0; p + 1 < count; p++) {
        fr_t b = blinds[p];
        pieces[p * poly_len + poly_len - 1] = b;
        pieces[(p + 1) * poly_len] = pieces[(p + 1) * poly_len] - b;
    }
}

// canonical big-endian key (fq.rs:152-164) as 4 x u64 for the radix sort
struct canon_key {
    uint64_t l[4];
};
struct canon_decomposer {
    __host__ __device__ ::cuda::std::tuple<uint64_t &, uint64_t &, uint64_t &, uint64_t &> operator()(
        canon_key &k) const
    {
        return {k.l[3], k.l[2], k.l[1], k.l[0]};
    }
};

__global__ void to_canon_kernel(const fr_t *__restrict__ in, canon_key *__restrict__ out, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    fr_t c = in[i].from_mont();
    canon_key k;
#pragma unroll
    for (int j = 0; j < 4; j++) k.l[j] = (uint64_t)c.v[2 * j] | ((uint64_t)c.v[2 * j + 1] << 32);
    out[i] = k;
}

__global__ void from_canon_kernel(const canon_key *__restrict__ in, fr_t *__restrict__ out, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    fr_t c;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        c.v[2 * j] = (uint32_t)in[i].l[j];
        c.v[2 * j + 1] = (uint32_t)(in[i].l[j] >> 32);
    }
    out[i] = c.to_mont();
}

void sort_canonical(fr_t *d, size_t n, cudaStream_t s)
{
    if (n < 2) return;
    dev_buf<canon_key> a(n, s), b(n, s);
    to_canon_kernel<<<blocks_for(n, 256), 256, 0, s>>>(d, a, n);
    GB_CHECK_LAUNCH();
    size_t temp = 0;
    GB_CUDA_OK(cub::DeviceRadixSort::SortKeys(nullptr, temp, a.get(), b.get(), (int64_t)n, canon_decomposer{}, 0, 256, s));
    dev_buf<uint8_t> t(temp, s);
    GB_CUDA_OK(cub::DeviceRadixSort::SortKeys(t.get(), temp, a.get(), b.get(), (int64_t)n, canon_decomposer{}, 0, 256, s));
    from_canon_kernel<<<blocks_for(n, 256), 256, 0, s>>>(b, d, n);
    GB_CHECK_LAUNCH();
}

// upload helper
static dev_buf<fr_t> upload(const fr_t *host, size_t n, cudaStream_t s)
{
    dev_buf<fr_t> d(n, s);
    h2d(d, host, n * sizeof(fr_t), s);
    return d;
}

}  // namespace gb

namespace gb {

static constexpr size_t kSuffixSlice = 8192;

__global__ void nonzero_init_kernel(unsigned long long *stats, size_t count, size_t len)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) {
        stats[i] = len;        // first nonzero (len: none)
        stats[count + i] = 0;  // nonzero count
    }
}

// block (slice, poly): the slice's first nonzero index and nonzero count,
// merged into the polynomial's by atomics
__global__ void nonzero_stats_kernel(unsigned long long *first, unsigned long long *live,
                                     const fr_t *__restrict__ values, size_t len)
{
    __shared__ unsigned long long f_sh[256], c_sh[256];
    const size_t p = blockIdx.y;
    const fr_t *poly = values + p * len;
    const size_t lo = (size_t)blockIdx.x * kSuffixSlice, hi = min(lo + kSuffixSlice, len);
    unsigned long long f = len, c = 0;
    for (size_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        if (!poly[i].is_zero()) {
            f = min(f, (unsigned long long)i);
            c++;
        }
    }
    f_sh[threadIdx.x] = f;
    c_sh[threadIdx.x] = c;
    __syncthreads();
    for (unsigned off = blockDim.x / 2; off; off >>= 1) {
        if (threadIdx.x < off) {
            f_sh[threadIdx.x] = min(f_sh[threadIdx.x], f_sh[threadIdx.x + off]);
            c_sh[threadIdx.x] += c_sh[threadIdx.x + off];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (f_sh[0] < len) atomicMin(first + p, f_sh[0]);
        if (c_sh[0]) atomicAdd(live + p, c_sh[0]);
    }
}

}  // namespace gb

using namespace gb;

extern "C" {

// ---------------------------------------------------------------- vector ops
// bls12_381_g1_msm.cu:3558-3600 (host vector in, result back in place)
RustError midnight_sppark_bls12_381_fr_mul_assign(RawFr *values_raw, RawFr scalar_raw, size_t len)
{
    fr_t *values = reinterpret_cast<fr_t *>(values_raw);
    const fr_t scalar = gb::from_raw(scalar_raw);
    if (len == 0) return ok();
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    auto d = upload(values, len, s);
    launch_mul_assign(d, scalar, len, s);
    d2h(values, d, len * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

RustError midnight_sppark_bls12_381_fr_mul_assign_zeta(RawFr *values_raw, RawFr first_raw, RawFr second_raw, size_t len)
{
    fr_t *values = reinterpret_cast<fr_t *>(values_raw);
    const fr_t first = gb::from_raw(first_raw);
    const fr_t second = gb::from_raw(second_raw);
    if (len == 0) return ok();
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    auto d = upload(values, len, s);
    launch_mul_assign_zeta(d, first, second, len, len, s);
    d2h(values, d, len * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

RustError midnight_sppark_bls12_381_fr_mul_assign_repeating(RawFr *values_raw, const RawFr *factors_raw, size_t factor_len, size_t len)
{
    fr_t *values = reinterpret_cast<fr_t *>(values_raw);
    const fr_t *factors = reinterpret_cast<const fr_t *>(factors_raw);
    if (len == 0) return ok();
    if (factor_len == 0 || !factors) return make_error((int)cudaErrorInvalidValue, "empty repeating factors");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    auto d = upload(values, len, s);
    auto f = upload(factors, factor_len, s);
    launch_mul_assign_repeating(d, f, factor_len, len, s);
    d2h(values, d, len * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:1225-1231 semantics (every element inverted, 0 -> 0),
// computed with Montgomery's trick instead of one exponentiation per element
RustError midnight_sppark_bls12_381_fr_invert_assign(RawFr *values_raw, size_t len)
{
    fr_t *values = reinterpret_cast<fr_t *>(values_raw);
    if (len == 0) return ok();
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    auto d = upload(values, len, s);
    batch_invert(d, d, len, nullptr, s);
    d2h(values, d, len * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

RustError midnight_sppark_bls12_381_fr_sort_canonical(RawFr *values_raw, size_t len)
{
    fr_t *values = reinterpret_cast<fr_t *>(values_raw);
    if (len < 2) return ok();
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    auto d = upload(values, len, s);
    sort_canonical(d, len, s);
    d2h(values, d, len * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:3558 region: out[i] = sum_k scalars[k] * polys[k][i]
RustError midnight_sppark_bls12_381_fr_poly_lincomb(RawFr *out_raw, const RawFr *polys_raw, size_t poly_len, size_t poly_count, const RawFr *scalars_raw)
{
    fr_t *out = reinterpret_cast<fr_t *>(out_raw);
    const fr_t *polys = reinterpret_cast<const fr_t *>(polys_raw);
    const fr_t *scalars = reinterpret_cast<const fr_t *>(scalars_raw);
    if (poly_len == 0) return ok();
    if (!out || (poly_count && (!polys || !scalars)))
        return make_error((int)cudaErrorInvalidValue, "invalid lincomb arguments");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    auto d = upload(polys, poly_len * poly_count, s);
    auto k = upload(scalars, poly_count, s);
    dev_buf<fr_t> o(poly_len, s);
    lincomb_kernel<<<blocks_for(poly_len, 256), 256, 0, s>>>(o, d, k, poly_len, poly_count);
    GB_CHECK_LAUNCH();
    d2h(out, o, poly_len * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:4303-4340 (permutation/prover.rs:36-43 semantics)
RustError midnight_sppark_bls12_381_fr_shifted_prefix_product(RawFr *values_raw, RawFr initial_raw, size_t len)
{
    fr_t *values = reinterpret_cast<fr_t *>(values_raw);
    const fr_t initial = gb::from_raw(initial_raw);
    if (len == 0) return ok();
    if (!values) return make_error((int)cudaErrorInvalidValue, "null values");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    auto d = upload(values, len, s);
    dev_buf<fr_t> prefix(len, s), init(1, s);
    h2d(init, &initial, sizeof(fr_t), s);
    prefix_product(prefix, d, len, s);
    shifted_apply_kernel<<<blocks_for(len, 256), 256, 0, s>>>(d, prefix, init, len);
    GB_CHECK_LAUNCH();
    d2h(values, d, len * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:4342-4449: z of every permutation set, resident
RustError midnight_sppark_bls12_381_fr_permutation_products(void **out, const RawFr *columns_raw, const RawFr *permutations_raw, size_t len, size_t column_count, size_t chunk_len, RawFr beta_raw, RawFr gamma_raw, RawFr omega_raw, const RawFr *delta_powers_raw, const RawFr *blind_values_raw, size_t blinding_factors)
{
    const fr_t *columns = reinterpret_cast<const fr_t *>(columns_raw);
    const fr_t *permutations = reinterpret_cast<const fr_t *>(permutations_raw);
    const fr_t beta = gb::from_raw(beta_raw);
    const fr_t gamma = gb::from_raw(gamma_raw);
    const fr_t omega = gb::from_raw(omega_raw);
    const fr_t *delta_powers = reinterpret_cast<const fr_t *>(delta_powers_raw);
    const fr_t *blind_values = reinterpret_cast<const fr_t *>(blind_values_raw);
    if (!out || len == 0 || column_count == 0 || chunk_len == 0 || !columns || !permutations || !delta_powers ||
        blinding_factors >= len || (blinding_factors != 0 && !blind_values))
        return make_error((int)cudaErrorInvalidValue, "invalid permutation product arguments");
    *out = nullptr;
    const size_t sets = (column_count + chunk_len - 1) / chunk_len;
    if (column_count > SIZE_MAX / len || sets > SIZE_MAX / len)
        return make_error((int)cudaErrorInvalidValue, "permutation product size overflow");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    auto dc = upload(columns, column_count * len, s);
    auto dp = upload(permutations, column_count * len, s);
    auto dd = upload(delta_powers, column_count, s);
    auto db = upload(blind_values, sets * blinding_factors, s);
    fr_device_vec *v = device_vec_new(sets * len, s);
    try {
        permutation_products(v->values, dc, nullptr, dp, len, column_count, chunk_len, beta, gamma, omega, dd, db,
                             blinding_factors, s);
        device_vec_mark_ready(v, s);
        lane_sync(s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// The permutation products over resident columns and permutation values
// (column_count x len each); delta powers and blinds are host arrays.
RustError gb_fr_permutation_products_device(void **out, const void *columns_vec, const void *permutations_vec,
                                            size_t len, size_t column_count, size_t chunk_len, RawFr beta_raw,
                                            RawFr gamma_raw, RawFr omega_raw, const RawFr *delta_powers_raw,
                                            const RawFr *blind_values_raw, size_t blinding_factors)
{
    const fr_t *delta_powers = reinterpret_cast<const fr_t *>(delta_powers_raw);
    const fr_t *blind_values = reinterpret_cast<const fr_t *>(blind_values_raw);
    if (!out || len == 0 || column_count == 0 || chunk_len == 0 || !columns_vec || !permutations_vec ||
        !delta_powers || blinding_factors >= len || (blinding_factors != 0 && !blind_values))
        return make_error((int)cudaErrorInvalidValue, "invalid resident permutation product arguments");
    *out = nullptr;
    const size_t sets = (column_count + chunk_len - 1) / chunk_len;
    if (column_count > SIZE_MAX / len || sets > SIZE_MAX / len)
        return make_error((int)cudaErrorInvalidValue, "permutation product size overflow");
    GB_ENTRY_BEGIN
    auto *cv = reinterpret_cast<const fr_device_vec *>(columns_vec);
    auto *pv = reinterpret_cast<const fr_device_vec *>(permutations_vec);
    if (cv->len < column_count * len || pv->len < column_count * len)
        return make_error((int)cudaErrorInvalidValue, "resident permutation columns too short");
    cudaStream_t s = lane_stream();
    device_vec_wait(cv, s);
    device_vec_wait(pv, s);
    auto dd = upload(delta_powers, column_count, s);
    auto db = upload(blind_values, sets * blinding_factors, s);
    fr_device_vec *v = device_vec_new(sets * len, s);
    try {
        permutation_products(v->values, cv->values, nullptr, pv->values, len, column_count, chunk_len,
                             gb::from_raw(beta_raw), gb::from_raw(gamma_raw), gb::from_raw(omega_raw), dd, db,
                             blinding_factors, s);
        device_vec_mark_ready(v, s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:4451-4548
RustError midnight_sppark_bls12_381_fr_lookup_products(void **out, const RawFr *compressed_inputs_raw, const RawFr *compressed_tables_raw, const RawFr *permuted_inputs_raw, const RawFr *permuted_tables_raw, size_t len, size_t lookup_count, RawFr beta_raw, RawFr gamma_raw, const RawFr *blind_values_raw, size_t blinding_factors)
{
    const fr_t *compressed_inputs = reinterpret_cast<const fr_t *>(compressed_inputs_raw);
    const fr_t *compressed_tables = reinterpret_cast<const fr_t *>(compressed_tables_raw);
    const fr_t *permuted_inputs = reinterpret_cast<const fr_t *>(permuted_inputs_raw);
    const fr_t *permuted_tables = reinterpret_cast<const fr_t *>(permuted_tables_raw);
    const fr_t beta = gb::from_raw(beta_raw);
    const fr_t gamma = gb::from_raw(gamma_raw);
    const fr_t *blind_values = reinterpret_cast<const fr_t *>(blind_values_raw);
    if (!out || len == 0 || lookup_count == 0 || !compressed_inputs || !compressed_tables || !permuted_inputs ||
        !permuted_tables || blinding_factors >= len || (blinding_factors != 0 && !blind_values))
        return make_error((int)cudaErrorInvalidValue, "invalid lookup product arguments");
    *out = nullptr;
    if (lookup_count > SIZE_MAX / len) return make_error((int)cudaErrorInvalidValue, "lookup product size overflow");
    GB_ENTRY_BEGIN
    const size_t total = lookup_count * len;
    cudaStream_t s = lane_stream();
    auto a = upload(compressed_inputs, total, s);
    auto b = upload(compressed_tables, total, s);
    auto c = upload(permuted_inputs, total, s);
    auto d = upload(permuted_tables, total, s);
    auto bl = upload(blind_values, lookup_count * blinding_factors, s);
    fr_device_vec *v = device_vec_new(total, s);
    try {
        lookup_products(v->values, a, b, c, d, len, lookup_count, beta, gamma, bl, blinding_factors, s);
        device_vec_mark_ready(v, s);
        lane_sync(s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:4550-4634: the four lookup columns already resident,
// laid out [compressed inputs | compressed tables | permuted inputs | permuted tables]
RustError midnight_sppark_bls12_381_fr_lookup_products_device(void **out, const void *trace_lagrange, size_t len, size_t lookup_count, RawFr beta_raw, RawFr gamma_raw, const RawFr *blind_values_raw, size_t blinding_factors)
{
    const fr_t beta = gb::from_raw(beta_raw);
    const fr_t gamma = gb::from_raw(gamma_raw);
    const fr_t *blind_values = reinterpret_cast<const fr_t *>(blind_values_raw);
    if (!out || len == 0 || lookup_count == 0 || !trace_lagrange || blinding_factors >= len ||
        (blinding_factors != 0 && !blind_values))
        return make_error((int)cudaErrorInvalidValue, "invalid resident lookup product arguments");
    *out = nullptr;
    if (lookup_count > SIZE_MAX / len)
        return make_error((int)cudaErrorInvalidValue, "resident lookup product size overflow");
    GB_ENTRY_BEGIN
    const size_t total = lookup_count * len;
    auto *tr = reinterpret_cast<const fr_device_vec *>(trace_lagrange);
    if (tr->len != total * 4) return make_error((int)cudaErrorInvalidValue, "resident lookup trace length mismatch");
    cudaStream_t s = lane_stream();
    device_vec_wait(tr, s);
    auto bl = upload(blind_values, lookup_count * blinding_factors, s);
    fr_device_vec *v = device_vec_new(total, s);
    try {
        const fr_t *base = tr->values;
        lookup_products(v->values, base, base + total, base + 2 * total, base + 3 * total, len, lookup_count, beta,
                        gamma, bl, blinding_factors, s);
        device_vec_mark_ready(v, s);
        lane_sync(s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:3181-3240 (vanishing/prover.rs:141-220,304-318)
RustError midnight_sppark_bls12_381_fr_device_quotient_pieces(void **out, const void *quotient_vec, size_t poly_len, size_t piece_count, const RawFr *blinds_raw, size_t blind_count)
{
    const fr_t *blinds = reinterpret_cast<const fr_t *>(blinds_raw);
    if (!out || !quotient_vec || poly_len < 2 || piece_count < 2 || blind_count != piece_count - 1 || !blinds ||
        piece_count > SIZE_MAX / poly_len)
        return make_error((int)cudaErrorInvalidValue, "invalid resident quotient piece arguments");
    *out = nullptr;
    GB_ENTRY_BEGIN
    auto *q = reinterpret_cast<const fr_device_vec *>(quotient_vec);
    if (q->len < (poly_len - 1) * piece_count)
        return make_error((int)cudaErrorInvalidValue, "resident quotient is too short");
    cudaStream_t s = lane_stream();
    device_vec_wait(q, s);
    auto b = upload(blinds, blind_count, s);
    fr_device_vec *v = device_vec_new(poly_len * piece_count, s);
    try {
        quotient_pieces_kernel<<<blocks_for(poly_len * piece_count, 256), 256, 0, s>>>(v->values, q->values, poly_len,
                                                                                     piece_count);
        GB_CHECK_LAUNCH();
        blind_quotient_pieces_kernel<<<1, 32, 0, s>>>(v->values, b, poly_len, piece_count);
        GB_CHECK_LAUNCH();
        device_vec_mark_ready(v, s);
        lane_sync(s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:3242-3278
RustError midnight_sppark_bls12_381_fr_device_poly_lincomb(void **out, const void *polys_vec, size_t poly_len, size_t poly_count, const RawFr *scalars_raw, size_t scalar_count)
{
    const fr_t *scalars = reinterpret_cast<const fr_t *>(scalars_raw);
    if (!out || !polys_vec || poly_len == 0 || poly_count == 0 || !scalars || scalar_count != poly_count)
        return make_error((int)cudaErrorInvalidValue, "invalid resident lincomb arguments");
    *out = nullptr;
    GB_ENTRY_BEGIN
    auto *pv = reinterpret_cast<const fr_device_vec *>(polys_vec);
    if (poly_count > SIZE_MAX / poly_len || pv->len < poly_len * poly_count)
        return make_error((int)cudaErrorInvalidValue, "resident lincomb source too short");
    cudaStream_t s = lane_stream();
    device_vec_wait(pv, s);
    auto k = upload(scalars, scalar_count, s);
    fr_device_vec *v = device_vec_new(poly_len, s);
    try {
        lincomb_kernel<<<blocks_for(poly_len, 256), 256, 0, s>>>(v->values, pv->values, k, poly_len, poly_count);
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

// ---------------------------------------------------------------- device vectors
// bls12_381_g1_msm.cu:2741-2780
RustError midnight_sppark_bls12_381_fr_device_vec_upload(void **out, const RawFr *values_raw, size_t len)
{
    const fr_t *values = reinterpret_cast<const fr_t *>(values_raw);
    if (!out || (len && !values)) return make_error((int)cudaErrorInvalidValue, "invalid device vector upload");
    *out = nullptr;
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    fr_device_vec *v = device_vec_new(len, s);
    try {
        h2d(v->values, values, len * sizeof(fr_t), s);
        device_vec_mark_ready(v, s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:2782-2830: several host slices concatenated
RustError midnight_sppark_bls12_381_fr_device_vec_upload_many(void **out, const RawFr *const *values_raw, const size_t *lengths, size_t count)
{
    const fr_t *const *values = reinterpret_cast<const fr_t *const *>(values_raw);
    if (!out || (count && (!values || !lengths)))
        return make_error((int)cudaErrorInvalidValue, "invalid device vector upload");
    *out = nullptr;
    GB_ENTRY_BEGIN
    size_t total = 0;
    for (size_t i = 0; i < count; i++) {
        if (lengths[i] && !values[i]) return make_error((int)cudaErrorInvalidValue, "null upload slice");
        total += lengths[i];
    }
    cudaStream_t s = lane_stream();
    fr_device_vec *v = device_vec_new(total, s);
    try {
        size_t off = 0;
        for (size_t i = 0; i < count; i++) {
            h2d(v->values + off, values[i], lengths[i] * sizeof(fr_t), s);
            off += lengths[i];
        }
        device_vec_mark_ready(v, s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:3000-3060
RustError midnight_sppark_bls12_381_fr_device_vec_download(RawFr *out_raw, const void *device_vec, size_t len)
{
    fr_t *out = reinterpret_cast<fr_t *>(out_raw);
    if (!device_vec || (len && !out)) return make_error((int)cudaErrorInvalidValue, "invalid device vector download");
    GB_ENTRY_BEGIN
    auto *v = reinterpret_cast<const fr_device_vec *>(device_vec);
    if (len > v->len) return make_error((int)cudaErrorInvalidValue, "download longer than device vector");
    cudaStream_t s = lane_stream();
    device_vec_wait(v, s);
    d2h(out, v->values, len * sizeof(fr_t), s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

__global__ void scatter_kernel(fr_t *dst, const uint32_t *__restrict__ idx, const fr_t *__restrict__ vals,
                               size_t count)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) dst[idx[i]] = vals[i];
}

// bls12_381_g1_msm.cu:2860-2905
RustError midnight_sppark_bls12_381_fr_device_vec_scatter_host(void *device_vec, const uint32_t *indices, const RawFr *values_raw, size_t count)
{
    const fr_t *values = reinterpret_cast<const fr_t *>(values_raw);
    if (!device_vec || (count && (!indices || !values)))
        return make_error((int)cudaErrorInvalidValue, "invalid device vector scatter");
    if (count == 0) return ok();
    GB_ENTRY_BEGIN
    auto *v = reinterpret_cast<fr_device_vec *>(device_vec);
    for (size_t i = 0; i < count; i++)
        if (indices[i] >= v->len) return make_error((int)cudaErrorInvalidValue, "scatter index out of range");
    cudaStream_t s = lane_stream();
    device_vec_wait(v, s);
    dev_buf<uint32_t> di(count, s);
    h2d(di, indices, count * sizeof(uint32_t), s);
    auto dv = upload(values, count, s);
    scatter_kernel<<<blocks_for(count, 256), 256, 0, s>>>(v->values, di, dv, count);
    GB_CHECK_LAUNCH();
    device_vec_mark_ready(v, s);
    lane_sync(s);
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:2907-2950: [prefix device vector | host suffix]
RustError midnight_sppark_bls12_381_fr_device_vec_concat_host(void **out, const void *prefix_device_vec, const RawFr *suffix_raw, size_t suffix_len)
{
    const fr_t *suffix = reinterpret_cast<const fr_t *>(suffix_raw);
    if (!out || !prefix_device_vec || (suffix_len && !suffix))
        return make_error((int)cudaErrorInvalidValue, "invalid device vector concat");
    *out = nullptr;
    GB_ENTRY_BEGIN
    auto *p = reinterpret_cast<const fr_device_vec *>(prefix_device_vec);
    cudaStream_t s = lane_stream();
    device_vec_wait(p, s);
    fr_device_vec *v = device_vec_new(p->len + suffix_len, s);
    try {
        if (p->len)
            GB_CUDA_OK(cudaMemcpyAsync(v->values, p->values, p->len * sizeof(fr_t), cudaMemcpyDeviceToDevice, s));
        h2d(v->values + p->len, suffix, suffix_len * sizeof(fr_t), s);
        device_vec_mark_ready(v, s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:2952-2998
RustError midnight_sppark_bls12_381_fr_device_vec_concat_many_host(void **out, const void *const *sources, size_t source_count, const RawFr *suffix_raw, size_t suffix_len)
{
    const fr_t *suffix = reinterpret_cast<const fr_t *>(suffix_raw);
    if (!out || (source_count && !sources) || (suffix_len && !suffix))
        return make_error((int)cudaErrorInvalidValue, "invalid device vector concat");
    *out = nullptr;
    GB_ENTRY_BEGIN
    size_t total = suffix_len;
    for (size_t i = 0; i < source_count; i++) {
        if (!sources[i]) return make_error((int)cudaErrorInvalidValue, "null concat source");
        total += reinterpret_cast<const fr_device_vec *>(sources[i])->len;
    }
    cudaStream_t s = lane_stream();
    fr_device_vec *v = device_vec_new(total, s);
    try {
        size_t off = 0;
        for (size_t i = 0; i < source_count; i++) {
            auto *src = reinterpret_cast<const fr_device_vec *>(sources[i]);
            device_vec_wait(src, s);
            if (src->len)
                GB_CUDA_OK(cudaMemcpyAsync(v->values + off, src->values, src->len * sizeof(fr_t),
                                           cudaMemcpyDeviceToDevice, s));
            off += src->len;
        }
        h2d(v->values + off, suffix, suffix_len * sizeof(fr_t), s);
        device_vec_mark_ready(v, s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:3062-3120: selected polynomials of a resident batch
RustError midnight_sppark_bls12_381_fr_device_vec_gather_polys(void **out, const void *source_device_vec,
                                                               size_t poly_len, const uint32_t *indices,
                                                               size_t index_count)
{
    if (!out || !source_device_vec || (index_count && !indices))
        return make_error((int)cudaErrorInvalidValue, "invalid device vector gather");
    *out = nullptr;
    GB_ENTRY_BEGIN
    auto *src = reinterpret_cast<const fr_device_vec *>(source_device_vec);
    for (size_t i = 0; i < index_count; i++)
        if (poly_len && ((size_t)indices[i] + 1) * poly_len > src->len)
            return make_error((int)cudaErrorInvalidValue, "gather index out of range");
    cudaStream_t s = lane_stream();
    device_vec_wait(src, s);
    fr_device_vec *v = device_vec_new(poly_len * index_count, s);
    try {
        for (size_t i = 0; i < index_count; i++)
            if (poly_len)
                GB_CUDA_OK(cudaMemcpyAsync(v->values + i * poly_len, src->values + (size_t)indices[i] * poly_len,
                                           poly_len * sizeof(fr_t), cudaMemcpyDeviceToDevice, s));
        device_vec_mark_ready(v, s);
    } catch (...) {
        device_vec_delete(v);
        throw;
    }
    *out = v;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:3101-3179: per polynomial the first nonzero
// coefficient (starts) and the nonzero count, then the suffixes from the
// first nonzero coefficient on, packed polynomial after polynomial.  With
// out == NULL and out_capacity == 0 only *out_len (the packed length) is
// returned.
RustError midnight_sppark_bls12_381_fr_device_vec_download_nonzero_suffixes(RawFr *out, size_t out_capacity,
                                                                           size_t *out_len, size_t *starts,
                                                                           size_t *nonzero_counts,
                                                                           const void *device_vec,
                                                                           size_t scalar_offset, size_t poly_len,
                                                                           size_t count)
{
    if (!out_len || !starts || !device_vec || poly_len == 0 || count == 0 || count > SIZE_MAX / poly_len ||
        (out_capacity != 0 && !out))
        return make_error((int)cudaErrorInvalidValue, "invalid nonzero suffix download arguments");
    *out_len = 0;
    auto *v = reinterpret_cast<const fr_device_vec *>(device_vec);
    const size_t required = poly_len * count;
    if (scalar_offset > v->len || required > v->len - scalar_offset)
        return make_error((int)cudaErrorInvalidValue, "nonzero suffix range exceeds device vector");
    GB_ENTRY_BEGIN
    cudaStream_t s = lane_stream();
    device_vec_wait(v, s);
    const fr_t *base = v->values + scalar_offset;
    dev_buf<unsigned long long> d_stats(2 * count, s);
    const uint32_t slices = (uint32_t)((poly_len + kSuffixSlice - 1) / kSuffixSlice);
    nonzero_init_kernel<<<blocks_for(count, 256), 256, 0, s>>>(d_stats, count, poly_len);
    GB_CHECK_LAUNCH();
    for (size_t c0 = 0; c0 < count; c0 += 65535) {
        const unsigned m = (unsigned)std::min<size_t>(65535, count - c0);
        nonzero_stats_kernel<<<dim3(slices, m), 256, 0, s>>>(d_stats.get() + c0, d_stats.get() + count + c0,
                                                             base + c0 * poly_len, poly_len);
        GB_CHECK_LAUNCH();
    }
    std::vector<unsigned long long> h(2 * count);
    d2h(h.data(), d_stats, 2 * count * sizeof(unsigned long long), s);
    lane_sync(s);
    size_t total = 0;
    for (size_t p = 0; p < count; p++) {
        starts[p] = (size_t)h[p];
        if (nonzero_counts) nonzero_counts[p] = (size_t)h[count + p];
        total += poly_len - starts[p];
    }
    if (!out && out_capacity == 0) {
        *out_len = total;
        return ok();
    }
    if (total > out_capacity) return make_error((int)cudaErrorInvalidValue, "nonzero suffix output is too small");
    size_t cursor = 0;
    for (size_t p = 0; p < count; p++) {
        const size_t n = poly_len - starts[p];
        if (n) d2h(out + cursor, base + p * poly_len + starts[p], n * sizeof(fr_t), s);
        cursor += n;
    }
    lane_sync(s);
    *out_len = total;
    return ok();
    GB_ENTRY_END
}

// bls12_381_g1_msm.cu:6406-6423 (test hooks): scales a resident vector in
// place on this lane after holding the lane's stream back for delay_ms; the
// vector's ready event moves past the scaling, so a reader on another lane
// waits for it
RustError midnight_sppark_test_delayed_scale(void *device_vec, RawFr scale, uint32_t delay_ms)
{
    if (!device_vec) return make_error((int)cudaErrorInvalidValue, "null device vector");
    GB_ENTRY_BEGIN
    auto *v = reinterpret_cast<fr_device_vec *>(device_vec);
    cudaStream_t s = lane_stream();
    device_vec_wait(v, s);
    lane_sync(s);
    stream_host_delay(s, delay_ms);
    if (v->len) launch_mul_assign(v->values, gb::from_raw(scale), v->len, s);
    device_vec_mark_ready(v, s);
    return ok();
    GB_ENTRY_END
}

void midnight_sppark_bls12_381_fr_device_vec_free(void *device_vec)
{
    device_vec_delete(reinterpret_cast<fr_device_vec *>(device_vec));
}

// Length of a resident vector (library extension used by the host mirror).
size_t gb_fr_device_vec_len(const void *device_vec)
{
    return device_vec ? reinterpret_cast<const fr_device_vec *>(device_vec)->len : 0;
}

}  // extern "C"
