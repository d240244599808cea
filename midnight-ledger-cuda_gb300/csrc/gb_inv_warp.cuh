// Inversion in Fp or Fr by one warp, for kernels that invert one value per
// block.
//
// Bernstein and Yang's division steps ("Fast constant-time gcd computation and
// modular inversion", 2019), with delta starting at 1/2: from (f, g) = (p, a)
// each step replaces (delta, f, g) by (1 - delta, g, (g - f) / 2) when delta >
// 0 and g is odd, else by (1 + delta, f, (g + (g mod 2) f) / 2), until g = 0
// and f = +-1.  The start at 1/2 and the variable-time order of the steps, runs
// of zeros and several bits of g at once, are those that libsecp256k1 describes
// in doc/safegcd_implementation.md.
//
// Thirty steps depend on the low 30 bits of f and g only and are one integer
// matrix (u v; q r) / 2^30, found by every lane alike; the matrix is applied to
// f and g, and mod p to (d, e) with d a = f, e a = g (mod p), with one 30-bit
// limb a lane: two or three products a lane and one carry from each side.  Limbs
// are signed and carried once, so they stay within 2^30 + 2 of zero and the
// products' sums within 2^62.
//
// A dependent chain of 30 (Fr: 20) x about 10 short loops instead of some 460
// (380) products: about 25 us for one warp against 400 us (150) for a Fermat
// power and 180 (120) for one thread's binary Euclid.  30 x 30 and 20 x 30
// steps are above the step count's bounds for 381 and 255 bits (878 and 588),
// and the result is checked all the same, with the Fermat power as the way out.
#pragma once

#include "gb_field.cuh"

#if defined(__CUDACC__) || defined(GB_WARP_ON_HOST)  // a test runs the lanes in turn
namespace gb {

// modulus and 2^(96 N) mod it in 32-bit words, 1 / modulus mod 2^30
static __constant__ uint32_t kFpWords[12] = {0xffffaaabu, 0xb9feffffu, 0xb153ffffu, 0x1eabfffeu, 0xf6b0f624u, 0x6730d2a0u, 0xf38512bfu, 0x64774b84u, 0x434bacd7u, 0x4b1ba7b6u, 0x397fe69au, 0x1a0111eau};
static __constant__ uint32_t kFpR3[12] = {0xd94ca1e0u, 0xed48ac6bu, 0x03a7adf8u, 0x315f831eu, 0x615e29ddu, 0x9a53352au, 0x921e1761u, 0x34c04e5eu, 0x65724728u, 0x2512d435u, 0x91755d4du, 0x0aa63460u};
static __constant__ uint32_t kFrWords[8] = {0x00000001u, 0xffffffffu, 0xfffe5bfeu, 0x53bda402u, 0x09a1d805u, 0x3339d808u, 0x299d7d48u, 0x73eda753u};
static __constant__ uint32_t kFrR3[8] = {0x439b73afu, 0xc62c1807u, 0x8cf06990u, 0x1b3e0d18u, 0xc7b5f418u, 0x73d13c71u, 0xc8db33e9u, 0x6e2a5bb9u};

template <class Cfg>
struct inv_cfg;
template <>
struct inv_cfg<FpCfg> {
    static constexpr int LIMBS = 13, BATCHES = 30;
    static constexpr uint32_t INV30 = 0x00030003u;
    static __device__ __forceinline__ const uint32_t *words() { return kFpWords; }
    static __device__ __forceinline__ const uint32_t *r3() { return kFpR3; }
};
template <>
struct inv_cfg<FrCfg> {
    static constexpr int LIMBS = 9, BATCHES = 20;
    static constexpr uint32_t INV30 = 0x00000001u;
    static __device__ __forceinline__ const uint32_t *words() { return kFrWords; }
    static __device__ __forceinline__ const uint32_t *r3() { return kFrR3; }
};

// one 30-bit limb a lane of a value's words (0 past the last limb)
template <class Cfg>
__device__ __forceinline__ int32_t inv_limb(const uint32_t *w, uint32_t lane)
{
    if (lane >= inv_cfg<Cfg>::LIMBS) return 0;
    const uint32_t bit = 30 * lane, k = bit >> 5, off = bit & 31;
    const uint32_t hi = k + 1 < Cfg::N ? w[k + 1] : 0u;
    return (int32_t)(__funnelshift_r(w[k], hi, off) & 0x3fffffffu);
}

// (u a + v b + m p) / 2^30, limb by limb; the sum's low 30 bits are zero
template <int LIMBS>
__device__ __forceinline__ int32_t inv_apply(int32_t a, int32_t b, int32_t u, int32_t v, int32_t m, int32_t p,
                                             uint32_t lane)
{
    const int64_t c = (int64_t)u * a + (int64_t)v * b + (int64_t)m * p;
    const int32_t lo = (int32_t)((uint32_t)c & 0x3fffffffu);
    const int32_t from_above = __shfl_down_sync(0xffffffffu, lo, 1);
    const int64_t n = (c >> 30) + (lane < LIMBS - 1 ? from_above : 0);
    const int32_t carry = (int32_t)(n >> 30);
    const int32_t from_below = __shfl_up_sync(0xffffffffu, carry, 1);
    // the top limb keeps its carry and sign
    return (lane < LIMBS - 1 ? (int32_t)((uint32_t)n & 0x3fffffffu) : (int32_t)n) + (lane ? from_below : 0);
}

// the division steps' inverse of *in (see inverse_warp), not yet checked.  Only
// the low bits of F and G count, which wrap around: unsigned.
template <class Cfg>
__device__ __forceinline__ mont_t<Cfg> inverse_steps(const mont_t<Cfg> *in)
{
    using C = inv_cfg<Cfg>;
    constexpr int L = C::LIMBS, N = Cfg::N;
    const uint32_t lane = threadIdx.x & 31u;
    const int32_t p = inv_limb<Cfg>(C::words(), lane);
    int32_t f = p, g = inv_limb<Cfg>(in->v, lane), d = 0, e = lane == 0;
    int32_t theta = 0;  // delta - 1/2
    for (int batch = 0; batch < C::BATCHES; batch++) {
        const uint32_t f0 = __shfl_sync(0xffffffffu, f, 0), f1 = __shfl_sync(0xffffffffu, f, 1);
        const uint32_t g0 = __shfl_sync(0xffffffffu, g, 0), g1 = __shfl_sync(0xffffffffu, g, 1);
        uint32_t F = f0 + (f1 << 30), G = g0 + (g1 << 30);
        int32_t u = 1, v = 0, q = 0, r = 1, left = 30;
        for (;;) {  // at most 30 turns: each but the last takes a bit or more
            const int z = __ffs((int)(G | 0xffffffffu << left)) - 1;
            G = (uint32_t)((int32_t)G >> z);
            u = (int32_t)((uint32_t)u << z);
            v = (int32_t)((uint32_t)v << z);
            theta += z;
            left -= z;
            if (left == 0) break;
            if (theta >= 0) {
                theta = -theta - 1;
                const uint32_t T = F;
                F = G, G = 0u - T;
                int32_t t = u;
                u = q, q = -t;
                t = v, v = r, r = -t;
            }
            // the next -theta steps keep f, so up to five bits of g go at
            // once: (3 F) ^ 2 is 1 / F mod 32
            const int bits = min(min(left, -theta), 5);
            const int32_t w = (int32_t)((0u - G) * ((3u * F) ^ 2u) & ((1u << bits) - 1u));
            G += F * (uint32_t)w;
            q += u * w;
            r += v * w;
        }
        const int32_t fn = inv_apply<L>(f, g, u, v, 0, p, lane);
        g = inv_apply<L>(f, g, q, r, 0, p, lane);
        f = fn;
        // multiples of p, centred, that clear the low 30 bits
        const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0), e0 = __shfl_sync(0xffffffffu, e, 0);
        const uint32_t td = (uint32_t)u * d0 + (uint32_t)v * e0, te = (uint32_t)q * d0 + (uint32_t)r * e0;
        const int32_t md = (int32_t)((0u - td * C::INV30) << 2) >> 2, me = (int32_t)((0u - te * C::INV30) << 2) >> 2;
        const int32_t dn = inv_apply<L>(d, e, u, v, md, p, lane);
        e = inv_apply<L>(d, e, q, r, me, p, lane);
        d = dn;
    }
    // |d| < 16 p: +-d + 16 p as 32-bit words, then mod p
    const int32_t sign = (__shfl_sync(0xffffffffu, f, 0) & 3) == 1 ? 1 : -1;
    const int64_t x = (int64_t)sign * d + 16ll * p;
    uint32_t w[N + 1];
    {
        int64_t carry = 0;
        uint64_t acc = 0;
        int have = 0, out = 0;
#pragma unroll
        for (int i = 0; i <= L; i++) {
            carry += i < L ? __shfl_sync(0xffffffffu, x, i) : 0;
            acc |= (uint64_t)((uint32_t)carry & 0x3fffffffu) << have;
            carry >>= 30;
            have += 30;
            if (have >= 32 && out <= N) {
                w[out++] = (uint32_t)acc;
                acc >>= 32;
                have -= 32;
            }
        }
    }
#pragma unroll
    for (int s = 4; s >= 0; s--) {
        uint32_t t[N + 1];
        uint64_t br = 0;
#pragma unroll
        for (int i = 0; i <= N; i++) {
            const uint32_t lo = i < N ? Cfg::mod(i < N ? i : 0) : 0u, below = i ? Cfg::mod(i ? i - 1 : 0) : 0u;
            const uint32_t m = s ? (lo << s) | (below >> (32 - s)) : lo;
            const uint64_t y = (uint64_t)w[i] - m - br;
            t[i] = (uint32_t)y;
            br = (y >> 32) & 1;
        }
#pragma unroll
        for (int i = 0; i <= N; i++) w[i] = br ? w[i] : t[i];
    }
    // w is 1 / (a R), R = 2^(32 N): times R^3 / R gives the Montgomery form
    mont_t<Cfg> y, r3;
#pragma unroll
    for (int i = 0; i < N; i++) y.v[i] = w[i], r3.v[i] = C::r3()[i];
    return y * r3;
}

// the inverse (Montgomery form in and out) of *in, nonzero; every lane of the
// warp takes part and returns it
template <class Cfg>
__device__ __noinline__ mont_t<Cfg> inverse_warp(const mont_t<Cfg> *in)
{
    mont_t<Cfg> y = inverse_steps<Cfg>(in);
    if (*in * y != mont_t<Cfg>::one()) y = in->inverse();
    return y;
}

}  // namespace gb
#endif
