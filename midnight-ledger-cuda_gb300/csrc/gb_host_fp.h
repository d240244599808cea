// Fp and G1 on the host, for the few point operations at the end of an MSM:
// 6 x 64-bit limbs, Montgomery products with 128-bit intermediates, the binary
// extended Euclid for inverses (blst's p1_to_affine is what the reference's
// Rust callers apply to every commitment).  Variable time, as the device's
// accumulation of the same sums is: commitments are public, and a caller whose
// scalars may not show in the time of a call masks them (the scrambled entry
// point).  A memory image of these types is that of fp_t and xyzz_t.
#pragma once

#include <stdint.h>

namespace gb {
namespace hostfp {

typedef unsigned __int128 u128;
struct fp64 {
    uint64_t l[6];
};

static const fp64 kP = {{0xb9feffffffffaaabull, 0x1eabfffeb153ffffull, 0x6730d2a0f6b0f624ull, 0x64774b84f38512bfull,
                         0x4b1ba7b6434bacd7ull, 0x1a0111ea397fe69aull}};
static const uint64_t kN0 = 0x89f3fffcfffcfffdull;  // -p^-1 mod 2^64
static const fp64 kOne = {{0x760900000002fffdull, 0xebf4000bc40c0002ull, 0x5f48985753c758baull, 0x77ce585370525745ull,
                           0x5c071a97a256ec6dull, 0x15f65ec3fa80e493ull}};  // R mod p
// R^3 mod p (R = 2^384): a Montgomery product with it takes the plain
// inverse of a Montgomery value zR to the Montgomery form of 1/z
static const fp64 kR3 = {{0xed48ac6bd94ca1e0ull, 0x315f831e03a7adf8ull, 0x9a53352a615e29ddull, 0x34c04e5e921e1761ull,
                          0x2512d43565724728ull, 0x0aa6346091755d4dull}};

inline bool is_zero(const fp64 &a)
{
    uint64_t t = 0;
    for (int i = 0; i < 6; i++) t |= a.l[i];
    return t == 0;
}

inline bool geq(const fp64 &a, const fp64 &b)
{
    for (int i = 5; i >= 0; i--)
        if (a.l[i] != b.l[i]) return a.l[i] > b.l[i];
    return true;
}

inline void sub_in(fp64 &a, const fp64 &b)
{
    uint64_t borrow = 0;
    for (int i = 0; i < 6; i++) {
        const u128 d = (u128)a.l[i] - b.l[i] - borrow;
        a.l[i] = (uint64_t)d;
        borrow = (uint64_t)(d >> 64) & 1;
    }
}

inline void add_in(fp64 &a, const fp64 &b)
{
    uint64_t carry = 0;
    for (int i = 0; i < 6; i++) {
        const u128 t = (u128)a.l[i] + b.l[i] + carry;
        a.l[i] = (uint64_t)t;
        carry = (uint64_t)(t >> 64);
    }
}

inline void shr1(fp64 &a)
{
    for (int i = 0; i < 5; i++) a.l[i] = (a.l[i] >> 1) | (a.l[i + 1] << 63);
    a.l[5] >>= 1;
}

// x / 2 mod p for x < p (x + p < 2^382: no carry out of six limbs)
inline void half_mod(fp64 &x)
{
    if (x.l[0] & 1) add_in(x, kP);
    shr1(x);
}

// a - b mod p for a, b < p
inline void sub_mod(fp64 &a, const fp64 &b)
{
    if (geq(a, b)) {
        sub_in(a, b);
    } else {
        add_in(a, kP);
        sub_in(a, b);
    }
}

inline void reduce(fp64 &a)
{
    while (geq(a, kP)) sub_in(a, kP);
}

// a b R^-1 mod p (CIOS), inputs < p, result < p
inline fp64 mont_mul(const fp64 &a, const fp64 &b)
{
    uint64_t t[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = 0; i < 6; i++) {
        uint64_t carry = 0;
        for (int j = 0; j < 6; j++) {
            const u128 x = (u128)a.l[j] * b.l[i] + t[j] + carry;
            t[j] = (uint64_t)x;
            carry = (uint64_t)(x >> 64);
        }
        u128 x = (u128)t[6] + carry;
        t[6] = (uint64_t)x;
        t[7] = (uint64_t)(x >> 64);
        const uint64_t m = t[0] * kN0;
        x = (u128)m * kP.l[0] + t[0];
        carry = (uint64_t)(x >> 64);
        for (int j = 1; j < 6; j++) {
            x = (u128)m * kP.l[j] + t[j] + carry;
            t[j - 1] = (uint64_t)x;
            carry = (uint64_t)(x >> 64);
        }
        x = (u128)t[6] + carry;
        t[5] = (uint64_t)x;
        t[6] = t[7] + (uint64_t)(x >> 64);
    }
    fp64 r;
    for (int i = 0; i < 6; i++) r.l[i] = t[i];
    if (t[6] || geq(r, kP)) sub_in(r, kP);
    return r;
}

// a^-1 mod p for 0 < a < p (binary extended Euclid: x1 a = u, x2 a = v)
inline fp64 inverse(const fp64 &a)
{
    fp64 u = a, v = kP, x1 = {{1, 0, 0, 0, 0, 0}}, x2 = {{0, 0, 0, 0, 0, 0}};
    auto is_one = [&](const fp64 &w) {
        for (int i = 1; i < 6; i++)
            if (w.l[i]) return false;
        return w.l[0] == 1;
    };
    while (!is_one(u) && !is_one(v)) {
        while (!(u.l[0] & 1)) {
            shr1(u);
            half_mod(x1);
        }
        while (!(v.l[0] & 1)) {
            shr1(v);
            half_mod(x2);
        }
        if (geq(u, v)) {
            sub_in(u, v);
            sub_mod(x1, x2);
        } else {
            sub_in(v, u);
            sub_mod(x2, x1);
        }
    }
    return is_one(u) ? x1 : x2;
}


// ---- XYZZ points (x = X / ZZ, y = Y / ZZZ; ZZ = 0 at infinity)

struct xyzz64 {
    fp64 x, y, zz, zzz;
};

inline fp64 sub(fp64 a, const fp64 &b)
{
    sub_mod(a, b);
    return a;
}

inline fp64 twice(fp64 a)
{
    add_in(a, a);
    if (geq(a, kP)) sub_in(a, kP);
    return a;
}

inline xyzz64 infinity()
{
    return xyzz64{kOne, kOne, {{0, 0, 0, 0, 0, 0}}, {{0, 0, 0, 0, 0, 0}}};
}

// dbl-2008-s-1
inline xyzz64 dbl(const xyzz64 &p)
{
    const fp64 u = twice(p.y);
    if (is_zero(p.zz) || is_zero(u)) return infinity();
    const fp64 v = mont_mul(u, u), w = mont_mul(u, v), s = mont_mul(p.x, v), xx = mont_mul(p.x, p.x);
    fp64 m = twice(xx);
    add_in(m, xx);
    if (geq(m, kP)) sub_in(m, kP);
    xyzz64 r;
    r.x = sub(mont_mul(m, m), twice(s));
    r.y = sub(mont_mul(m, sub(s, r.x)), mont_mul(w, p.y));
    r.zz = mont_mul(v, p.zz);
    r.zzz = mont_mul(w, p.zzz);
    return r;
}

// add-2008-s with the equal and opposite cases
inline xyzz64 add(const xyzz64 &p, const xyzz64 &q)
{
    if (is_zero(p.zz)) return q;
    if (is_zero(q.zz)) return p;
    const fp64 u1 = mont_mul(p.x, q.zz), s1 = mont_mul(p.y, q.zzz);
    const fp64 d = sub(mont_mul(q.x, p.zz), u1), e = sub(mont_mul(q.y, p.zzz), s1);
    if (is_zero(d)) return is_zero(e) ? dbl(p) : infinity();
    const fp64 dd = mont_mul(d, d), ddd = mont_mul(d, dd), t = mont_mul(u1, dd);
    xyzz64 r;
    r.x = sub(sub(mont_mul(e, e), ddd), twice(t));
    r.y = sub(mont_mul(e, sub(t, r.x)), mont_mul(s1, ddd));
    r.zz = mont_mul(mont_mul(p.zz, q.zz), dd);
    r.zzz = mont_mul(mont_mul(p.zzz, q.zzz), ddd);
    return r;
}

}  // namespace hostfp
}  // namespace gb
