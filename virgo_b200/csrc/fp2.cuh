// F_{p^2} arithmetic, p = 2^61 - 1, i^2 = -1, shared by device kernels and
// host code.
//
// Element layout is {img, real} (two uint64, img first), the in-memory layout
// of prime_field::field_element (reference include/linear_gkr/prime_field.h:93),
// so buffers cross the C ABI unchanged.  Every operation returns a canonical
// value in [0, p) for canonical inputs; the reference's operators do the same
// (prime_field.h:114-172), so results agree bit for bit whatever the order of
// evaluation.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define VG_HD __host__ __device__ __forceinline__
#else
#define VG_HD inline
#endif

namespace vg {

constexpr uint64_t P = 0x1FFFFFFFFFFFFFFFull;  // 2^61 - 1

struct alignas(16) fe {
    uint64_t img, real;
};

VG_HD fe fe_make(uint64_t real, uint64_t img) { fe r; r.real = real; r.img = img; return r; }
VG_HD fe fe_zero() { return fe_make(0, 0); }
VG_HD fe fe_one() { return fe_make(1, 0); }
VG_HD bool fe_eq(fe a, fe b) { return a.real == b.real && a.img == b.img; }
VG_HD bool fe_is_zero(fe a) { return (a.real | a.img) == 0; }

// ---- F_p ----
// For canonical a, b: a + b - p is negative (as a signed 64-bit value)
// exactly when a + b < p, and a - b exactly when a < b; the sign picks the
// result without a 64-bit comparison.
VG_HD uint64_t addp(uint64_t a, uint64_t b)
{
    const uint64_t s = a + b, t = s - P;
    return (int64_t)t < 0 ? s : t;
}
VG_HD uint64_t subp(uint64_t a, uint64_t b)
{
    const uint64_t d = a - b;
    return (int64_t)d < 0 ? d + P : d;
}
VG_HD uint64_t negp(uint64_t a) { return a ? P - a : 0; }

// 64 x 64 -> 128 bits, as one 128-bit product rather than a low and a high one
// formed separately (a * b, __umul64hi): the multiply pipe bounds the field
// kernels, and an F_p2 product took 30.1 clocks per warp that way, 26.8 through
// this type (measured; the halves share their partial products).
typedef unsigned __int128 u128;
VG_HD u128 mul128(uint64_t a, uint64_t b) { return (u128)a * b; }

// x mod p for x < 2^64, partly reduced: the result is below 2^61 + 8.
VG_HD uint64_t foldp(uint64_t x) { return (x & P) + (x >> 61); }
// x mod p, canonical, for x < 2p: x + 1 reaches 2^61 exactly when x >= p.
VG_HD uint64_t canonp(uint64_t x) { return (x + ((x + 1) >> 61)) & P; }

// x mod p as (x & p) + (x >> 61), for x <= 7 * 2^122: x >> 61 is at most
// 7 * 2^61 and x & p at most p, so the sum stays below 2^64.  The callers' sums
// are at most 6 p^2, which folds to at most 7p; with a canonical addend that is
// 8p - 1 = 2^64 - 9, the top of canon64's range.
VG_HD uint64_t fold128(u128 x)
{
    const uint64_t lo = (uint64_t)x, hi = (uint64_t)(x >> 64);
    return (lo & P) + ((hi << 3) | (lo >> 61));
}
// z mod p, canonical, for z <= 2^64 - 9.  With z = q 2^61 + s = q p + (q + s),
// floor(z / p) is q, plus one when q + s >= p, i.e. when q + s + 1 carries into
// bit 61; so floor(z / p) = (z + q + 1) >> 61 and z minus that many p is
// (z + floor(z / p)) mod 2^61: seven instructions where a fold and canonp
// take ten.
VG_HD uint64_t canon64(uint64_t z)
{
    const uint64_t k = (z + (z >> 61) + 1) >> 61;
    return (z + k) & P;
}

// a*b mod p for a, b < 2^61 (canonical).  x = a*b <= (p-1)^2, and
// x = (x >> 61) * 2^61 + (x & p) == (x >> 61) + (x & p) (mod p); both terms are
// at most p and not both p (x < p 2^61 + p), so the sum is below 2p.
VG_HD uint64_t mulp(uint64_t a, uint64_t b) { return canonp(fold128(mul128(a, b))); }

// ---- F_{p^2} ----
VG_HD fe operator+(fe a, fe b) { return fe_make(addp(a.real, b.real), addp(a.img, b.img)); }
VG_HD fe operator-(fe a, fe b) { return fe_make(subp(a.real, b.real), subp(a.img, b.img)); }
VG_HD fe operator-(fe a) { return fe_make(negp(a.real), negp(a.img)); }

// x + (ar + i ai)(br + i bi) for a, x canonical and b of components at most
// 2p, with three products whose 128-bit values are combined before any
// reduction.  With n = 2p - bi and u = ai n (== -ai bi):
//   real: ar br + u <= 4 p^2;
//   img:  t - ar br + u = ar bi + ai br + 2p ai <= 6 p^2, t = (ar + ai)(br + bi)
// (no offset is needed: both are sums of nonnegative products), so each folds
// once to at most 7p, plus x below 8p = 2^64 - 8, the range of canon64.
// 26.4 clocks per warp where the products were folded one by one and the
// result made canonical in two steps (31.9).
VG_HD fe fe_fma2(fe x, fe a, uint64_t br, uint64_t bi)
{
    const u128 ac = mul128(a.real, br), u = mul128(a.img, 2 * P - bi);
    const u128 t = mul128(a.real + a.img, br + bi);
    return fe_make(canon64(fold128(ac + u) + x.real), canon64(fold128(t - ac + u) + x.img));
}
// x + a*b, all canonical: as fe_fma2 with n = p - bi (p is all ones, so one
// exclusive or per word), the sums at most 2 p^2 and 3 p^2.
VG_HD fe fe_fma(fe x, fe a, fe b)
{
    const u128 ac = mul128(a.real, b.real), u = mul128(a.img, b.img ^ P);
    const u128 t = mul128(a.real + a.img, b.real + b.img);
    return fe_make(canon64(fold128(ac + u) + x.real), canon64(fold128(t - ac + u) + x.img));
}
VG_HD fe operator*(fe a, fe b)
{
    const u128 ac = mul128(a.real, b.real), u = mul128(a.img, b.img ^ P);
    const u128 t = mul128(a.real + a.img, b.real + b.img);
    return fe_make(canon64(fold128(ac + u)), canon64(fold128(t - ac + u)));
}
// x + m (v1 - v0), all canonical, the difference left unreduced (v1 + p - v0)
VG_HD fe fe_fma_diff(fe x, fe m, fe v0, fe v1)
{
    return fe_fma2(x, m, v1.real + P - v0.real, v1.img + P - v0.img);
}
// a*b + c*d, all canonical: the products meet in 128 bits (the real sum at
// most 4 p^2, the imaginary one 6 p^2) and are reduced once, 36.6 clocks per
// warp where a product and a fused one took 50.7.
VG_HD fe fe_dot2(fe a, fe b, fe c, fe d)
{
    const u128 ac = mul128(a.real, b.real) + mul128(c.real, d.real);
    const u128 u = mul128(a.img, b.img ^ P) + mul128(c.img, d.img ^ P);
    const u128 t = mul128(a.real + a.img, b.real + b.img) + mul128(c.real + c.img, d.real + d.img);
    return fe_make(canon64(fold128(ac + u)), canon64(fold128(t - ac + u)));
}

// The fold x0 + r (x1 - x0) by a challenge used many times.  The constants are
// 8 rr, 8 ri and 8 (p - ri): the factor 8 puts floor(y / 2^61) of a sum of
// products y into the high word of 8 y, and y mod 2^61 is its low word >> 3, so
// the reduction needs no shift across words.  Four products (the imaginary
// part as dr ri + di rr) with the differences unreduced (x1 + p - x0 < 2p):
// 8 y < 2 (2p)(8p) < 2^127, high word < 4p, low >> 3 <= p, plus x0: below 6p.
// 30 clocks per warp in the paired rounds where a canonical difference and
// fe_fma took 38.
struct fold_r {
    uint64_t r, i, n;
};
VG_HD fold_r fold_prep(fe r)
{
    fold_r f;
    f.r = r.real << 3;
    f.i = r.img << 3;
    f.n = (r.img ^ P) << 3;
    return f;
}
VG_HD uint64_t fold128_8(u128 x) { return (uint64_t)(x >> 64) + ((uint64_t)x >> 3); }
VG_HD fe fe_fold(fe x0, fe x1, fold_r f)
{
    const uint64_t dr = x1.real + P - x0.real, di = x1.img + P - x0.img;
    return fe_make(canon64(fold128_8(mul128(dr, f.r) + mul128(di, f.n)) + x0.real),
                   canon64(fold128_8(mul128(dr, f.i) + mul128(di, f.r)) + x0.img));
}

VG_HD fe fe_double(fe a) { return a + a; }

// The element whose components are given as sums of 21-, 21- and 19-bit limbs
// (i0 + 2^21 i1 + 2^42 i2, and r likewise) over at most 2^21 values, so each sum
// is below 2^42: i1 << 21 is below 2^63, the 2^42 term splits into at most p and
// i2 >> 19 below 2^21, i0 is below 2^42, and the four stay below 2^64 - 9.
VG_HD fe fe_from_limbs(uint64_t i0, uint64_t i1, uint64_t i2, uint64_t r0, uint64_t r1, uint64_t r2)
{
    return fe_make(canon64(r0 + (r1 << 21) + ((r2 << 42) & P) + (r2 >> 19)),
                   canon64(i0 + (i1 << 21) + ((i2 << 42) & P) + (i2 >> 19)));
}

// Operands in F_p (imaginary part zero), such as every layer value of a
// circuit (integer inputs, gates with coefficients in F_p): two products of
// the field's three or four.  v is at most 2p, so each part is below 2p^2.
VG_HD fe fe_fma_real(fe x, fe m, uint64_t v)
{
    return fe_make(canon64(fold128(mul128(m.real, v)) + x.real), canon64(fold128(mul128(m.img, v)) + x.img));
}
VG_HD fe fe_mul_real(fe m, uint64_t v)
{
    return fe_make(canon64(fold128(mul128(m.real, v))), canon64(fold128(mul128(m.img, v))));
}
// x0 + r (x1 - x0) for x0, x1 in F_p (canonical)
VG_HD fe fe_fold_real(uint64_t x0, uint64_t x1, fold_r f)
{
    const uint64_t d = x1 + P - x0;
    return fe_make(canon64(fold128_8(mul128(d, f.r)) + x0), canon64(fold128_8(mul128(d, f.i))));
}

// a * 2^k for canonical a and 0 <= k <= 60: since 2^61 = 1 (mod p), this is a
// left rotation of each 61-bit component
VG_HD uint64_t rotp(uint64_t x, int k) { return ((x << k) | (x >> (61 - k))) & P; }
VG_HD fe fe_mul_pow2(fe a, int k) { return fe_make(rotp(a.real, k), rotp(a.img, k)); }

// multiplication by an element of F_p (img = 0)
VG_HD fe fe_scale(fe a, uint64_t s) { return fe_make(mulp(a.real, s), mulp(a.img, s)); }

VG_HD fe fe_pow(fe x, uint64_t e)
{
    fe r = fe_one();
    while (e) {
        if (e & 1) r = r * x;
        x = x * x;
        e >>= 1;
    }
    return r;
}

// x^(p^2 - 2) = x^-1; p^2 - 2 does not fit 64 bits, so exponentiate by the
// 128-bit value with two 64-bit words.
VG_HD fe fe_inv(fe x)
{
    // p^2 - 2 = (2^61-1)^2 - 2 = 2^122 - 2^62 - 1
    const uint64_t e_hi = (1ull << 58) - 1;            // bits 64..121 of 2^122 - 2^62 - 1
    const uint64_t e_lo = 0xBFFFFFFFFFFFFFFFull;       // low 64 bits
    fe r = fe_one();
    fe b = x;
    for (int i = 0; i < 64; ++i) {
        if ((e_lo >> i) & 1) r = r * b;
        b = b * b;
    }
    for (int i = 0; i < 58; ++i) {
        if ((e_hi >> i) & 1) r = r * b;
        b = b * b;
    }
    return r;
}

// Root of unity of order 2^log_order: the generator of the 2-adic subgroup of
// order 2^62 (real 2^31, img 1033321771269002680), squared 62 - log_order times.
// Same construction as the reference (src/linear_gkr/prime_field.cpp:60-73).
VG_HD fe fe_root_of_unity(int log_order)
{
    fe r = fe_make(2147483648ull, 1033321771269002680ull);
    for (int i = 0; i < 62 - log_order; ++i) r = r * r;
    return r;
}

}  // namespace vg
