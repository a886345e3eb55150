// The forms of virgo_b200/csrc/fp2.cuh at the ends of the ranges that the
// kernels use them over (host build of the same code), against schoolbook
// arithmetic reduced by %, p = 2^61 - 1, i^2 = -1: products with a factor in F_p
// of up to 2p, folds of values in F_p, a product whose left factor is only partly
// reduced (at most p + 7 per component), and elements put together from limb
// sums over up to 2^21 values.  Exit status 0 when everything agrees.  Built and
// run by tests/test_field_bounds.py.
#include <cstdio>
#include <cstdint>
#include <random>

#include "fp2.cuh"

using u128 = unsigned __int128;
static const uint64_t P = vg::P;

static uint64_t mod(u128 x) { return (uint64_t)(x % P); }
static uint64_t mulm(uint64_t a, uint64_t b) { return mod((u128)mod(a) * mod(b)); }
static uint64_t addm(uint64_t a, uint64_t b) { return mod((u128)a + b); }
static vg::fe mul(vg::fe a, vg::fe b)
{
    return vg::fe_make(mod((u128)mulm(a.real, b.real) + P - mulm(a.img, b.img)), addm(mulm(a.real, b.img), mulm(a.img, b.real)));
}

static long n = 0;
static bool check(vg::fe x, vg::fe m, uint64_t v, uint64_t v1, vg::fe lazy)
{
    ++n;
    const vg::fe mv = vg::fe_make(mulm(m.real, v), mulm(m.img, v));
    const uint64_t c0 = mod(v), c1 = mod(v1), d = mod((u128)c1 + P - c0);
    if (vg::fe_eq(vg::fe_mul_real(m, v), mv) &&
        vg::fe_eq(vg::fe_fma_real(x, m, v), vg::fe_make(addm(x.real, mv.real), addm(x.img, mv.img))) &&
        vg::fe_eq(vg::fe_fold_real(c0, c1, vg::fold_prep(m)), vg::fe_make(addm(c0, mulm(d, m.real)), mulm(d, m.img))) &&
        vg::fe_eq(lazy * m, mul(lazy, m)) && vg::fe_eq(lazy * x, mul(lazy, x)))
        return true;
    printf("mismatch at case %ld\n", n);
    return false;
}

int main()
{
    std::mt19937_64 rng(67);
    const uint64_t canon[] = {0, 1, P - 1, P - 2, P >> 1, 0xFFFFFFFFull};                  // canonical
    const uint64_t twice[] = {0, 1, P - 1, P, P + 1, 2 * P - 1, 2 * P};                    // up to 2p
    const uint64_t part[] = {0, 1, P - 1, P, P + 1, P + 6, P + 7};                         // up to p + 7
    for (uint64_t a : canon) for (uint64_t b : canon) for (uint64_t c : canon) for (uint64_t d : canon)
        for (uint64_t v : twice) for (uint64_t w : twice) for (uint64_t e : part) for (uint64_t f : part)
            if (!check(vg::fe_make(a, b), vg::fe_make(c, d), v, w, vg::fe_make(e, f))) return 1;
    for (long i = 0; i < 1000000; ++i)
        if (!check(vg::fe_make(rng() % P, rng() % P), vg::fe_make(rng() % P, rng() % P), rng() % (2 * P + 1), rng() % (2 * P + 1),
                   vg::fe_make(rng() % (P + 8), rng() % (P + 8))))
            return 1;
    // limb sums: of 2^21 values with every limb full, and random ones below that
    const uint64_t full[3] = {0x1fffffull << 21, 0x1fffffull << 21, 0x7ffffull << 21};
    for (long i = 0; i < 1000000; ++i) {
        uint64_t l[6];
        for (int j = 0; j < 6; ++j) l[j] = i % 64 < 63 && (i >> j) % 2 ? rng() % (full[j % 3] + 1) : full[j % 3];
        const auto want = [](const uint64_t *q) { return mod((u128)q[0] + ((u128)q[1] << 21) + ((u128)q[2] << 42)); };
        if (!vg::fe_eq(vg::fe_from_limbs(l[0], l[1], l[2], l[3], l[4], l[5]), vg::fe_make(want(l + 3), want(l)))) {
            printf("limbs, case %ld\n", i);
            return 1;
        }
    }
    printf("field bounds: %ld cases agree\n", n);
    return 0;
}
