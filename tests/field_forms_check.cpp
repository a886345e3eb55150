// The fused forms of virgo_b200/csrc/fp2.cuh (host build of the code the
// kernels run) against schoolbook products reduced by %, p = 2^61 - 1,
// i^2 = -1: canon64 over its range, x + m (v1 - v0), a b + c d, and the fold
// x0 + r (x1 - x0), on edge values (where the bounds of the unreduced sums are
// reached) and on random ones.  Exit status 0 when everything agrees.
// Built and run by tests/test_field_forms.py.
#include <cstdio>
#include <cstdint>
#include <random>

#include "fp2.cuh"

using u128 = unsigned __int128;
static const uint64_t P = vg::P;

static uint64_t mod(u128 x) { return (uint64_t)(x % P); }
static uint64_t sub(uint64_t a, uint64_t b) { return mod((u128)a + P - b); }
static vg::fe mul(vg::fe a, vg::fe b)
{
    return vg::fe_make(sub(mod((u128)a.real * b.real), mod((u128)a.img * b.img)),
                       mod((u128)mod((u128)a.real * b.img) + mod((u128)a.img * b.real)));
}
static vg::fe add(vg::fe a, vg::fe b) { return vg::fe_make(mod((u128)a.real + b.real), mod((u128)a.img + b.img)); }
static vg::fe dif(vg::fe a, vg::fe b) { return vg::fe_make(sub(a.real, b.real), sub(a.img, b.img)); }

static long n = 0;
static bool check(vg::fe x, vg::fe a, vg::fe b, vg::fe c, vg::fe d)
{
    ++n;
    if (vg::fe_eq(vg::fe_fma_diff(x, a, b, c), add(x, mul(a, dif(c, b)))) &&
        vg::fe_eq(vg::fe_dot2(a, b, c, d), add(mul(a, b), mul(c, d))) &&
        vg::fe_eq(vg::fe_fold(a, b, vg::fold_prep(c)), add(a, mul(c, dif(b, a)))))
        return true;
    printf("mismatch at case %ld\n", n);
    return false;
}

int main()
{
    std::mt19937_64 rng(61);
    for (long i = 0; i < 2000000; ++i) {   // canon64: multiples of p and of 2^61, the top of the range, random
        uint64_t z = rng();
        if (i % 4 == 0) z = (rng() % 9) * (i % 8 ? P : (1ull << 61)) + (rng() % 32) - 16;
        if (z > ~0ull - 8) z = ~0ull - 8 - (rng() & 15);
        if (vg::canon64(z) != z % P) {
            printf("canon64(%llu)\n", (unsigned long long)z);
            return 1;
        }
    }
    const uint64_t edge[] = {0, 1, P - 1, P - 2, P >> 1, 0xFFFFFFFFull, 0x1FFFFFFF00000000ull};
    const int ne = sizeof edge / sizeof edge[0];
    for (long i = 0; i < (long)ne * ne * ne * ne * ne * ne; ++i) {
        long k = i;
        uint64_t e[6];
        for (int j = 0; j < 6; ++j, k /= ne) e[j] = edge[k % ne];
        const vg::fe a = vg::fe_make(e[0], e[1]), b = vg::fe_make(e[2], e[3]), c = vg::fe_make(e[4], e[5]);
        if (!check(vg::fe_make(P - 1, P - 1), a, b, c, a) || !check(b, a, b, c, vg::fe_make(e[5], e[0]))) return 1;
    }
    auto rnd = [&]() { return vg::fe_make(rng() % P, rng() % P); };
    for (long i = 0; i < 1000000; ++i)
        if (!check(rnd(), rnd(), rnd(), rnd(), rnd())) return 1;
    printf("field forms: %ld cases agree\n", n);
    return 0;
}
