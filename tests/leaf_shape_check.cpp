// The launch shapes of the leaf-hash chains (virgo_b200/csrc/leaf_shape.h) over
// chain counts from 1 to 2^21: every chain is covered, shared memory stays
// within the limit the kernels are given, CTA sizes set by hand are taken.
// Exit status 0 when everything agrees.  Built and run by
// tests/test_leaf_shape.py.
#include <cstdio>
#include <initializer_list>
#include "leaf_shape.h"

static int fail(const char *what, bool pairs, int knob, long n)
{
    printf("%s: pairs %d, threads %d, %ld chains\n", what, pairs, knob, n);
    return 1;
}

int main()
{
    long cases = 0;
    for (long n = 1; n <= 1L << 21; n += n < 2048 ? 1 : 977)
        for (int knob : {64, 128, 256})
            for (bool pairs : {false, true}) {
                const ChainShape s = chain_shape(pairs, knob, n);
                ++cases;
                if (knob != 256 && s.threads != knob) return fail("size set by hand", pairs, knob, n);
                if (s.threads != 64 && s.threads != 128 && s.threads != 256) return fail("size", pairs, knob, n);
                if (s.thread_chains < 0 || s.thread_chains > n || (!pairs && s.thread_chains != n))
                    return fail("split", pairs, knob, n);
                const long T = s.threads, nt = (s.thread_chains + T - 1) / T;   // k_leaf_chains' own split of the grid
                const long covered = (long)(s.grid - nt) * (T / 2);
                if (s.grid < nt || covered < n - s.thread_chains || covered >= n - s.thread_chains + T / 2)
                    return fail("grid", pairs, knob, n);
                if (s.smem < 0 || s.smem > CHAIN_MAX_SMEM || s.smem % 128) return fail("shared memory", pairs, knob, n);
                if (s.smem && (228L << 10) / (s.smem + 1024) * CHAIN_SMS < s.grid) return fail("room", pairs, knob, n);
            }
    // above 24 warps per scheduler CTAs of 256; below, 64 and with pairs 128
    if (chain_shape(true, 256, 24 * SCHEDULERS * 32).threads != 256 || chain_shape(false, 256, 1L << 20).threads != 256 ||
        chain_shape(true, 256, 2048).threads != 128 || chain_shape(true, 256, 1L << 17).threads != 64)
        return fail("rule", true, 256, 0);
    printf("%ld shapes agree\n", cases);
    return 0;
}
