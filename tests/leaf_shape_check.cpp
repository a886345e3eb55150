// The launch shapes of the leaf-hash chains (virgo_b200/csrc/leaf_shape.h) over
// chain counts from 1 to 2^21: every chain is covered, shared memory stays
// within the limit the kernels are given, CTA sizes set by hand are taken.
// Exit status 0 when everything agrees.  Built and run by
// tests/test_leaf_shape.py.
#include <cstdio>
#include <initializer_list>
#include "leaf_shape.h"

static int fail(const char *what, ChainForm form, int knob, long n)
{
    printf("%s: form %d, threads %d, %ld chains\n", what, (int)form, knob, n);
    return 1;
}

int main()
{
    long cases = 0;
    for (long n = 1; n <= 1L << 21; n += n < 2048 ? 1 : 977)
        for (int knob : {64, 128, 256})
            for (ChainForm form : {CHAIN_PAIRS, CHAIN_SHA3, CHAIN_SHA256}) {
                const ChainShape s = chain_shape(form, knob, n);
                ++cases;
                if (knob != 256 && s.threads != knob) return fail("size set by hand", form, knob, n);
                if (s.threads != 64 && s.threads != 128 && s.threads != 256) return fail("size", form, knob, n);
                if (s.thread_chains < 0 || s.thread_chains > n || (form != CHAIN_PAIRS && s.thread_chains != n))
                    return fail("split", form, knob, n);
                const long T = s.threads, nt = (s.thread_chains + T - 1) / T;   // k_leaf_chains' own split of the grid
                const long covered = (long)(s.grid - nt) * (T / 2);
                if (s.grid < nt || covered < n - s.thread_chains || covered >= n - s.thread_chains + T / 2)
                    return fail("grid", form, knob, n);
                if (s.smem < 0 || s.smem > CHAIN_MAX_SMEM || s.smem % 128) return fail("shared memory", form, knob, n);
                if (s.smem && (228L << 10) / (s.smem + 1024) * CHAIN_SMS < s.grid) return fail("room", form, knob, n);
            }
    // above 24 warps per scheduler CTAs of 256; below, 64 and with pairs 128
    if (chain_shape(CHAIN_PAIRS, 256, 24 * SCHEDULERS * 32).threads != 256 || chain_shape(CHAIN_SHA3, 256, 1L << 20).threads != 256 ||
        chain_shape(CHAIN_PAIRS, 256, 2048).threads != 128 || chain_shape(CHAIN_PAIRS, 256, 1L << 17).threads != 64)
        return fail("rule", CHAIN_PAIRS, 256, 0);
    // SHA-256: by the warps per scheduler, 18944 chains for each
    for (long w = 1; w < 24; ++w)
        for (long n : {w * 18944 - 18943, w * 18944})
            if (chain_shape(CHAIN_SHA256, 256, n).threads != (w % 2 ? 128 : 256)) return fail("rule", CHAIN_SHA256, 256, n);
    printf("%ld shapes agree\n", cases);
    return 0;
}
