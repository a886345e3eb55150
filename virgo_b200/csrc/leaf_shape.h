// Launch shapes of the leaf-hash chains (k_leaf_chains, hash.cu), by the number
// of chains, the hash and VG_TUNE_LEAF_THREADS.  Host code without CUDA
// headers, so that it can be checked on any machine.
#pragma once

constexpr long CHAIN_SMS = 148, SCHEDULERS = CHAIN_SMS * 4;

// How many of `chains` SHA3 chains get a thread each.  Every scheduler of the
// chip (4 per SM) runs whole warps, and one warp of 32 chains keeps it busy for
// a full chain's time, so a last round of warps on some of them costs as much
// as one on all.  Up to half a warp per scheduler is left over as pairs of
// lanes instead, whose warps take about half as long: 98304 chains (5.2 warps
// per scheduler) 1.69 -> 1.57 ms, 24576 (1.3) 571 -> 436 us, 2048 569 -> 169
// us.  From six warps on the rounds average out.
inline long thread_chains(long chains)
{
    const long warps = (chains + 31) / 32, full = warps / SCHEDULERS, rest = warps % SCHEDULERS;
    return full >= 6 || 2 * rest > SCHEDULERS ? chains : full * SCHEDULERS * 32;
}

// Shared memory of a chain launch that leaves room for `ctas` CTAs on an SM
// (228 KB, of which a CTA takes 1 KB for itself), at most CHAIN_MAX_SMEM, the
// one for two.
constexpr int spread_smem(long ctas) { return (int)(((228L << 10) / ctas - 1024) & ~127L); }
constexpr int CHAIN_MAX_SMEM = spread_smem(2);

struct ChainShape {
    long thread_chains;   // the first chains, one thread each; the others on pairs of lanes
    int threads;          // per CTA
    unsigned grid;
    int smem;
};

enum ChainForm { CHAIN_PAIRS, CHAIN_SHA3, CHAIN_SHA256 };   // SHA3 with pairs of lanes, SHA3 on threads, SHA-256

// knob: VG_TUNE_LEAF_THREADS
inline ChainShape chain_shape(ChainForm form, int knob, long chains)
{
    ChainShape s;
    s.thread_chains = form == CHAIN_PAIRS ? thread_chains(chains) : chains;
    // one warp more or less per scheduler matters while there are few: small
    // CTAs spread them (131072 chains 2.26 ms in CTAs of 256, 1.99 of 64);
    // CTAs of 128 put one warp of threads on every scheduler of an SM.  64 and
    // 128 set by hand are taken as they are.
    // SHA-256 takes CTAs of 256, two warps per scheduler that start together,
    // where they come out even: 65 slices of 32768 chains (at most two warps
    // per scheduler) 293 us against 334 in CTAs of 128 and 340 of 64, 65536
    // (four) 579 against 619 and 632.  With an odd number they leave a warp's
    // place empty and CTAs of 128 are faster: 4096 (one) 170 against 291,
    // 49152 (three) 475 against 578, 131072 (seven) 1059 against 1148.
    const long warps = (chains + 31) / 32, per_scheduler = (warps + SCHEDULERS - 1) / SCHEDULERS;
    if (knob != 256) s.threads = knob;
    else if (s.thread_chains < chains) s.threads = 128;
    else if (chains >= 24 * SCHEDULERS * 32) s.threads = 256;
    else if (form == CHAIN_SHA256) s.threads = per_scheduler % 2 ? 128 : 256;
    else s.threads = 64;
    const int T = s.threads;
    s.grid = (unsigned)((s.thread_chains + T - 1) / T + (chains - s.thread_chains + T / 2 - 1) / (T / 2));
    // Room for no more CTAs on an SM than an even spread takes (by shared
    // memory the kernel does not use): beside another stream's kernel the
    // SMs come free one after another, and the first ones took up to 768
    // threads each while others stayed without (73728 chains beside a
    // sumcheck 1707 -> 1166 us; alone 1142).
    const long even = (s.grid + CHAIN_SMS - 1) / CHAIN_SMS;
    s.smem = even > 1 && even < 768 / T ? spread_smem(even) : 0;
    return s;
}
