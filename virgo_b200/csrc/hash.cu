// Hash kernels: batched 64-byte hashing, Merkle trees and the FRI leaf hash
// chains.  All are integer-ALU bound (Keccak-f[1600]: 24 rounds of 64-bit
// xor/and-not/rotate; SHA-256: 2 x 64 rounds of 32-bit ops).
#include <algorithm>
#include <cstring>
#include <mutex>
#include "common.cuh"
// 2^n, n < 32, for the multiply-pipe rotations (VG_MROT_*); filled per device
// at first use (pow2_table)
#define VG_HASH_MULROT 1
static __constant__ uint32_t vg_pow2c[32];
#include "hash.cuh"
#include "merkle.cuh"
#include "leaf_shape.h"

void virgo_hash64_kind(int kind, const void *src, void *dst);   // host/src/hash_host.cpp

namespace {

constexpr int HASH_THREADS = 128;

__device__ __forceinline__ void load_digest(const uint64_t *p, uint64_t h[4])
{
    const ulonglong2 a = reinterpret_cast<const ulonglong2 *>(p)[0], b = reinterpret_cast<const ulonglong2 *>(p)[1];
    h[0] = a.x;
    h[1] = a.y;
    h[2] = b.x;
    h[3] = b.y;
}
__device__ __forceinline__ void load_digest2(const uint64_t *p, uint64_t w[8])
{
    const ulonglong2 *q = (const ulonglong2 *)p;
    ulonglong2 a = q[0], b = q[1], c = q[2], d = q[3];
    w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y; w[4] = c.x; w[5] = c.y; w[6] = d.x; w[7] = d.y;
}
__device__ __forceinline__ void store_digest(uint64_t *p, const uint64_t d[4])
{
    ulonglong2 *q = (ulonglong2 *)p;
    q[0] = make_ulonglong2(d[0], d[1]);
    q[1] = make_ulonglong2(d[2], d[3]);
}

template <int KIND>
__global__ void k_hash64(const uint64_t *__restrict__ msgs, uint64_t *__restrict__ out, long n)
{
    long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t w[8], d[4];
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = msgs[i * 8 + k];
    vg::hash64<KIND>(w, d);
#pragma unroll
    for (int k = 0; k < 4; ++k) out[i * 4 + k] = d[k];
}

}  // namespace

// ---- Merkle trees ----
// Padding leaves are all H(0^64), so a subtree of 2^h of them has one digest
// per height; a ragged tree's levels write it where such nodes are instead of
// hashing (70001 leaves: 70 thousand hashes, not 192 thousand).  The digests
// are constants of the hash, formed on the host.
static void pad_digests(int kind, uint64_t *pad)
{
    uint64_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int h = 0; h < PAD_HEIGHTS; ++h) {
        virgo_hash64_kind(kind, w, pad + 4 * h);
        for (int i = 0; i < 8; ++i) w[i] = pad[4 * h + (i & 3)];
    }
}
static const uint64_t *pad_table(int kind)
{
    struct Table {
        uint64_t d[2][4 * PAD_HEIGHTS];
        Table()
        {
            pad_digests(0, d[0]);
            pad_digests(1, d[1]);
        }
    };
    static const Table t;
    return t.d[kind == VG_HASH_SHA256 ? 1 : 0];
}

// tree[0] cleared, the leaves and the padding after them: 16 bytes per thread
__global__ void k_tree_leaves(const ulonglong2 *leaves, long n, long size, ulonglong2 p0, ulonglong2 p1, ulonglong2 *tree)
{
    const long stride = (long)gridDim.x * blockDim.x;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < 2 * size; i += stride)
        tree[2 * size + i] = i < 2 * n ? leaves[i] : (i & 1 ? p1 : p0);
    if (blockIdx.x == 0 && threadIdx.x < 2) tree[threadIdx.x] = make_ulonglong2(0, 0);
}

// ---- leaf hash chains ----
// Leaf k of a codeword set with per-slice length n: h = 0; for s:
// h = H(c[s][k] || c[s][k + n/2] || h).  Several sets in one launch: chain t is
// leaf t - begin of the job whose range holds t.  One thread per chain (a
// warp reads 32 consecutive k of one slice, 512 contiguous bytes per load; the
// next slice's pair is loaded before the current hash), except the chains from
// thread_chains on, which take a pair of lanes each (vg_leaf_chains chooses).
// A launch may stop before the last slice and another go on from the digests
// it left (jobs.first).
__device__ __forceinline__ int chain_job(const ChainJobs &jobs, long t)
{
    int q = 0;
    while (q + 1 < jobs.count && t >= jobs.j[q + 1].begin) ++q;
    return q;
}

template <int KIND, int ROT>
__device__ __forceinline__ void thread_chain(const ChainJobs &jobs, long t)
{
    const int q = chain_job(jobs, t);
    const fe *__restrict__ c = jobs.j[q].cw;
    const long n = jobs.j[q].n, half = n >> 1, k = t - jobs.j[q].begin;
    uint64_t h[4] = {0, 0, 0, 0};
    if (jobs.first) load_digest(jobs.j[q].leaves + 4 * k, h);
    fe a = c[(long)jobs.first * n + k], b = c[(long)jobs.first * n + k + half];
    for (int s = jobs.first; s < jobs.slices; ++s) {
        fe na = a, nb = b;
        if (s + 1 < jobs.slices) {
            na = c[(long)(s + 1) * n + k];
            nb = c[(long)(s + 1) * n + k + half];
        }
        uint64_t w[8] = {a.img, a.real, b.img, b.real, h[0], h[1], h[2], h[3]};
        vg::hash64_rot<KIND, ROT>(w, h);
        a = na;
        b = nb;
    }
    store_digest(jobs.j[q].leaves + 4 * k, h);
}

// a chain on lanes 2j and 2j + 1; t at most total - 1 (every lane takes part
// in the shuffles), stored when `active`
__device__ __forceinline__ void pair_chain(const ChainJobs &jobs, long t, bool active)
{
    const bool odd = threadIdx.x & 1;
    const int q = chain_job(jobs, t);
    const fe *__restrict__ c = jobs.j[q].cw;
    const long n = jobs.j[q].n, half = n >> 1, k = t - jobs.j[q].begin;
    uint32_t s25[25];
#pragma unroll
    for (int i = 0; i < 4; ++i) s25[i] = 0;
    if (jobs.first && active) {
        uint64_t h[4];
        load_digest(jobs.j[q].leaves + 4 * k, h);
#pragma unroll
        for (int i = 0; i < 4; ++i) s25[i] = vg::pair_half(h[i], odd);
    }
    fe a = c[(long)jobs.first * n + k], b = c[(long)jobs.first * n + k + half];
    for (int s = jobs.first; s < jobs.slices; ++s) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s25[4 + i] = s25[i];
        s25[0] = vg::pair_half(a.img, odd);
        s25[1] = vg::pair_half(a.real, odd);
        s25[2] = vg::pair_half(b.img, odd);
        s25[3] = vg::pair_half(b.real, odd);
        if (s + 1 < jobs.slices) {
            a = c[(long)(s + 1) * n + k];
            b = c[(long)(s + 1) * n + k + half];
        }
        vg::sha3_256_64_pair(s25, odd);
    }
    uint32_t *out = reinterpret_cast<uint32_t *>(jobs.j[q].leaves + 4 * k) + (odd ? 1 : 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t w = vg::pair_word(s25[i], odd);
        if (active) out[2 * i] = w;
    }
}

template <int KIND, int T, int ROT>
__global__ void __launch_bounds__(T, 768 / T) k_leaf_chains(const __grid_constant__ ChainJobs jobs)
{
    const long nt = (jobs.thread_chains + T - 1) / T;   // CTAs of one thread per chain
    if (blockIdx.x < nt) {
        const long t = blockIdx.x * (long)T + threadIdx.x;
        if (t < jobs.thread_chains) thread_chain<KIND, ROT>(jobs, t);
    } else if (KIND == VG_HASH_SHA3_256 && ROT == 3) {
        const long t = jobs.thread_chains + (blockIdx.x - nt) * (T / 2) + (threadIdx.x >> 1);
        pair_chain(jobs, min(t, jobs.total - 1), t < jobs.total);
    }
}

// ---- leaf chains, one warp per chain (SHA3-256 only) ----
// Lanes 0..3 load the chain's next pair (a.img, a.real, b.img, b.real) as the
// first four message words; lanes 4..7 take the running digest, which the
// previous permutation left in lanes 0..3; lanes 8 and 16 hold the padding.
__device__ __forceinline__ uint64_t chain_word(const fe *__restrict__ c, long off, long half, int l)
{
    const uint64_t *p = (const uint64_t *)(c + off + (l < 2 ? 0 : half));
    return p[l & 1];
}

__device__ __forceinline__ void warp_chain(const fe *__restrict__ c, int n_slices, long n, long k,
                                           uint64_t *__restrict__ out)
{
    const unsigned FULL = 0xffffffffu;
    const int l = threadIdx.x & 31;
    const long half = n >> 1;
    const vg::KeccakLanes K = vg::keccak_lanes(l);
    uint32_t lo = 0, hi = 0;
    uint64_t word = l < 4 ? chain_word(c, k, half, l) : 0;
    for (int s = 0; s < n_slices; ++s) {
        const uint64_t next = (l < 4 && s + 1 < n_slices) ? chain_word(c, (long)(s + 1) * n + k, half, l) : 0;
        const uint32_t dl = __shfl_sync(FULL, lo, (l - 4) & 31), dh = __shfl_sync(FULL, hi, (l - 4) & 31);
        if (l < 4) {
            lo = (uint32_t)word;
            hi = (uint32_t)(word >> 32);
        } else if (l < 8) {
            lo = dl;
            hi = dh;
        } else {
            lo = l == 8 ? 0x06u : 0u;
            hi = l == 16 ? 0x80000000u : 0u;
        }
        vg::keccak_f_warp(lo, hi, K);
        word = next;
    }
    if (l < 4) out[l] = lo | ((uint64_t)hi << 32);
}

constexpr int WARP_CHAIN_THREADS = 128;

__global__ void __launch_bounds__(WARP_CHAIN_THREADS) k_leaf_chains_warp(const __grid_constant__ ChainJobs jobs)
{
    const long w = ((long)blockIdx.x * WARP_CHAIN_THREADS + threadIdx.x) >> 5;
    if (w >= jobs.total) return;   // whole warps
    const int q = chain_job(jobs, w);
    const long k = w - jobs.j[q].begin;
    warp_chain(jobs.j[q].cw, jobs.slices, jobs.j[q].n, k, jobs.j[q].leaves + 4 * k);
}

static unsigned warp_chain_grid(long chains)
{
    return (unsigned)((chains * 32 + WARP_CHAIN_THREADS - 1) / WARP_CHAIN_THREADS);
}

// leaf hashing form for a launch of `chains` chains: one warp per chain when
// SHA3 and at most VG_TUNE_LEAF_WARP_MAX chains
static bool use_warp_chains(vg_ctx *c, long chains)
{
    return c->hash_kind == VG_HASH_SHA3_256 && chains <= vg_tune_value(c->device, VG_TUNE_LEAF_WARP_MAX);
}

// One Merkle level (parents of height `height`) of every tree that still has
// more than MERKLE_SUB_MAX parents there, one thread per parent.
template <int KIND>
__global__ void __launch_bounds__(HASH_THREADS) k_merkle_levels(const __grid_constant__ TreeJobs jobs, int height, long total)
{
    long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (t >= total) return;
    int q = 0;
    for (; q < jobs.count; ++q) {
        const long cnt = jobs.t[q].nleaves >> height;
        if (cnt <= MERKLE_SUB_MAX) continue;
        if (t < cnt) break;
        t -= cnt;
    }
    if (q >= jobs.count) return;
    const long p = (jobs.t[q].nleaves >> height) + t;
    uint64_t w[8], d[4];
    if (jobs.padded && (t << height) >= jobs.t[q].nreal) {
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = jobs.pad[4 * height + i];
    } else {
        load_digest2(jobs.t[q].tree + 8 * p, w);
        vg::hash64<KIND>(w, d);
    }
    store_digest(jobs.t[q].tree + 4 * p, d);
}

// Subtrees: a CTA hashes 64 neighbouring parents of a tree's next level, then
// their 32 parents, up to seven levels, the digests of a level staying in
// shared memory for the next.  The levels are a chain of dependent hashes, so
// what counts is one hash's latency: SHA3 runs on pairs of lanes.  Trees of up
// to 2^14 leaves take two launches of 14 such levels where one CTA took 4.6 us
// and more for each of the top nine and a launch went to each level below.
struct SubJobs {
    struct {
        uint64_t *tree;
        long cnt;       // parents of the first level
        int begin;      // first CTA
    } t[MAX_HASH_JOBS];
    int count;
    uint64_t *roots;    // 4 words per tree, or null
    int root_at[MAX_HASH_JOBS];
};
template <int KIND>
__global__ void __launch_bounds__(2 * SUB_WIDTH) k_merkle_sub(const __grid_constant__ SubJobs J)
{
    // two levels' digests in turn: SHA3 as (even, odd) halves of 4 words
    __shared__ __align__(16) uint32_t sd[2][SUB_WIDTH][8];
    const int t = threadIdx.x;
    int q = 0;
    while (q + 1 < J.count && (int)blockIdx.x >= J.t[q + 1].begin) ++q;
    uint64_t *tree = J.t[q].tree;
    const long first = ((long)blockIdx.x - J.t[q].begin) * SUB_WIDTH;   // of this CTA among the level's parents
    long cnt = J.t[q].cnt;                                              // the level's parents
    int own = (int)min((long)SUB_WIDTH, cnt);                           // of them this CTA's
    for (int lvl = 0; own >= 1; ++lvl, own >>= 1, cnt >>= 1) {
        const long p0 = cnt + (first >> lvl);   // first parent's node
        if (KIND == VG_HASH_SHA3_256) {
            const bool odd = t & 1;
            const int j = t >> 1;
            if ((t & ~31) < 2 * own) {   // whole warps
                const int jj = min(j, own - 1);
                uint32_t a[25];
                if (lvl == 0) {
                    uint64_t w[8];
                    load_digest2(tree + 8 * (p0 + jj), w);
#pragma unroll
                    for (int i = 0; i < 8; ++i) a[i] = vg::pair_half(w[i], odd);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) a[i] = sd[lvl & 1][2 * jj + (i >> 2)][2 * (i & 3) + odd];
                }
                vg::sha3_256_64_pair(a, odd);
                uint32_t *out = reinterpret_cast<uint32_t *>(tree + 4 * (p0 + jj)) + (odd ? 1 : 0);
                uint32_t w32[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w32[i] = vg::pair_word(a[i], odd);
                if (j < own) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) out[2 * i] = w32[i];
                    if (cnt == 1 && J.roots) {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            reinterpret_cast<uint32_t *>(J.roots + 4 * J.root_at[q])[2 * i + odd] = w32[i];
                    }
                }
                if (j < own) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) sd[~lvl & 1][j][2 * i + odd] = a[i];
                }
            }
        } else if (t < own) {
            uint64_t w[8], d[4];
            if (lvl == 0) {
                load_digest2(tree + 8 * (p0 + t), w);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) w[i] = reinterpret_cast<const uint64_t *>(sd[lvl & 1][2 * t + (i >> 2)])[i & 3];
            }
            vg::hash64<KIND>(w, d);
            store_digest(tree + 4 * (p0 + t), d);
            if (cnt == 1 && J.roots)
                for (int i = 0; i < 4; ++i) J.roots[4 * J.root_at[q] + i] = d[i];
#pragma unroll
            for (int i = 0; i < 4; ++i) reinterpret_cast<uint64_t *>(sd[~lvl & 1][t])[i] = d[i];
        }
        __syncthreads();
    }
}

// fills vg_pow2c on the current device, once per device
static int pow2_table(int dev)
{
    static std::mutex mu;
    static std::vector<bool> done;
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= (int)done.size()) done.resize(dev + 1, false);
    if (!done[dev]) {
        uint32_t p[32];
        for (int i = 0; i < 32; ++i) p[i] = 1u << i;
        VG_CHECK_CUDA(cudaMemcpyToSymbol(vg_pow2c, p, sizeof p));
        done[dev] = true;
    }
    return VG_OK;
}

// The kernel attribute belongs to the kernel on the device, not to a launch:
// it is raised once to the largest launch's size, since setting it to the
// launch's own size races with launches of other sizes from other threads (a
// launch above the value of the moment is refused).
template <int KIND, int T, int ROT>
static int chain_smem_attribute(int dev)
{
    static std::mutex mu;
    static std::vector<bool> done;
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= (int)done.size()) done.resize(dev + 1, false);
    if (!done[dev]) {
        VG_CHECK_CUDA(cudaFuncSetAttribute(k_leaf_chains<KIND, T, ROT>, cudaFuncAttributeMaxDynamicSharedMemorySize, CHAIN_MAX_SMEM));
        done[dev] = true;
    }
    return VG_OK;
}

int vg_leaf_chains(vg_ctx *c, const ChainJobs &jobs_in)
{
    if (jobs_in.total < 1) return VG_OK;
    ChainJobs jobs = jobs_in;
    double bytes = 0;
    for (int q = 0; q < jobs.count; ++q)
        bytes += 16.0 * (jobs.slices - jobs.first) * (double)jobs.j[q].n + (jobs.first ? 64.0 : 32.0) * (double)(jobs.j[q].n >> 1);
    ProfScope ps(c, KF_LEAF_CHAIN, bytes);
    if (jobs.first == 0 && use_warp_chains(c, jobs.total)) {
        k_leaf_chains_warp<<<warp_chain_grid(jobs.total), WARP_CHAIN_THREADS, 0, c->stream>>>(jobs);
    } else {
        const int rot = c->hash_kind == VG_HASH_SHA3_256 ? (int)vg_tune_value(c->device, VG_TUNE_LEAF_ROT) : 0;
        if (rot == 1 || rot == 2) VG_TRY(pow2_table(c->device));
        const ChainForm form = c->hash_kind == VG_HASH_SHA256 ? CHAIN_SHA256 : (rot == 3 ? CHAIN_PAIRS : CHAIN_SHA3);
        const ChainShape shape = chain_shape(form, (int)vg_tune_value(c->device, VG_TUNE_LEAF_THREADS), jobs.total);
        const int T = shape.threads, smem = shape.smem;
        const unsigned grid = shape.grid;
        jobs.thread_chains = shape.thread_chains;
#define VG_CHAINS_ONE(KIND, TT, ROT)                                          \
    {                                                                         \
        if (smem > 48 * 1024) VG_TRY((chain_smem_attribute<KIND, TT, ROT>(c->device))); \
        k_leaf_chains<KIND, TT, ROT><<<grid, TT, smem, c->stream>>>(jobs);    \
    }
#define VG_CHAINS_LAUNCH(TT)                                                      \
    {                                                                             \
        if (c->hash_kind == VG_HASH_SHA256) VG_CHAINS_ONE(VG_HASH_SHA256, TT, 0)  \
        else if (rot == 1) VG_CHAINS_ONE(VG_HASH_SHA3_256, TT, 1)                 \
        else if (rot == 2) VG_CHAINS_ONE(VG_HASH_SHA3_256, TT, 2)                 \
        else if (rot == 3) VG_CHAINS_ONE(VG_HASH_SHA3_256, TT, 3)                 \
        else VG_CHAINS_ONE(VG_HASH_SHA3_256, TT, 0)                               \
    }
        if (T == 64) VG_CHAINS_LAUNCH(64)
        else if (T == 256) VG_CHAINS_LAUNCH(256)
        else VG_CHAINS_LAUNCH(128)
#undef VG_CHAINS_LAUNCH
#undef VG_CHAINS_ONE
    }
    VG_LAUNCHED(c);
    return VG_OK;
}

int vg_merkle_trees(vg_ctx *c, const TreeJobs &jobs, uint64_t *roots_dev)
{
    if (jobs.count < 1) return VG_OK;
    for (int height = 1;; ++height) {
        long total = 0;
        for (int q = 0; q < jobs.count; ++q) {
            const long cnt = jobs.t[q].nleaves >> height;
            if (cnt > MERKLE_SUB_MAX) total += cnt;
        }
        if (total == 0) break;
        ProfScope ps(c, KF_MERKLE, 96.0 * (double)total);
        if (c->hash_kind == VG_HASH_SHA256)
            k_merkle_levels<VG_HASH_SHA256><<<grid_for(total, HASH_THREADS), HASH_THREADS, 0, c->stream>>>(jobs, height, total);
        else
            k_merkle_levels<VG_HASH_SHA3_256><<<grid_for(total, HASH_THREADS), HASH_THREADS, 0, c->stream>>>(jobs, height, total);
        VG_LAUNCHED(c);
    }
    // the levels below, seven at a time
    long cnt[MAX_HASH_JOBS];
    for (int q = 0; q < jobs.count; ++q) cnt[q] = std::min(jobs.t[q].nleaves >> 1, MERKLE_SUB_MAX);
    for (;;) {
        SubJobs J{};
        J.roots = roots_dev;
        int ctas = 0;
        double parents = 0;
        for (int q = 0; q < jobs.count; ++q) {
            if (cnt[q] < 1) continue;
            J.t[J.count] = {jobs.t[q].tree, cnt[q], ctas};
            J.root_at[J.count++] = q;
            ctas += (int)((cnt[q] + SUB_WIDTH - 1) / SUB_WIDTH);
            parents += 2.0 * (double)cnt[q];
            cnt[q] >>= SUB_LEVELS;
        }
        if (!ctas) break;
        ProfScope ps(c, KF_MERKLE, 96.0 * parents);
        if (c->hash_kind == VG_HASH_SHA256)
            k_merkle_sub<VG_HASH_SHA256><<<ctas, 2 * SUB_WIDTH, 0, c->stream>>>(J);
        else
            k_merkle_sub<VG_HASH_SHA3_256><<<ctas, 2 * SUB_WIDTH, 0, c->stream>>>(J);
        VG_LAUNCHED(c);
    }
    return VG_OK;
}

// ------------------------------------------------------------------ host
int vg_merkle_build(vg_ctx *c, uint64_t *tree, long n_leaves_padded)
{
    // leaves already in tree[sz .. 2 sz); builds nodes 1 .. sz-1
    TreeJobs j{};
    j.t[0] = {tree, n_leaves_padded, n_leaves_padded};
    j.count = 1;
    return vg_merkle_trees(c, j, nullptr);
}

int vg_leaf_chain_dev(vg_ctx *c, const fe *cw, int n_slices, long n, uint64_t *leaves)
{
    ChainJobs j{};
    j.j[0] = {cw, n, leaves, 0};
    j.count = 1;
    j.total = n >> 1;
    j.slices = n_slices;
    return vg_leaf_chains(c, j);
}

extern "C" int vg_hash64(vg_ctx *c, const void *msgs, void *digests, long n)
{
    if (!c || !msgs || !digests || n < 0) return vg_fail(VG_ERR_ARG, "vg_hash64: bad argument");
    if (n == 0) return VG_OK;
    if (c->hash_kind == VG_HASH_SHA256)
        k_hash64<VG_HASH_SHA256><<<grid_for(n, HASH_THREADS), HASH_THREADS, 0, c->stream>>>((const uint64_t *)msgs, (uint64_t *)digests, n);
    else
        k_hash64<VG_HASH_SHA3_256><<<grid_for(n, HASH_THREADS), HASH_THREADS, 0, c->stream>>>((const uint64_t *)msgs, (uint64_t *)digests, n);
    VG_LAUNCHED(c);
    return VG_OK;
}

extern "C" int vg_merkle_tree(vg_ctx *c, const vg_digest *leaves, long n, vg_digest *tree)
{
    if (!c || !leaves || !tree || n < 1) return vg_fail(VG_ERR_ARG, "vg_merkle_tree: bad argument");
    long sz = 1;
    while (sz < n) sz <<= 1;
    TreeJobs j{};
    j.t[0] = {(uint64_t *)tree, sz, n};
    j.count = 1;
    const uint64_t *pad = pad_table(c->hash_kind);
    j.padded = n < sz;
    memcpy(j.pad, pad, sizeof j.pad);
    const vg_digest *src = leaves;
    if (!vg_reads_in_place(leaves, c->device)) {   // copied first
        VG_CHECK_CUDA(cudaMemcpyAsync(tree + sz, leaves, n * sizeof(vg_digest), cudaMemcpyDeviceToDevice, c->stream));
        src = tree + sz;
    }
    k_tree_leaves<<<std::min<unsigned>(grid_for(2 * sz, 256), 148u * 8u), 256, 0, c->stream>>>(
        (const ulonglong2 *)src, n, sz, make_ulonglong2(pad[0], pad[1]), make_ulonglong2(pad[2], pad[3]), (ulonglong2 *)tree);
    VG_LAUNCHED(c);
    return vg_merkle_trees(c, j, nullptr);
}

extern "C" int vg_leaf_chain(vg_ctx *c, const vg_fe *cw, int n_slices, long n, vg_digest *leaves)
{
    if (!c || !cw || !leaves || n_slices < 1 || n < 2 || (n & (n - 1)))
        return vg_fail(VG_ERR_ARG, "vg_leaf_chain: bad argument");
    return vg_leaf_chain_dev(c, (const fe *)cw, n_slices, n, (uint64_t *)leaves);
}
