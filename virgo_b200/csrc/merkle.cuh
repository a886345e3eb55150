// Internal entry points shared by the commitment code.
#pragma once
#include "common.cuh"

// Builds nodes 1 .. sz-1 of a heap-ordered tree (digest words, 4 uint64 per
// node) whose sz = n_leaves_padded leaves are already stored at [sz, 2 sz).
int vg_merkle_build(vg_ctx *c, uint64_t *tree, long n_leaves_padded);
// Leaf hash chains of a slice-major codeword set (see vg_leaf_chain).
int vg_leaf_chain_dev(vg_ctx *c, const fe *cw, int n_slices, long n, uint64_t *leaves);

// Batched leaf chains and Merkle trees of one proof.
constexpr int MAX_HASH_JOBS = 16;
// A tree's levels with at most this many parents are built by CTAs that own a
// subtree of SUB_WIDTH parents and its levels above (vg_merkle_trees)
constexpr long MERKLE_SUB_MAX = 8192;
constexpr int SUB_WIDTH = 64, SUB_LEVELS = 7;
constexpr int PAD_HEIGHTS = 24;   // of the levels above that, which reach 2^(13 + 24) leaves
struct ChainJob {
    const fe *cw;       // slice-major codeword set, slices of n
    long n;
    uint64_t *leaves;   // n / 2 digests
    long begin;         // first thread of this job
};
struct ChainJobs {
    ChainJob j[MAX_HASH_JOBS];
    int count, slices;
    int first;    // first slice: 0, or the leaves hold the digests of the slices before it and the chains go on from them
    long total;   // chains = sum of n / 2
    long thread_chains;   // of those, the first ones hashed by one thread each; the others by two lanes each
};
struct TreeJob {
    uint64_t *tree;   // heap-ordered, leaves at [nleaves, 2 nleaves)
    long nleaves;     // power of two
    long nreal;       // leaves before the padding (H(0^64), the last ones); nleaves when there is none
};
struct TreeJobs {
    TreeJob t[MAX_HASH_JOBS];
    int count;
    bool padded;                      // some nreal < nleaves; then
    uint64_t pad[4 * PAD_HEIGHTS];    // the digest of a subtree of 2^h padding leaves at 4 h
};
int vg_leaf_chains(vg_ctx *c, const ChainJobs &jobs);
// Builds every tree; roots_dev (or null) receives 4 words per tree of at least two leaves, in job order.
int vg_merkle_trees(vg_ctx *c, const TreeJobs &jobs, uint64_t *roots_dev);
