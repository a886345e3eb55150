// Shared definitions for the virgo_b200 CUDA library: the context object,
// error reporting and launch bookkeeping, and block reductions over F_{p^2}.
#pragma once
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>
#include <string>
#include <vector>
#include "fp2.cuh"
#include "virgo_b200.h"

using vg::fe;

struct TwEntry {
    uint64_t key_real, key_img;  // the root
    int logn;
    fe *lo;   // w^i, i < 4096
    fe *hi;   // w^(4096 j), j < max(1, n / 4096)
    fe *full = nullptr;   // w^e, e < n, for the NTT's column twiddles (small n only), or null
};

// Kernel families timed by the optional per-launch profiler (vg_ctx_profile).
enum KernelFamily {
    KF_NTT = 0, KF_LEAF_CHAIN, KF_MERKLE, KF_FRI_FOLD, KF_VIRTUAL_ORACLE, KF_EVAL, KF_SCATTER1, KF_SCATTER2,
    KF_FINALIZE, KF_ROUND, KF_REDUCE, KF_OTHER, KF_GATHER_ROUND, KF_COUNT
};
struct ProfRec {
    int fam;
    cudaEvent_t a, b;
    double bytes;
    bool shared_a;   // a is the previous record's b (back-to-back launches)
};
struct TraceRec {
    int fam;
    double ms, bytes;
};

struct vg_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    int hash_kind = VG_HASH_SHA3_256;
    long long launches = 0;
    std::vector<TwEntry> tw_cache;
    // reusable device scratch (grown on demand, freed with the context)
    void *scratch = nullptr;
    size_t scratch_cap = 0;
    void *scratch2 = nullptr;
    size_t scratch2_cap = 0;
    fe *partials = nullptr;  // block partial sums of reductions
    size_t partials_cap = 0;
    unsigned long long *gsum = nullptr;   // grid_sum's limb sums and counter (vg_grid_scratch), zero between launches
    fe *pinned = nullptr;    // pinned host staging for small results
    size_t pinned_cap = 0;
    // pinned ring for uploads from pageable host memory (vg_h2d_staged)
    static constexpr int RING = 4;
    char *ring = nullptr;    // RING chunks, ring_next the one to fill next
    int ring_next = 0;
    std::vector<void *> retired_pinned;   // outgrown pinned blocks, freed with the context
    cudaEvent_t ring_ev[RING] = {};
    // per-launch profiler: event pairs around launches of each kernel family
    bool profiling = false;
    std::vector<ProfRec> prof;
    std::vector<cudaEvent_t> event_pool;
    std::vector<TraceRec> trace;   // every profiled launch in order
    long long prof_launches[KF_COUNT] = {0};
    double prof_ms[KF_COUNT] = {0}, prof_bytes[KF_COUNT] = {0};
    // back-to-back profiled launches share one event (the end of one is the
    // start of the next), so the profiler adds one event per launch
    bool prof_chain = false;
    cudaEvent_t prof_prev_end = nullptr;
    long long prof_prev_launches = -1;
};

// Profiler hooks around one launch: no-ops unless profiling is on.  Events are
// recorded on the context stream without synchronising; vg_ctx_profile_read
// resolves them.
void vg_prof_begin(vg_ctx *c, int fam, ProfRec *r);
void vg_prof_end(vg_ctx *c, ProfRec *r, double bytes);
struct ProfScope {
    vg_ctx *c;
    ProfRec r;
    double bytes;
    bool on;
    ProfScope(vg_ctx *ctx, int fam, double b) : c(ctx), bytes(b), on(ctx->profiling)
    {
        if (on) vg_prof_begin(c, fam, &r);
    }
    ~ProfScope()
    {
        if (on) vg_prof_end(c, &r, bytes);
    }
};

// ---- errors ----
int vg_fail(int code, const char *fmt, ...);
#define VG_CHECK_CUDA(call)                                                              \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess)                                                           \
            return vg_fail(VG_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call,        \
                           cudaGetErrorString(e_));                                      \
    } while (0)
#define VG_TRY(expr)                   \
    do {                               \
        int rc_ = (expr);              \
        if (rc_ != VG_OK) return rc_;  \
    } while (0)
#define VG_LAUNCHED(ctx)                                                                   \
    do {                                                                                   \
        (ctx)->launches++;                                                                 \
        cudaError_t e_ = cudaGetLastError();                                               \
        if (e_ != cudaSuccess)                                                             \
            return vg_fail(VG_ERR_CUDA, "%s:%d launch: %s", __FILE__, __LINE__,             \
                           cudaGetErrorString(e_));                                        \
    } while (0)

// Host-to-device copy on the context stream.  Pageable sources go through the
// context's ring of pinned chunks (the host copies one while those before it
// are on their way, across calls as well), so concurrent sessions do not
// serialise on the driver's staging.  A pageable source may be reused on return; a pinned or device
// source is copied directly and must stay valid until the stream reaches the
// copy.
int vg_h2d_staged(vg_ctx *c, void *dst, const void *src, size_t bytes);

// Grows a pinned host buffer geometrically without synchronising: the
// outgrown block is retired (freed when the context is destroyed), since
// cudaFreeHost would wait for the whole device.
int vg_pinned_grow(vg_ctx *c, void **p, size_t *cap, size_t bytes);

// stream-ordered device memory from the device pool (see ctx.cu)
int vg_alloc(vg_ctx *c, void **p, size_t bytes);
void vg_release(vg_ctx *c, void *p);

// scratch buffers owned by the context; contents do not survive other calls
int vg_scratch(vg_ctx *ctx, size_t bytes, void **p);
int vg_scratch2(vg_ctx *ctx, size_t bytes, void **p);
int vg_partials(vg_ctx *ctx, size_t n, fe **p);
// Pinned host blocks of at least `bytes` (cap receives the size), kept for the
// next taker when given back; null is ignored.  Synchronise the streams that
// use a block before giving it back.
int vg_pinned_take(void **p, size_t bytes, size_t *cap);
void vg_pinned_give(void *p);
int vg_pinned(vg_ctx *ctx, size_t n, fe **p);
void vg_gkr_context_gone(const vg_ctx *x);   // gkr.cu: x is about to be destroyed, its stream is done
// grid_sum's device words for the context's kernels (up to 14 values per sum)
int vg_grid_scratch(vg_ctx *ctx, unsigned long long **gacc, unsigned **counter);
int vg_twiddles(vg_ctx *ctx, fe root, int logn, const fe **lo, const fe **hi);
bool vg_is_device_ptr(const void *p);
bool vg_reads_in_place(const void *p, int device);   // reads_in_place (memory_place.h) of what p points to

static inline unsigned grid_for(long n, int threads)
{
    long g = (n + threads - 1) / threads;
    return (unsigned)(g < 1 ? 1 : g);
}

// ---- reductions ----
__device__ __forceinline__ fe shfl_down_fe(fe x, int off)
{
    fe r;
    r.real = __shfl_down_sync(0xffffffffu, x.real, off);
    r.img = __shfl_down_sync(0xffffffffu, x.img, off);
    return r;
}
__device__ __forceinline__ fe warp_sum(fe x)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x = x + shfl_down_fe(x, off);
    return x;
}
// Sum of K values over the block; result valid in thread 0.  sm holds
// K * 32 elements.  Field addition is exact and commutative, so the result is
// independent of the reduction order.
template <int K>
__device__ __forceinline__ void block_sum(fe (&v)[K], fe *sm)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = warp_sum(v[k]);
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) sm[k * 32 + wid] = v[k];
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            fe x = lane < nw ? sm[k * 32 + lane] : vg::fe_zero();
            v[k] = warp_sum(x);
        }
    }
}

// Sums of K values over a grid, exact and fast at the end of a kernel: each
// 61-bit component is cut into limbs of 21, 21 and 19 bits, one warp-wide
// integer reduction adds a limb over a warp (26 bits), the warps' sums meet
// in shared memory (30 bits) and the CTAs' in 64-bit atomics.  A tree of field
// additions over shuffles (block_sum) is five dependent steps of some 60
// clocks each at two levels, then again over the CTAs' partials.
constexpr int LIMBS = 6;   // limbs of a field element
// limb sums of x over the calling warp (all 32 lanes), the same in every lane
__device__ __forceinline__ void warp_limbs(fe x, uint32_t (&l)[LIMBS])
{
    const uint32_t M = 0x1fffff;
    l[0] = __reduce_add_sync(0xffffffffu, (uint32_t)x.img & M);
    l[1] = __reduce_add_sync(0xffffffffu, (uint32_t)(x.img >> 21) & M);
    l[2] = __reduce_add_sync(0xffffffffu, (uint32_t)(x.img >> 42));
    l[3] = __reduce_add_sync(0xffffffffu, (uint32_t)x.real & M);
    l[4] = __reduce_add_sync(0xffffffffu, (uint32_t)(x.real >> 21) & M);
    l[5] = __reduce_add_sync(0xffffffffu, (uint32_t)(x.real >> 42));
}
// Sums acc over the grid (at most 16 warps per CTA, at most 2^10 CTAs): true
// in the last CTA to finish, with the K totals in tot (shared memory) for
// every thread; false in the others.  gacc: 6 K words, zero before the launch
// and again after it, as *counter.
template <int K>
__device__ __forceinline__ bool grid_sum(const fe (&acc)[K], uint32_t (&sw)[16][LIMBS * K], fe (&tot)[K],
                                         unsigned long long *gacc, unsigned *counter)
{
    __shared__ bool last;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        uint32_t l[LIMBS];
        warp_limbs(acc[k], l);
        if (lane == 0) {
#pragma unroll
            for (int j = 0; j < LIMBS; ++j) sw[wid][LIMBS * k + j] = l[j];
        }
    }
    __syncthreads();
    unsigned long long s = 0;
    if (t < LIMBS * K) {
        for (int w = 0; w < nw; ++w) s += sw[w][t];
        if (gridDim.x > 1) atomicAdd(&gacc[t], s);
    }
    if (gridDim.x > 1) {
        __threadfence();
        __syncthreads();
        if (t == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
        __syncthreads();
        if (!last) return false;
        __threadfence();
        if (t < LIMBS * K) {
            s = __ldcg(&gacc[t]);
            gacc[t] = 0;
        }
        if (t == 0) *counter = 0;
    }
    // the limbs of value k are in six consecutive threads of the first warps
    __shared__ unsigned long long sl[LIMBS * K];
    if (t < LIMBS * K) sl[t] = s;
    __syncthreads();
    if (t < K) tot[t] = vg::fe_from_limbs(sl[6 * t], sl[6 * t + 1], sl[6 * t + 2], sl[6 * t + 3], sl[6 * t + 4], sl[6 * t + 5]);
    __syncthreads();
    return true;
}

// sum of `nparts` groups of K partials (layout [part][K]) into out[K]
int vg_reduce_partials(vg_ctx *ctx, const fe *parts, int nparts, int K, fe *out_dev);

// The device's launch-shape parameter `key` (VG_TUNE_*; tune.cu).
long vg_tune_value(int device, int key);
