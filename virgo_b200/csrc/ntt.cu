// Batched number-theoretic transform over F_{p^2}, natural order in and out.
//
// n = 2^logn is split into factors F_1 .. F_P (each <= 2^10).  Passes 1..P-1
// are "column passes": inside every block of the current size A, DFTs of size
// F_q run down the columns (stride A / F_q) and output k of column c is scaled
// by w_A^(c k), in place.  Pass P is a "row pass": each contiguous block of
// F_P elements is transformed and written to its natural-order position
// k_1 + F_1 (k_2 + F_2 (... + F_{P-1} k_P)).  This is the four-step
// decomposition applied recursively, so no separate bit-reversal pass is
// needed and every pass reads and writes runs of >= G contiguous elements.
//
// Inside a CTA each sub-DFT is a decimation-in-time transform (bit-reversed
// load, natural-order result) in steps of three radix-2 stages held in
// registers, the tile in shared memory between steps.  The 8-point DFT of a
// step needs no products: the 4th root of unity is i, and the 8th roots are
// +-2^30 (1 +- i) (2^30 is 1/sqrt 2 mod 2^61 - 1), a sum and a rotation of the
// 61-bit words; its sums stay unreduced until they are stored.  What remains
// are the seven twiddle products per eight elements and step, 0.29 per element
// and stage against 0.38 in radix 4: the multiply pipe bounds the pass.
//
// CTAs loop over tiles and fetch the next one (asynchronous copies into the
// other half of their shared memory) while they transform the current one.
// 65 slices of 2^16 from 2^11 coefficients take 117 us (163 us with radix-4
// steps, reduced sums, loads waited for and the padding transformed; 124 us
// with radix-4 steps in 80 registers and three CTAs per SM), one 2^22
// transform 216 us (284).
//
// A zero-padded input (encoding: 2^11 coefficients into 2^16) leaves the first
// stages of the first pass with one nonzero entry per group, which they only
// copy: the pass starts at the first stage that has work (PassArgs::z).
//
// Twiddles: w^e for e < n comes from two small tables, lo[e & 4095] *
// hi[e >> 12], built once per root and cached in the context; for n up to
// 2^TW_FULL_MAX_LOG every pass reads w^e from a full table instead
// (one load in place of two loads and a product per element).
#include "common.cuh"
#include <algorithm>
#include <mutex>
#include <vector>

namespace {

constexpr int NTT_THREADS = 256, NTT_CTAS = 2;   // 128 registers: an 8-point step and its twiddles
constexpr int MAX_LM = 10, MAX_TILE_LOG = 13;

struct PassArgs {
    const fe *in;
    fe *out;
    long in_len;        // valid input elements per batch item (first pass), zero beyond
    long in_bstride, out_bstride;
    int logn, lm, logG;
    int kind;           // 0 column pass, 1 row pass, 2 single pass
    int logA;           // column pass: block size
    int nfac;           // row pass: number of previous factors
    int fac[6];         // row pass: their logs, F_1 first
    const fe *tw_lo, *tw_hi;
    const fe *tw_full;  // w^e for every e < n, or null
    int tw_shift;       // tw_full's root is w_n^(2^tw_shift): w_n^e at e >> tw_shift
    int z;              // stages skipped: only rows below 2^(lm - z) are nonzero
    int c8;             // w_8 = (2^30 (1 + i))^c8, c8 odd: results of the fixed 8-point DFT are permuted by it
    long nblocks;       // tiles per batch item
    long ntiles;        // tiles of the whole batch
    int rot;            // last pass: multiply by 2^rot (n^-1 = 2^(61 - logn)), 0 none
};

// a table entry (never written while a transform runs)
__device__ __forceinline__ fe ld_tab(const fe *p)
{
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(p));
    fe x;
    x.img = v.x;
    x.real = v.y;
    return x;
}
__device__ __forceinline__ fe tw_pow(const fe *__restrict__ lo, const fe *__restrict__ hi, uint64_t e)
{
    fe a = ld_tab(lo + (e & 4095));
    uint64_t h = e >> 12;
    if (h) a = a * ld_tab(hi + h);
    return a;
}

__device__ __forceinline__ int bitrev(int x, int bits) { return bits ? (int)(__brev((unsigned)x) >> (32 - bits)) : 0; }

// ---- small DFTs on lazily reduced values ----
// Inputs: x[0] at most p + 7 per component, the others canonical (products, or
// values from memory).  Sums wrap mod 2^64 on the way; each result carries the
// multiple of p that makes it nonnegative and is below 2^64, then folds once
// (fold: at most p + 7).  Inputs in bit-reversed order, outputs in natural
// order of the root i.
using vg::P;
__device__ __forceinline__ fe raw(uint64_t re, uint64_t im) { return vg::fe_make(re, im); }
__device__ __forceinline__ fe fold(uint64_t re, uint64_t im) { return vg::fe_make(vg::foldp(re), vg::foldp(im)); }

__device__ __forceinline__ void dft_regs(fe (&x)[2])
{
    const fe a = x[0], b = x[1];
    x[0] = fold(a.real + b.real, a.img + b.img);
    x[1] = fold(a.real + 2 * P - b.real, a.img + 2 * P - b.img);
}
__device__ __forceinline__ void dft_regs(fe (&x)[4])
{
    const fe E = raw(x[0].real + x[1].real, x[0].img + x[1].img);     // [0, 2p + 7]
    const fe O = raw(x[0].real - x[1].real, x[0].img - x[1].img);     // [-p, p + 7]
    const fe F = raw(x[2].real + x[3].real, x[2].img + x[3].img);     // [0, 2p]
    const fe D = raw(x[3].img - x[2].img, x[2].real - x[3].real);     // i (x2 - x3): [-p, p]
    x[0] = fold(E.real + F.real, E.img + F.img);
    x[1] = fold(O.real + 2 * P + D.real, O.img + 2 * P + D.img);
    x[2] = fold(E.real + 2 * P - F.real, E.img + 2 * P - F.img);
    x[3] = fold(O.real + 2 * P - D.real, O.img + 2 * P - D.img);
}
// v 2^30 for a signed v above -2^63: in [-2^32, p + 2^32]
__device__ __forceinline__ uint64_t rot30(uint64_t v) { return ((v << 30) & P) + (uint64_t)((int64_t)v >> 31); }
__device__ __forceinline__ void dft_regs(fe (&x)[8])
{
    // C: the 4-point DFT of x0..x3; D: of x4..x7 (all canonical, so each
    // component of D, and D + i D, is within +-4 (p - 1), a signed word)
    const fe A0 = raw(x[0].real + x[1].real, x[0].img + x[1].img), B0 = raw(x[0].real - x[1].real, x[0].img - x[1].img);
    const fe A1 = raw(x[2].real + x[3].real, x[2].img + x[3].img), B1 = raw(x[3].img - x[2].img, x[2].real - x[3].real);
    const fe A2 = raw(x[4].real + x[5].real, x[4].img + x[5].img), B2 = raw(x[4].real - x[5].real, x[4].img - x[5].img);
    const fe A3 = raw(x[6].real + x[7].real, x[6].img + x[7].img), B3 = raw(x[7].img - x[6].img, x[6].real - x[7].real);
    const fe C0 = raw(A0.real + A1.real, A0.img + A1.img);                            // [0, 4p + 7]
    const fe C2 = raw(A0.real + 4 * P - A1.real, A0.img + 4 * P - A1.img);            // 4p + [-2p, 2p + 7]
    const fe C1 = raw(B0.real + 4 * P + B1.real, B0.img + 4 * P + B1.img);            // 4p + [-2p, 2p + 7]
    const fe C3 = raw(B0.real + 4 * P - B1.real, B0.img + 4 * P - B1.img);
    const fe D0 = fold(A2.real + A3.real, A2.img + A3.img);                           // [0, p + 3]
    const fe E2 = fold(A2.real + 2 * P - A3.real, A2.img + 2 * P - A3.img);           // [0, p + 3]
    const fe E1 = raw(B2.real + B3.real, B2.img + B3.img), E3 = raw(B2.real - B3.real, B2.img - B3.img);   // +-2p
    // times the 8th root: (1 + i) 2^30; times its cube: i (1 + i) 2^30
    const fe D1 = raw(rot30(E1.real - E1.img), rot30(E1.real + E1.img));
    const fe G3 = raw(rot30(E3.real - E3.img), rot30(E3.real + E3.img));
    x[0] = fold(C0.real + D0.real, C0.img + D0.img);                                  // at most 5p + 10
    x[4] = fold(C0.real + 2 * P - D0.real, C0.img + 2 * P - D0.img);
    x[1] = fold(C1.real + D1.real, C1.img + D1.img);                                  // [p - 2^32, 7p + 2^32]
    x[5] = fold(C1.real - D1.real, C1.img - D1.img);
    x[2] = fold(C2.real - E2.img, C2.img + E2.real);                                  // i E2
    x[6] = fold(C2.real + E2.img, C2.img - E2.real);
    x[3] = fold(C3.real - G3.img, C3.img + G3.real);                                  // i G3
    x[7] = fold(C3.real + G3.img, C3.img - G3.real);
}
// x at most 2^61 + 6 per component, canonical
__device__ __forceinline__ fe canon(fe x) { return vg::fe_make(vg::canonp(x.real), vg::canonp(x.img)); }

// A tile: m rows of G columns (or items) of one batch item.
struct Tile {
    const fe *in;
    fe *out;
    long col_base, C;                // column pass: element (g, r) at col_base + g + r C
    long row_base, rowW, pos_rest;   // row pass: element (g, r) at row_base + g rowW m + r
};

__device__ __forceinline__ Tile tile_at(const PassArgs &a, long tile)
{
    Tile T{};
    const long item = tile / a.nblocks, blk = tile - item * a.nblocks;
    T.in = a.in + item * a.in_bstride;
    T.out = a.out + item * a.out_bstride;
    if (a.kind == 0) {
        T.C = (1L << a.logA) >> a.lm;
        const int lc = a.logA - a.lm - a.logG;           // tiles per block (log)
        T.col_base = ((blk >> lc) << a.logA) + ((blk & ((1L << lc) - 1)) << a.logG);
    } else if (a.kind == 1) {
        T.rowW = (1L << a.logn >> a.lm) >> a.fac[0];      // transforms per k_1 value
        const long t_rest = blk % T.rowW, k10 = (blk / T.rowW) << a.logG;
        T.row_base = (k10 * T.rowW + t_rest) << a.lm;
        // natural position of the digits k_2..k_{P-1} held by t_rest
        long tmp = t_rest, acc = 0;
        int shift_lo = 0;
        for (int q = 0; q < a.nfac; ++q) shift_lo += a.fac[q];
        for (int q = a.nfac - 1; q >= 1; --q) {
            shift_lo -= a.fac[q];
            const long kq = tmp & ((1L << a.fac[q]) - 1);
            tmp >>= a.fac[q];
            acc += kq << shift_lo;
        }
        T.pos_rest = acc + k10;
    } else {   // G whole items
        T.in = a.in + (blk << a.logG) * a.in_bstride;
        T.out = a.out + (blk << a.logG) * a.out_bstride;
    }
    return T;
}

// Starts the copy of a tile into shared memory: entry e of column g holds row
// bitrev(e) (after z skipped stages, row bitrev(e >> z)), zero beyond in_len.
__device__ __forceinline__ void fetch_tile(const PassArgs &a, const Tile &T, fe *S)
{
    const int mg = 1 << (a.lm + a.logG), G = 1 << a.logG;
    for (int idx = threadIdx.x; idx < mg; idx += NTT_THREADS) {
        int g, r0, e0;
        if (a.kind == 2 && a.z == 0) {   // lanes along an item
            r0 = idx & ((1 << a.lm) - 1);
            g = idx >> a.lm;
            e0 = bitrev(r0, a.lm);
        } else {
            g = idx & (G - 1);
            const int x = idx >> a.logG;
            if (a.z) {   // entries in order, each from the row its stages would have copied
                e0 = x;
                r0 = bitrev(x >> a.z, a.lm - a.z);
            } else {     // rows in order: 4 rows of a column per warp, 64 contiguous bytes
                r0 = x;
                e0 = bitrev(x, a.lm);
            }
        }
        long gi;
        const fe *src = T.in;
        if (a.kind == 0) {
            gi = T.col_base + g + (long)r0 * T.C;
        } else if (a.kind == 1) {
            gi = T.row_base + (((long)g * T.rowW) << a.lm) + r0;
        } else {
            src += g * a.in_bstride;
            gi = r0;
        }
        const unsigned dst = (unsigned)__cvta_generic_to_shared(S + (e0 << a.logG) + g);
        const unsigned bytes = gi < a.in_len ? 16 : 0;   // none: the entry is filled with zeros
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src + (bytes ? gi : 0)), "r"(bytes)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// the column pass's scale of output k of column g: w_A^(c k)
__device__ __forceinline__ fe out_twiddle(const PassArgs &a, const Tile &T, int g, int k)
{
    const long c = (T.col_base & ((1L << a.logA) - 1)) + g;
    const uint64_t e = ((uint64_t)c * (uint64_t)k) << (a.logn - a.logA);   // c k < A, so e < n
    return a.tw_full ? ld_tab(a.tw_full + (e >> a.tw_shift)) : tw_pow(a.tw_lo, a.tw_hi, e);
}
// output k of column (item) g, y at most 2^61 + 6 per component, w its scale
__device__ __forceinline__ void store_out(const PassArgs &a, const Tile &T, int g, int k, fe y, fe w)
{
    if (a.kind == 0) {
        T.out[T.col_base + g + (long)k * T.C] = y * w;
        return;
    }
    y = canon(y);
    if (a.rot) y = vg::fe_mul_pow2(y, a.rot);
    if (a.kind == 1) T.out[T.pos_rest + g + ((long)k << (a.logn - a.lm))] = y;
    else T.out[g * a.out_bstride + k] = y;
}

// One step of R radix-2 stages (s .. s + R - 1): entries i0 + (k << s), k < 2^R,
// of each group of 2^(s + R) at position pos < 2^s are multiplied by
// u^rev(k), u = w_m^(pos 2^(lm - R - s)), and replaced by their DFT.
template <int R>
__device__ __forceinline__ void ntt_step(const PassArgs &a, const Tile &T, int s, fe *S, const fe *W)
{
    constexpr int N = 1 << R;
    const int G = 1 << a.logG, mg = 1 << (a.lm + a.logG);
    const bool first = s == a.z, to_global = s + R == a.lm && a.kind != 2;
    for (int b = threadIdx.x; b < (mg >> R); b += NTT_THREADS) {
        const int g = b & (G - 1), q = b >> a.logG;
        const int pos = q & ((1 << s) - 1), i0 = ((q >> s) << (s + R)) + pos;
        fe *p = S + (i0 << a.logG) + g;
        const int st = 1 << (s + a.logG);
        fe x[N], w[N];
#pragma unroll
        for (int k = 0; k < N; ++k) x[k] = p[k * st];
        if (to_global && a.kind == 0) {   // in flight during the products
#pragma unroll
            for (int k = 0; k < N; ++k) w[k] = out_twiddle(a, T, g, i0 + (((k * a.c8) & (N - 1)) << s));
        }
        if (pos) {
            const int u = pos << (a.lm - R - s);
            if (R == 3) {
                constexpr int rev[8] = {0, 4, 2, 6, 1, 5, 3, 7};
#pragma unroll
                for (int k = 1; k < N; ++k) x[k] = x[k] * W[u * rev[k & 7]];
            } else if (R == 2) {
                x[1] = x[1] * W[2 * u];
                x[2] = x[2] * W[u];
                x[3] = x[3] * W[3 * u];
            } else {
                x[1] = x[1] * W[u];
            }
        } else if (!first) {   // products leave canonical values, as the first step's inputs are
#pragma unroll
            for (int k = 1; k < N; ++k) x[k] = canon(x[k]);
        }
        dft_regs(x);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const int j = (k * a.c8) & (N - 1);
            if (to_global) store_out(a, T, g, i0 + (j << s), x[k], w[k]);
            else p[j * st] = x[k];
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(NTT_THREADS, NTT_CTAS) k_ntt_pass(const __grid_constant__ PassArgs a)
{
    extern __shared__ fe smem[];
    const int m = 1 << a.lm, G = 1 << a.logG, mg = m << a.logG;
    fe *W = smem + 2 * mg;   // w_m^e, e < m; before it two tiles [m][G]
    Tile T = tile_at(a, blockIdx.x);
    fetch_tile(a, T, smem);
    for (int e = threadIdx.x; e < m; e += NTT_THREADS) {
        const uint64_t x = (uint64_t)e << (a.logn - a.lm);
        W[e] = a.tw_full ? ld_tab(a.tw_full + (x >> a.tw_shift)) : tw_pow(a.tw_lo, a.tw_hi, x);
    }
    int cur = 0;
    for (long tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x, cur ^= 1) {
        fe *S = smem + cur * mg;
        Tile next = T;
        if (tile + gridDim.x < a.ntiles) {
            next = tile_at(a, tile + gridDim.x);
            fetch_tile(a, next, smem + (cur ^ 1) * mg);   // every read of that half is behind the last step's barrier
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        for (int s = a.z; s < a.lm;) {
            const int left = a.lm - s;
            if (left == 1) {
                ntt_step<1>(a, T, s, S, W);
                s += 1;
            } else if (left == 2 || left == 4) {
                ntt_step<2>(a, T, s, S, W);
                s += 2;
            } else {
                ntt_step<3>(a, T, s, S, W);
                s += 3;
            }
        }
        if (a.kind == 2 || a.z == a.lm) {
            // whole items, lanes along an item; or a column pass with one
            // nonzero row, every output of a column being its entry
            for (int idx = threadIdx.x; idx < mg; idx += NTT_THREADS) {
                const int k = a.kind == 2 ? idx & (m - 1) : idx >> a.logG, g = a.kind == 2 ? idx >> a.lm : idx & (G - 1);
                store_out(a, T, g, k, S[(k << a.logG) + g], a.kind == 0 ? out_twiddle(a, T, g, k) : vg::fe_zero());
            }
            __syncthreads();
        }
        T = next;
    }
}

// w^e for every e < n, from the two small tables
__global__ void k_tw_full(const fe *__restrict__ lo, const fe *__restrict__ hi, long n, fe *__restrict__ full)
{
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x)
        full[e] = tw_pow(lo, hi, (uint64_t)e);
}

__global__ void k_tw_build(fe w, fe w4096, fe *lo, fe *hi, int nhi)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 4096) lo[i] = vg::fe_pow(w, (uint64_t)i);
    if (i < nhi) hi[i] = vg::fe_pow(w4096, (uint64_t)i);
}

// n = 2^logn as ceil(logn / max_lm) factors of nearly equal size (the
// radix: VG_TUNE_NTT_MAX_LOG, at most MAX_LM)
void plan_factors(int logn, int max_lm, std::vector<int> &f)
{
    f.clear();
    if (logn <= max_lm) {
        f.push_back(logn);
        return;
    }
    int P = (logn + max_lm - 1) / max_lm;
    int base = logn / P, extra = logn % P;
    for (int q = 0; q < P; ++q) f.push_back(base + (q < extra ? 1 : 0));
}

// columns (or whole items) of a tile: two tiles of m * G elements in
// 2^tile_log (VG_TUNE_NTT_TILE_LOG, at most MAX_TILE_LOG), fewer when that
// leaves SMs without a tile (down to 4 columns, 64 contiguous bytes)
int pick_logG(int lm, long avail_log, int tile_log, long total)
{
    int lg = tile_log - 1 - lm;
    if (lg < 0) lg = 0;
    if (lg > avail_log) lg = (int)avail_log;
    while (lg > 2 && (total >> (lm + lg)) < 2 * 148) --lg;
    return lg;
}

// stages that only copy when `rows` rows of 2^lm are nonzero
int skipped(int lm, long rows)
{
    int z = lm;
    while (z > 0 && (1L << (lm - z)) < rows) --z;
    return z;
}

}  // namespace

int vg_twiddles(vg_ctx *c, fe root, int logn, const fe **lo, const fe **hi)
{
    for (auto &t : c->tw_cache)
        if (t.key_real == root.real && t.key_img == root.img && t.logn == logn) {
            *lo = t.lo;
            *hi = t.hi;
            return VG_OK;
        }
    TwEntry t;
    t.key_real = root.real;
    t.key_img = root.img;
    t.logn = logn;
    int nhi = logn > 12 ? (1 << (logn - 12)) : 1;
    VG_TRY(vg_alloc(c, (void **)&t.lo, 4096 * sizeof(fe)));
    VG_TRY(vg_alloc(c, (void **)&t.hi, nhi * sizeof(fe)));
    fe w4096 = vg::fe_pow(root, 4096);
    k_tw_build<<<grid_for(std::max(4096, nhi), 256), 256, 0, c->stream>>>(root, w4096, t.lo, t.hi, nhi);
    VG_LAUNCHED(c);
    if (c->tw_cache.size() >= 64) {
        vg_release(c, c->tw_cache.front().lo);
        vg_release(c, c->tw_cache.front().hi);
        if (c->tw_cache.front().full) vg_release(c, c->tw_cache.front().full);
        c->tw_cache.erase(c->tw_cache.begin());
    }
    c->tw_cache.push_back(t);
    *lo = t.lo;
    *hi = t.hi;
    return VG_OK;
}

// The full table w^e, e < 2^logn, of a cached root (built on first use), or
// null when n is above 2^TW_FULL_MAX_LOG or the context's full tables would
// pass TW_FULL_BUDGET bytes: the column passes then form w^e from lo and hi.
constexpr int TW_FULL_MAX_LOG = 20;
constexpr size_t TW_FULL_BUDGET = 64u << 20;

static int twiddles_full(vg_ctx *c, fe root, int logn, const fe **full)
{
    *full = nullptr;
    if (logn > TW_FULL_MAX_LOG) return VG_OK;
    const fe *lo, *hi;
    VG_TRY(vg_twiddles(c, root, logn, &lo, &hi));
    size_t used = 0;
    TwEntry *mine = nullptr;
    for (auto &t : c->tw_cache) {
        if (t.full) used += ((size_t)1 << t.logn) * sizeof(fe);
        if (t.key_real == root.real && t.key_img == root.img && t.logn == logn) mine = &t;
    }
    if (!mine) return VG_OK;
    if (!mine->full) {
        const size_t bytes = ((size_t)1 << logn) * sizeof(fe);
        if (used + bytes > TW_FULL_BUDGET) return VG_OK;
        // never allocate inside a stream capture (the table would belong to the graph)
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        VG_CHECK_CUDA(cudaStreamIsCapturing(c->stream, &cs));
        if (cs != cudaStreamCaptureStatusNone) return VG_OK;
        VG_TRY(vg_alloc(c, (void **)&mine->full, bytes));
        k_tw_full<<<std::min<unsigned>(grid_for(1L << logn, 256), 148u * 8u), 256, 0, c->stream>>>(mine->lo, mine->hi,
                                                                                                   1L << logn, mine->full);
        VG_LAUNCHED(c);
    }
    *full = mine->full;
    return VG_OK;
}

static bool tw_cached(const vg_ctx *c, fe root, int logn)
{
    for (const auto &t : c->tw_cache)
        if (t.key_real == root.real && t.key_img == root.img && t.logn == logn) return true;
    return false;
}

// The full table of root^(2^f) (order 2^(logn - f)), or null, and root's own
// small tables again: an entry added to a full cache drops the oldest one, so
// both must be there after the last addition (never inside a stream capture).
static int block_table(vg_ctx *c, fe root, int logn, int f, const fe **lo, const fe **hi, const fe **full)
{
    *full = nullptr;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    VG_CHECK_CUDA(cudaStreamIsCapturing(c->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone || logn - f > TW_FULL_MAX_LOG) return VG_OK;
    fe w = root;
    for (int k = 0; k < f; ++k) w = w * w;
    VG_TRY(twiddles_full(c, w, logn - f, full));
    VG_TRY(vg_twiddles(c, root, logn, lo, hi));
    if (!tw_cached(c, w, logn - f)) *full = nullptr;
    return VG_OK;
}

// Largest dynamic shared memory of a pass: two tiles of m * G elements, together
// at most 2^MAX_TILE_LOG (pick_logG), plus m <= 1024 twiddles.  The kernel attribute is
// process-wide per device, so it is raised once to this bound: setting it per
// launch to the launch's own size races with other threads' launches of other
// sizes.
constexpr size_t NTT_MAX_SMEM = ((1 << MAX_TILE_LOG) + (1 << MAX_LM)) * sizeof(fe);

static int ntt_smem_attribute(int dev)
{
    static std::mutex mu;
    static std::vector<bool> done;
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= (int)done.size()) done.resize(dev + 1, false);
    if (!done[dev]) {
        VG_CHECK_CUDA(cudaFuncSetAttribute(k_ntt_pass, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NTT_MAX_SMEM));
        done[dev] = true;
    }
    return VG_OK;
}

static int launch_pass(vg_ctx *c, PassArgs &a, long nblocks, int batch)
{
    const int m = 1 << a.lm, G = 1 << a.logG;
    const size_t sm = (2 * (size_t)m * G + m) * sizeof(fe);
    if (sm > NTT_MAX_SMEM) return vg_fail(VG_ERR_ARG, "ntt pass: %zu bytes of shared memory", sm);
    if (sm > 48 * 1024) VG_TRY(ntt_smem_attribute(c->device));
    a.nblocks = nblocks;
    a.ntiles = nblocks * batch;
    // what is resident at once: NTT_CTAS per SM by registers, fewer by shared memory
    const long per_sm = std::max(1L, std::min((long)NTT_CTAS, (long)(227 * 1024 / (sm + 1024))));
    {
        ProfScope ps(c, KF_NTT, 2.0 * 16.0 * (double)batch * (double)(1L << a.logn));
        k_ntt_pass<<<(unsigned)std::min(a.ntiles, 148 * per_sm), NTT_THREADS, sm, c->stream>>>(a);
    }
    VG_LAUNCHED(c);
    return VG_OK;
}

extern "C" int vg_ntt(vg_ctx *c, const vg_fe *in_, long in_len, long in_bstride, vg_fe *out_, int logn,
                      long out_bstride, int batch, vg_fe root_, int scale_inv_n)
{
    if (!c || !in_ || !out_ || logn < 0 || logn > 30 || batch < 1 || in_len < 0 || in_len > (1L << logn))
        return vg_fail(VG_ERR_ARG, "vg_ntt: bad argument (logn=%d in_len=%ld batch=%d)", logn, in_len, batch);
    if (batch > 65535) return vg_fail(VG_ERR_ARG, "vg_ntt: batch %d > 65535", batch);
    const fe *in = (const fe *)in_;
    fe *out = (fe *)out_;
    fe root;
    root.real = root_.real;
    root.img = root_.img;
    const long n = 1L << logn;
    const fe *lo, *hi, *full;
    VG_TRY(vg_twiddles(c, root, logn, &lo, &hi));
    VG_TRY(twiddles_full(c, root, logn, &full));
    // n^-1 = 2^-logn = 2^(61 - logn)
    const int rot = scale_inv_n && logn ? 61 - logn : 0;
    // which primitive 8th root (2^30 (1 + i))^c the transform's is (odd c), or
    // which 4th root i^c when n = 4
    int c8 = 1;
    if (logn >= 2) {
        fe w = root;
        for (int k = logn; k > 3; --k) w = w * w;
        if (logn == 2) {
            c8 = w.img == 1 ? 1 : 3;
        } else {
            const bool re = w.real == 1ull << 30, im = w.img == 1ull << 30;
            c8 = im ? (re ? 1 : 3) : (re ? 7 : 5);
        }
    }

    std::vector<int> f;
    const int max_lm = std::min(MAX_LM, (int)vg_tune_value(c->device, VG_TUNE_NTT_MAX_LOG));
    const int tile_log = std::min(MAX_TILE_LOG, (int)vg_tune_value(c->device, VG_TUNE_NTT_TILE_LOG));
    plan_factors(logn, max_lm, f);
    const int P = (int)f.size();

    // passes after the first of a transform too large for a full table: the
    // blocks' own root w_A = w_n^F_1 is of order n / F_1, its full table smaller
    const fe *fullA = nullptr;
    if (!full && P > 1) VG_TRY(block_table(c, root, logn, f[0], &lo, &hi, &fullA));

    if (P == 1) {
        PassArgs a{};
        a.in = in; a.out = out; a.in_len = in_len; a.in_bstride = in_bstride; a.out_bstride = out_bstride;
        a.logn = logn; a.lm = logn; a.kind = 2; a.tw_lo = lo; a.tw_hi = hi; a.tw_full = full; a.rot = rot; a.c8 = c8;
        a.z = skipped(logn, in_len);
        // G whole items per CTA, G must divide batch
        int lg = pick_logG(logn, 30, tile_log, 1L << 62);
        while (lg > 0 && ((batch % (1 << lg)) != 0 || (batch >> lg) < 2 * 148)) --lg;
        a.logG = lg;
        VG_TRY(launch_pass(c, a, batch >> lg, 1));
        return VG_OK;
    }

    // intermediate buffer: passes 1..P-1 write tmp in place; the last pass writes out
    fe *tmp = out;
    bool in_place_ok = (in == out) ? (in_len == n && in_bstride == out_bstride) : false;
    const bool overlap = (in != out) && !((const char *)in + (size_t)batch * in_bstride * sizeof(fe) <= (const char *)out ||
                                          (const char *)out + (size_t)batch * out_bstride * sizeof(fe) <= (const char *)in);
    if (overlap && !in_place_ok) return vg_fail(VG_ERR_ARG, "vg_ntt: in and out overlap");
    // the row pass reads tmp and writes out in a permuted order, so tmp != out
    void *s;
    VG_TRY(vg_scratch(c, (size_t)batch * n * sizeof(fe), &s));
    tmp = (fe *)s;

    int logA = logn;
    for (int q = 0; q < P - 1; ++q) {
        PassArgs a{};
        a.in = q == 0 ? in : tmp;
        a.out = tmp;
        a.in_len = q == 0 ? in_len : n;
        a.in_bstride = q == 0 ? in_bstride : n;
        a.out_bstride = n;
        a.logn = logn; a.lm = f[q]; a.kind = 0; a.logA = logA;
        a.tw_lo = lo; a.tw_hi = hi; a.c8 = c8;
        a.tw_full = q && fullA ? fullA : full;
        a.tw_shift = q && fullA ? f[0] : 0;
        long logC = logA - f[q];
        a.z = q == 0 ? skipped(f[q], (in_len + (1L << logC) - 1) >> logC) : 0;
        a.logG = pick_logG(f[q], logC, tile_log, n * batch);
        long nblocks = (n >> logA) * ((1L << logC) >> a.logG);
        VG_TRY(launch_pass(c, a, nblocks, batch));
        logA -= f[q];
    }
    {
        PassArgs a{};
        a.in = tmp; a.out = out; a.in_len = n; a.in_bstride = n; a.out_bstride = out_bstride;
        a.logn = logn; a.lm = f[P - 1]; a.kind = 1;
        a.nfac = P - 1;
        for (int q = 0; q < P - 1; ++q) a.fac[q] = f[q];
        a.tw_lo = lo; a.tw_hi = hi; a.rot = rot; a.c8 = c8;
        a.tw_full = fullA ? fullA : full;
        a.tw_shift = fullA ? f[0] : 0;
        a.logG = pick_logG(f[P - 1], f[0], tile_log, n * batch);
        long T_all = n >> f[P - 1];
        long nblocks = T_all >> a.logG;
        VG_TRY(launch_pass(c, a, nblocks, batch));
    }
    return VG_OK;
}
