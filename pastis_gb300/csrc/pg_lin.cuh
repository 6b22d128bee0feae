// pg_lin.cuh -- the alignment DP and its traceback when the affine recurrence
// collapses to a linear one (sm_103a).
//
// With a first gap position that costs less than the further ones (go > ge,
// what PASTIS's parameters become when they are passed as it passes them),
// E(i, j) = max(E(i, j-1) + ge, H(i, j-1) + go) is always H(i, j-1) + go,
// strictly: E <= H and ge < go.  The same holds for F.  So
//     H(i, j) = max(H(i-1, j-1) + s, H(i-1, j) + go, H(i, j-1) + go [, 0])
// and every gap of the traceback was opened, whatever the tie policy says of
// gap ties.  What bounds the DP is the integer ALU pipe (two cycles a warp
// instruction), so the form below is built to need few ALU operations:
//
//  - two cells per 32-bit register (int16 halves: the low half R rows, the
//    high half the R rows below them one column behind), values scaled by 4;
//  - the decision rides in the two free bits: a term carries its tag (diagonal
//    3 on identical residues, 2 otherwise; of F and E the one the tie policy
//    prefers 1, the other 0), so the maximum picks the larger H and on a tie
//    the larger tag, and no comparison is needed to know which term won.  The
//    local form subtracts its tags (diagonal 1, F / E 2 and 3): at H = 0 the floor
//    of the maximum, 0 itself, then wins every tie, and tag 0 marks the cells
//    where a traceback ends;
//  - per row and two cells: one prmt (score), one add, two DPX add-max, one
//    logic op to clear the tag; the tags are gathered by multiply-adds on the
//    FMA pipe (the sum of the tagged against the sum of the cleared values).
// That is 5 ALU operations for 2 cells against 17 in the affine form.
//
// A direction word holds 2 bits per cell: the 2 x 8 rows of a lane's two
// virtual lanes at one wavefront step in one 32-bit word; eight steps of a
// lane fill a 32-byte sector, written as two 16-byte stores.
//
// Work units.  Regions are listed by class (lanes L x rows per lane R) and
// column count.  A region of up to 16 R rows takes 8 lanes, 32 R rows 16 lanes,
// 64 R rows a warp, so that a warp works 4, 2 or 1 regions of the same class
// and nearly the same column count together: a wavefront spends a step per
// virtual lane filling and another draining, and the fewer lanes a region has
// the shorter those ramps, at 8 rows per lane that spread a step's fixed cost
// (shuffle, residue, profile reads, store) over 16 cells.  Taller regions, and
// those whose scaled values could leave int16, run as stripes of 64 R rows, one
// warp each, pipelined: a stripe waits for the stripe above only 32 columns at
// a time (boundary row and progress word in HBM), and its lanes keep their
// values relative to a base that follows them, so no region is too large.
#pragma once
#include <cstdint>
#include <type_traits>

#include "pg_kernels.cuh"
#include "pg_lin.h"

namespace pg {

// ------------------------------------------------------------- host rule
// scores the tagged 16-bit form takes: gap scores as above; substitution
// scores that fit an int8 profile after scaling; a gap that costs less than the
// sentinel's -128 after scaling.  H moves by at most 31 + 31 from a neighbour,
// so a lane's values stay inside int16 and positive for the 32 columns between two
// base moves (LIN_MID +- (32 + 16) cells x 4 x 62 = 11904)
constexpr int LIN_SMAX = 31;
__host__ __forceinline__ bool lin_supported(int go, int ge, int smin, int smax)
{
    return go > ge && go < 0 && go >= -LIN_SMAX && smin >= -LIN_SMAX && smax <= LIN_SMAX;
}

// ------------------------------------------------------------- work list
// one region, or one stripe of a region that runs in stripes (its stripes are
// consecutive entries)
struct LinReg {
    uint64_t v, h;        // first row / column residue (offsets into the sides' residues)
    uint32_t key;         // X-drop: 2 * pair + seed; SW: pair
    uint32_t off;         // its direction words, in 32-byte units of the arena
    uint16_t m, n;
    uint16_t stripe, nstripe;
};
static_assert(sizeof(LinReg) == 32, "two 16-byte loads");

// classes: 0-3 stripes with R = 8..5; 4-7 a warp, R = 8..5; 8-11 16 lanes,
// R = 8..5; 12-17 8 lanes, R = 8, 7, 6, 5, 4, 2.  The list runs by class and in a
// class by column count, the long first.
constexpr int LIN_CLS = 18;
constexpr int LIN_LEV = 48;                        // column-count levels per class
constexpr int LIN_NB = LIN_CLS * LIN_LEV;
// Columns from which a region's walk has a warp of its own.  The walk kernel, us:
// 400k X-drop pairs 1068 / 861 / 839 / 1075 at 256 / 384 / 512 / 1024, 60k uneven
// ones 373 / 365 / 405 / 598; 100k Smith-Waterman pairs 643 / 376 / 530 at 512 / 768 /
// 1024, 8k uneven ones 512 / 527 / 530.
__host__ __device__ __forceinline__ constexpr int lin_wide(bool local) { return local ? 768 : 384; }

struct LinTotals {
    unsigned long long units;                      // arena need in 32-byte units
    unsigned long long cursor;                     // arena units handed out by k_lin_place
    unsigned long long work[LIN_CLS];              // DP instructions of each class, about
    uint32_t entries, jobs;
    uint32_t wide, wcursor;                        // regions of lin_wide columns; their list's cursor
    uint32_t next_job[LIN_CLS];                    // work counters of k_lin_dp
    uint32_t cls[2 * LIN_CLS];                     // per class: first list entry, entries
};
struct LinParams {
    KParams kp;
    uint64_t p0, p1;                               // pairs of this pass
    uint32_t *cnt;                                 // LIN_NB bucket sizes
    uint32_t *cur;                                 // LIN_NB bucket cursors
    LinTotals *tot;
    LinReg *list;
    int4 *dp;                                      // per entry: score; local: low / high halves that reach it, have
    uint32_t *prog;                                // per entry: columns of its boundary row written
    uint32_t *wlist;                               // list positions of the wide regions
    uint8_t *arena;
    int4 *walk;                                    // X-drop, per key: score, matches, diagonals, gap runs
    int smax;
    int e_first;                                   // H ties: E before F
};

__host__ __device__ __forceinline__ int lin_seg_lanes(int cls) { return cls < 8 ? 32 : cls < 12 ? 16 : 8; }
__host__ __device__ __forceinline__ int lin_seg_rows(int cls)
{
    return cls < 16 ? 8 - (cls & 3) : cls == 16 ? 4 : 2;
}
__host__ __device__ __forceinline__ int lin_seg_group(int cls) { return cls < 8 ? 1 : cls < 12 ? 2 : 4; }

__device__ __forceinline__ int lin_class(const LinParams &lp, bool local, int m, int n)
{
    // every scaled value of the region provably inside int16 (no base):
    // above smax per diagonal, below the all-gaps path plus the rows past m
    const int lo = local ? 0 : -lp.kp.go * (m + n + 20);
    const bool plain = 4 * lp.smax * min(m, n) <= 31000 && 4 * lo <= 30000;
    if (m > 512 || !plain) {
        const int stripes = (m + 511) >> 9;
        const int r = (m + 64 * stripes - 1) / (64 * stripes);
        return r <= 5 ? 3 : 8 - r;
    }
    if (m > 256) { const int r = (m + 63) >> 6; return 4 + 8 - r; }
    if (m > 128) { const int r = (m + 31) >> 5; return 8 + 8 - r; }
    const int r = (m + 15) >> 4;
    return r <= 2 ? 17 : r <= 4 ? 16 : 12 + 8 - r;
}
__device__ __forceinline__ int lin_bucket(int cls, int n)
{
    const int l = n < 256 ? n >> 3 : n < 1024 ? 32 + ((n - 256) >> 6) : n < 4096 ? 44 + ((n - 1024) >> 10) : 47;
    return cls * LIN_LEV + LIN_LEV - 1 - l;
}
// stripes of a region (1 for the classes that do not run in stripes)
__host__ __device__ __forceinline__ int lin_stripes(int cls, int m)
{
    return cls < 4 ? (m + 64 * lin_seg_rows(cls) - 1) / (64 * lin_seg_rows(cls)) : 1;
}
// 8-step tiles of one stripe, in 32-byte units; boundary row of one stripe
__host__ __device__ __forceinline__ uint32_t lin_tile_units(int lanes, int n)
{
    return (uint32_t)((n + 2 * lanes - 1 + 7) >> 3) * (uint32_t)lanes;
}
__host__ __device__ __forceinline__ uint32_t lin_row_units(int n) { return (uint32_t)((n + 1 + 7) >> 3); }
// 32-step chunks of one stripe
__host__ __device__ __forceinline__ uint32_t lin_chunks(int lanes, int n) { return (uint32_t)((n + 2 * lanes - 1 + 31) >> 5); }
// Arena of a region, planes of `ns` stripes each, in 32-byte units: direction
// words; in the local form the lanes' edge words (same layout), their rows'
// values at each chunk's start, the bases those are relative to (stripes) and the
// chunk of each half's maximum; last, the boundary rows between stripes.
struct LinPlanes {
    uint32_t tile, snap, base, ids;                  // units of one stripe
    __host__ __device__ __forceinline__ LinPlanes(bool local, int cls, int n)
    {
        const int l = lin_seg_lanes(cls);
        const uint32_t ch = local ? lin_chunks(l, n) : 0;
        tile = lin_tile_units(l, n);
        snap = ch * (uint32_t)l;
        base = cls < 4 ? ch * 4u : 0u;
        ids = local ? (uint32_t)l / 8u : 0u;
    }
    __host__ __device__ __forceinline__ uint32_t stripe(bool local) const
    {
        return tile * (local ? 2u : 1u) + snap + base + ids;
    }
};
__host__ __device__ __forceinline__ uint32_t lin_units(bool local, int cls, int m, int n)
{
    const uint32_t s = (uint32_t)lin_stripes(cls, m);
    return s * LinPlanes(local, cls, n).stripe(local) + (s - 1) * lin_row_units(n);
}

// the DP regions of pair p: X-drop up to two (one per seed), SW one
struct LinPair {
    uint64_t v[2], h[2];
    int m[2], n[2];
    bool dp[2];
    bool bad;              // a sequence index out of range
};
template <bool XDROP>
__device__ __forceinline__ LinPair lin_pair(const KParams &kp, uint64_t p)
{
    LinPair lp;
    lp.dp[0] = lp.dp[1] = false;
    lp.m[0] = lp.m[1] = lp.n[0] = lp.n[1] = 0;
    lp.v[0] = lp.v[1] = lp.h[0] = lp.h[1] = 0;
    const pg_pair pr = kp.pairs[p];
    const uint64_t r = (uint64_t)pr.row + kp.roff, c = (uint64_t)pr.col + kp.coff;
    lp.bad = r >= kp.nr || c >= kp.nc;
    if (lp.bad) return lp;
    const uint64_t r0 = kp.roffs[r], c0 = kp.coffs[c];
    if (XDROP) {
        const XdRec a = kp.xd[2 * p], b = kp.xd[2 * p + 1];
        lp.dp[0] = !(a.flags & (XF_NONE | XF_BADIDX)) && a.ev > a.bv && a.eh > a.bh;
        const bool same = !(a.flags & XF_NONE) && b.bv == a.bv && b.ev == a.ev && b.bh == a.bh && b.eh == a.eh;
        lp.dp[1] = !(b.flags & (XF_NONE | XF_SAME | XF_BADIDX)) && !same && b.ev > b.bv && b.eh > b.bh;
        lp.v[0] = r0 + a.bv; lp.h[0] = c0 + a.bh; lp.m[0] = a.ev - a.bv; lp.n[0] = a.eh - a.bh;
        lp.v[1] = r0 + b.bv; lp.h[1] = c0 + b.bh; lp.m[1] = b.ev - b.bv; lp.n[1] = b.eh - b.bh;
    } else {
        lp.v[0] = r0; lp.h[0] = c0;
        lp.m[0] = (int)(kp.roffs[r + 1] - r0);
        lp.n[0] = (int)(kp.coffs[c + 1] - c0);
        lp.dp[0] = lp.m[0] > 0 && lp.n[0] > 0;
    }
    return lp;
}

constexpr int LIN_PT = 256;                        // threads of the list kernels
constexpr int LIN_PP = 4;                          // pairs per thread and pass

// bucket sizes and arena need of the pass
template <bool XDROP>
__global__ void __launch_bounds__(LIN_PT) k_lin_hist(const LinParams lp)
{
    __shared__ uint32_t h[LIN_NB];
    __shared__ unsigned long long su, hw[LIN_CLS];
    for (int b = threadIdx.x; b < LIN_NB; b += LIN_PT) h[b] = 0;
    if (threadIdx.x < LIN_CLS) hw[threadIdx.x] = 0;
    if (threadIdx.x == 0) su = 0;
    __syncthreads();
    unsigned long long units = 0;
    uint32_t wide = 0;
    for (uint64_t p = lp.p0 + (uint64_t)blockIdx.x * LIN_PT + threadIdx.x; p < lp.p1;
         p += (uint64_t)gridDim.x * LIN_PT) {
        const LinPair r = lin_pair<XDROP>(lp.kp, p);
#pragma unroll
        for (int s = 0; s < (XDROP ? 2 : 1); ++s) {
            if (!r.dp[s]) continue;
            const int cls = lin_class(lp, !XDROP, r.m[s], r.n[s]);
            atomicAdd(&h[lin_bucket(cls, r.n[s])], (uint32_t)lin_stripes(cls, r.m[s]));
            units += lin_units(!XDROP, cls, r.m[s], r.n[s]);
            // a region's share of its warp's steps, about 20 + 8 R instructions each
            atomicAdd(&hw[cls], (unsigned long long)(lin_stripes(cls, r.m[s]) * (r.n[s] + 2 * lin_seg_lanes(cls)) *
                                                     (20 + 8 * lin_seg_rows(cls)) / lin_seg_group(cls)));
            wide += r.n[s] >= lin_wide(!XDROP) ? 1u : 0u;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) units += __shfl_xor_sync(FULL, units, o);
    wide = __reduce_add_sync(FULL, wide);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&su, units);
        if (wide) atomicAdd(&lp.tot->wide, wide);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < LIN_NB; b += LIN_PT)
        if (h[b]) atomicAdd(&lp.cnt[b], h[b]);
    if (threadIdx.x < LIN_CLS && hw[threadIdx.x]) atomicAdd(&lp.tot->work[threadIdx.x], hw[threadIdx.x]);
    if (threadIdx.x == 0 && su) atomicAdd(&lp.tot->units, su);
}

// bucket starts (exclusive prefix) and the classes' places in the list and in
// the job order; one block of 1024 threads
static __global__ void __launch_bounds__(1024) k_lin_scan(const LinParams lp)
{
    static_assert(LIN_NB <= 1024, "one bucket per thread");
    __shared__ uint32_t w[32], start[LIN_NB + 1];
    const int t = threadIdx.x, lane = t & 31;
    const uint32_t c = t < LIN_NB ? lp.cnt[t] : 0;
    uint32_t x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) w[t >> 5] = x;
    __syncthreads();
    if (t < 32) {
        uint32_t y = w[t];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t z = __shfl_up_sync(FULL, y, o);
            if (lane >= o) y += z;
        }
        w[t] = y;
    }
    __syncthreads();
    const uint32_t inc = x + (t >= 32 ? w[(t >> 5) - 1] : 0);
    if (t < LIN_NB) { start[t] = inc - c; lp.cur[t] = inc - c; }
    if (t == LIN_NB - 1) start[LIN_NB] = inc;
    __syncthreads();
    if (t < LIN_CLS) {
        const uint32_t b = start[t * LIN_LEV], n = start[(t + 1) * LIN_LEV] - b, g = (uint32_t)lin_seg_group(t);
        lp.tot->cls[t] = b;
        lp.tot->cls[LIN_CLS + t] = n;
        atomicAdd(&lp.tot->jobs, (n + g - 1) / g);
    }
    if (t == 0) lp.tot->entries = start[LIN_NB];
}

// the list, in bucket order; arena units by one atomic per block and pass.  A
// pair without a region in SW gets its (empty) result here.
template <bool XDROP>
__global__ void __launch_bounds__(LIN_PT) k_lin_place(const LinParams lp)
{
    __shared__ uint32_t h[LIN_NB];
    __shared__ uint32_t su;
    __shared__ unsigned long long ubase;
    const uint64_t step = (uint64_t)LIN_PT * LIN_PP;
    unsigned long long cells = 0;
    for (uint64_t c0 = lp.p0 + blockIdx.x * step; c0 < lp.p1; c0 += gridDim.x * step) {
        for (int b = threadIdx.x; b < LIN_NB; b += LIN_PT) h[b] = 0;
        if (threadIdx.x == 0) su = 0;
        __syncthreads();
        constexpr int NS = XDROP ? 2 : 1;
        uint32_t rank[LIN_PP * NS], off[LIN_PP * NS];
#pragma unroll
        for (int q = 0; q < LIN_PP; ++q) {
            const uint64_t p = c0 + (uint64_t)q * LIN_PT + threadIdx.x;
            LinPair r;
            r.dp[0] = r.dp[1] = false;
            if (p < lp.p1) r = lin_pair<XDROP>(lp.kp, p);
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                rank[q * NS + s] = off[q * NS + s] = 0;
                if (!r.dp[s]) continue;
                const int cls = lin_class(lp, !XDROP, r.m[s], r.n[s]);
                rank[q * NS + s] = atomicAdd(&h[lin_bucket(cls, r.n[s])], (uint32_t)lin_stripes(cls, r.m[s]));
                off[q * NS + s] = atomicAdd(&su, lin_units(!XDROP, cls, r.m[s], r.n[s]));
                cells += (unsigned long long)r.m[s] * (unsigned long long)r.n[s];
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) ubase = su ? atomicAdd(&lp.tot->cursor, (unsigned long long)su) : 0;
        for (int b = threadIdx.x; b < LIN_NB; b += LIN_PT) {
            const uint32_t k = h[b];
            if (k) h[b] = atomicAdd(&lp.cur[b], k);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < LIN_PP; ++q) {
            const uint64_t p = c0 + (uint64_t)q * LIN_PT + threadIdx.x;
            if (p >= lp.p1) continue;
            const LinPair r = lin_pair<XDROP>(lp.kp, p);
            if (!XDROP && !r.dp[0]) {
                pg_result o = empty_result();
                if (r.bad) atomicOr(lp.kp.status, ST_BAD_INDEX);
                else apply_filter(o, r.m[0], r.n[0], lp.kp.cov_thr, lp.kp.ani_thr);
                lp.kp.out[p] = o;
            }
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                if (!r.dp[s]) continue;
                const int cls = lin_class(lp, !XDROP, r.m[s], r.n[s]);
                const int ns = lin_stripes(cls, r.m[s]);
                uint32_t pos = h[lin_bucket(cls, r.n[s])] + rank[q * NS + s];
                LinReg e;
                e.v = r.v[s]; e.h = r.h[s];
                e.key = XDROP ? (uint32_t)(2 * p + s) : (uint32_t)p;
                e.off = (uint32_t)(ubase + off[q * NS + s]);
                e.m = (uint16_t)r.m[s]; e.n = (uint16_t)r.n[s];
                e.nstripe = (uint16_t)ns;
                if (r.n[s] >= lin_wide(!XDROP)) lp.wlist[atomicAdd(&lp.tot->wcursor, 1u)] = pos;
                for (int k = 0; k < ns; ++k, ++pos) {
                    e.stripe = (uint16_t)k;
                    const uint4 *src = reinterpret_cast<const uint4 *>(&e);
                    uint4 *dst = reinterpret_cast<uint4 *>(lp.list + pos);
                    dst[0] = src[0];
                    dst[1] = src[1];
                    lp.prog[pos] = 0;
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cells += __shfl_xor_sync(FULL, cells, o);
    if ((threadIdx.x & 31) == 0 && cells) atomicAdd(lp.kp.exec_cells + 1, cells);
}

// ------------------------------------------------------------------ the DP
constexpr int LIN_ROWB = 36;                       // byte stride of a score-table row: 9 words spread the banks
constexpr int LIN_NC = NCODES + 1;                 // the residues and the sentinel past either end
constexpr int LIN_PROF = 2 * LIN_NC * 32 * 8;      // bytes per warp
constexpr int LIN_DYN = WARPS * LIN_PROF;
constexpr uint32_t LIN_CLR = 0xFFFCFFFCu;          // clears both halves' tags
constexpr int LIN_NEG = -32000;
constexpr int LIN_MID = 16384;

// tagged score table: row a, byte b = 4 * s(a, b) + (a == b ? 3 : 2), in the local
// form 4 * s(a, b) - 1; the sentinel row and the sentinel column -128
__device__ __forceinline__ void lin_table(int8_t *t, const int8_t *sm, bool local)
{
    for (int k = threadIdx.x; k < LIN_NC * LIN_ROWB; k += blockDim.x) {
        const int a = k / LIN_ROWB, b = k - a * LIN_ROWB;
        t[k] = a < PG_NRES && b < PG_NRES ? (int8_t)(4 * (int)sm[a * PG_NRES + b] + (local ? -1 : a == b ? 3 : 2)) : (int8_t)-128;
    }
}

// This lane's score profile for rows row0 .. row0 + 2R - 1 of V (0-based; rows
// past m: sentinel): for each residue code, NG words per half, byte r of word g
// = the tagged score of row 4 g + r.  Four rows' table words (four codes each)
// are transposed with 8 byte permutes, 28 prmt per code group in place of a
// table read and four logic ops per entry.
template <int R>
__device__ __forceinline__ void lin_profile(const uint32_t *tab, const uint8_t *V, int row0, int m,
                                            bool on, uint32_t *prof)
{
    constexpr int NG = (R + 3) / 4;
    const int lane = threadIdx.x & 31;
    uint32_t a[2 * NG * 4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < NG * 4; ++r) {
            const int i = row0 + h * R + r;
            a[h * NG * 4 + r] = (uint32_t)(r < R && on && i < m ? (int)__ldg(V + i) : PG_NRES) * (LIN_ROWB / 4);
        }
    for (int w = 0; w < (LIN_NC + 3) / 4; ++w) {
        uint32_t y[4][2 * NG];
#pragma unroll
        for (int g = 0; g < 2 * NG; ++g) {
            const uint32_t x0 = tab[a[4 * g] + w], x1 = tab[a[4 * g + 1] + w];
            const uint32_t x2 = tab[a[4 * g + 2] + w], x3 = tab[a[4 * g + 3] + w];
            const uint32_t t0 = prmt(x0, x1, 0x5140u), t1 = prmt(x2, x3, 0x5140u);
            const uint32_t t2 = prmt(x0, x1, 0x7362u), t3 = prmt(x2, x3, 0x7362u);
            y[0][g] = prmt(t0, t1, 0x5410u);
            y[1][g] = prmt(t0, t1, 0x7632u);
            y[2][g] = prmt(t2, t3, 0x5410u);
            y[3][g] = prmt(t2, t3, 0x7632u);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = 4 * w + q;
            if (c >= LIN_NC) break;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t *d = prof + ((h * LIN_NC + c) * 32 + lane) * NG;
                if (NG == 2) *reinterpret_cast<uint2 *>(d) = make_uint2(y[q][h * NG], y[q][h * NG + 1]);
                else *d = y[q][h];
            }
        }
    }
}

// the column residues of a lane, four at a time from aligned words; bytes past
// the sequence read as the sentinel.  A word is loaded a group ahead and masked
// only when it is used, so that nothing waits on the load in between.
struct LinCols {
    const uint32_t *w;      // the word last loaded
    int y, n;               // its first byte, as a column index
    uint32_t cur, nxt;
    uint32_t sh;
    __device__ __forceinline__ uint32_t load() const
    {
        uint32_t v = 0x19191919u;
        if (n > 0 && (unsigned)(y + 3) < (unsigned)(n + 3)) v = __ldg(w);
        return v;
    }
    __device__ __forceinline__ uint32_t masked(uint32_t v) const
    {
        if (y + 4 > n && y < n) {
            const uint32_t keep = (1u << (8 * (n - y))) - 1u;      // 1..3 bytes
            v = (v & keep) | (0x19191919u & ~keep);
        }
        return v;
    }
    // x0: column index (0-based) of the first residue wanted
    __device__ __forceinline__ void init(const uint8_t *H, int n_, int x0)
    {
        static_assert(NCODES == 25, "0x19 is the sentinel's code");
        n = n_;
        const uint8_t *p = H + x0;
        const int a = (int)(reinterpret_cast<uintptr_t>(p) & 3u);
        sh = 8u * (uint32_t)a;
        w = reinterpret_cast<const uint32_t *>(p - a);
        y = x0 - a;
        cur = masked(load());
        ++w; y += 4;
        nxt = load();
    }
    __device__ __forceinline__ uint32_t next()
    {
        const uint32_t v = masked(nxt);
        const uint32_t r = __funnelshift_r(cur, v, sh);
        cur = v;
        ++w; y += 4;
        nxt = load();
        return r;
    }
};

// maximum of a column's rows, per half, with a running one
template <int R>
__device__ __forceinline__ uint32_t lin_max(uint32_t s, const uint32_t (&H)[R])
{
#pragma unroll
    for (int r = 0; r + 1 < R; r += 2) s = __vimax3_s16x2(s, H[r], H[r + 1]);
    return R & 1 ? v16max(s, H[R - 1]) : s;
}

// where a lane of the local form leaves what lin_locate needs
struct LinTrack {
    uint8_t *snap;          // [chunk][lane] 32 bytes: its rows at the chunk's start
    int *base;              // [chunk][lane] their base (stripes)
    uint32_t *ids;          // [lane] chunk of the low and the high half's maximum
};
template <int R>
__device__ __forceinline__ void lin_snap(uint8_t *dst, const uint32_t (&H)[R])
{
    uint32_t v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = r < R ? H[r < R ? r : 0] : 0u;
    reinterpret_cast<uint4 *>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
    if (R > 4) reinterpret_cast<uint4 *>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
}
// the halves whose maximum rose during chunk c
__device__ __forceinline__ void lin_chunk(uint32_t sbs, uint32_t &seen, uint32_t &cid, int c)
{
    const uint32_t x = sbs ^ seen;
    if (x & 0xffffu) cid = (cid & 0xffff0000u) | (uint32_t)c;
    if (x >> 16) cid = (cid & 0xffffu) | ((uint32_t)c << 16);
    seen = sbs;
}

struct LinConst {
    uint32_t goL, goU;      // packed 4 go + tag of E / F
    uint32_t four, one;     // from memory: the multiply-adds below stay on the FMA pipe
    int go4;
};

// one column of the lane's 2R rows; returns the direction word
template <int R, bool LOCAL, bool BASE>
__device__ __forceinline__ uint32_t lin_rows(uint32_t (&H)[R], uint32_t dgH, uint32_t in_h,
                                             const uint32_t *pl, const uint32_t *ph,
                                             const LinConst &c, uint32_t floor2)
{
    constexpr int NG = (R + 3) / 4;
    uint32_t lo[NG], hi[NG];
    if (NG == 2) {
        const uint2 a = *reinterpret_cast<const uint2 *>(pl), b = *reinterpret_cast<const uint2 *>(ph);
        lo[0] = a.x; lo[NG - 1] = a.y; hi[0] = b.x; hi[NG - 1] = b.y;
    } else {
        lo[0] = *pl; hi[0] = *ph;
    }
    uint32_t dl[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t s2 = prmt(lo[r >> 2], hi[r >> 2], sx_sel(r & 3));
        uint32_t dg = v16add(r ? H[r ? r - 1 : 0] : dgH, s2);
        if (LOCAL && BASE) dg = v16max(dg, floor2);
        dl[r] = __viaddmax_s16x2(H[r], c.goL, dg);
    }
    uint32_t up = in_h, wa = 0, wb = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t t = LOCAL && !BASE ? __viaddmax_s16x2_relu(up, c.goU, dl[r])
                                          : __viaddmax_s16x2(up, c.goU, dl[r]);
        // local: round up to the multiple of 4 (both halves of t are positive: no carry)
        if (LOCAL) up = (t * c.one + 0x00030003u) & LIN_CLR;
        else up = t & LIN_CLR;
        H[r] = up;
        wa = wa * c.four + t;
        wb = wb * c.four + up;
    }
    return LOCAL ? wb - wa : wa - wb;
}

// Regions of the L-lane classes: each L lanes of the warp pass their own region
// (m = 0: none).  The result is that of the lane's region.
template <bool LOCAL, int L, int R>
__device__ __forceinline__ int4 lin_sub(const uint32_t *tab, uint32_t *prof, const LinConst &c,
                                        const uint8_t *V, int m, const uint8_t *Hs, int n, uint8_t *dir,
                                        const LinTrack &tr)
{
    constexpr int NG = (R + 3) / 4;
    const int lane = threadIdx.x & 31;
    const int sl = lane & (L - 1);
    const bool has = m > 0 && n > 0;
    const int v_last = has ? (m - 1) / R : -1;       // <= 2L - 1
    const int t_last = v_last >> 1;
    const bool on = sl <= t_last;
    const int hi_on = 2 * sl + 1 <= v_last ? 1 : 0;
    const int i_base = 2 * sl * R;
    const int own = has ? n + v_last : 0;            // this region's steps
    const unsigned lim = on ? (unsigned)(n + hi_on) : 0u;
    __syncwarp();
    lin_profile<R>(tab, V, i_base, m, on, prof);
    __syncwarp();
    // column 0 of the low half's rows, column -1 (sentinels) of the high half's
    uint32_t H[R];
#pragma unroll
    for (int r = 0; r < R; ++r) H[r] = pk16(LOCAL ? 0 : c.go4 * (i_base + r + 1), LIN_NEG);
    const int up0 = LOCAL ? 0 : c.go4 * i_base, lo0 = LOCAL ? 0 : c.go4 * (i_base + R);
    const int hi0 = LOCAL ? 0 : c.go4 * (i_base + 2 * R);
    uint32_t in_h = pk16(up0, lo0), out_h = pk16(lo0, hi0);
    uint32_t bord = LOCAL ? 0u : (uint32_t)c.go4 << 16;       // H(0, j) of the first lane, in the high half
    const uint32_t bstep = LOCAL ? 0u : (uint32_t)c.go4 << 16;
    LinCols cols;
    cols.init(Hs, has ? n : 0, -2 * sl);
    const char *lbase = reinterpret_cast<const char *>(prof + lane * NG);
    const char *pa = lbase + PG_NRES * (128 * NG);   // the sentinel's profile: column 0 of the high half
    uint32_t sbs = 0, seen = 0, cid = 0;
    // steps of the longest region; the steps where every lane that holds rows is
    // inside its columns need no test per lane (the others compute in vain there):
    // with the residues masked at their use, 400k X-drop pairs' DP 5.83 -> 4.82 ms
    int nsteps = own, ks = on ? 2 * sl : 0, ke = has ? n : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        nsteps = max(nsteps, __shfl_xor_sync(FULL, nsteps, o));
        ks = max(ks, __shfl_xor_sync(FULL, ks, o));
        ke = min(ke, __shfl_xor_sync(FULL, ke, o));
    }
    uint8_t *dst = dir + sl * 32;
    const size_t plane = (size_t)lin_tile_units(L, n) * 32u;
    // one step's inputs: the row above both halves; returns the diagonal's
    auto step = [&]() {
        const uint32_t rh = __shfl_up_sync(FULL, out_h, 1, L);
        const uint32_t dgH = in_h;
        const uint32_t th = sl == 0 ? bord : rh;
        if (!LOCAL) bord += bstep;
        in_h = prmt(th, out_h, 0x5432u);
        return dgH;
    };
    auto rows_of = [&](const uint32_t dgH, const uint32_t code) {
        const char *ph = pa + LIN_NC * (128 * NG);
        pa = lbase + code * (128 * NG);
        const uint32_t w = lin_rows<R, LOCAL, false>(H, dgH, in_h, reinterpret_cast<const uint32_t *>(pa),
                                                     reinterpret_cast<const uint32_t *>(ph), c, 0u);
        out_h = H[R - 1];
        if (LOCAL) sbs = lin_max<R>(sbs, H);
        return w;
    };
    // four steps (a lambda, for its two uses: the steps where every lane that holds
    // rows is inside its columns, and the ramps, where each lane is tested)
    auto group = [&](const int k0, const uint32_t res4, auto test) {
        uint32_t w[4], e[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t dgH = step();
            w[s] = 0;
            if (!decltype(test)::value || (unsigned)(k0 + s - 2 * sl) < lim)
                w[s] = rows_of(dgH, (res4 >> (8 * s)) & 0xffu);
            e[s] = out_h;
        }
        if (on && k0 < own) {
            uint8_t *d = dst + (size_t)(k0 >> 3) * (L * 32) + (k0 & 4) * 4;
            *reinterpret_cast<uint4 *>(d) = make_uint4(w[0], w[1], w[2], w[3]);
            if (LOCAL) *reinterpret_cast<uint4 *>(d + plane) = make_uint4(e[0], e[1], e[2], e[3]);
        }
    };
    for (int k0 = 0; k0 < nsteps; k0 += 4) {
        if (LOCAL && (k0 & 31) == 0 && k0) {
            lin_chunk(sbs, seen, cid, (k0 >> 5) - 1);
            if (on && k0 < own) lin_snap<R>(tr.snap + ((size_t)(k0 >> 5) * L + sl) * 32, H);
        }
        const uint32_t res4 = cols.next();
        if (k0 >= ks && k0 + 4 <= ke) group(k0, res4, std::false_type());
        else group(k0, res4, std::true_type());
    }
    int4 res = make_int4(0, 0, 0, 0);
    if (LOCAL) {
        lin_chunk(sbs, seen, cid, (nsteps - 1) >> 5);
        if (has) tr.ids[sl] = cid;
        if (!on) sbs = 0;
        int bs = max(lo16(sbs), hi16(sbs));
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) bs = max(bs, __shfl_xor_sync(FULL, bs, o));
        const int g = lane & ~(L - 1);
        const uint32_t lm = L == 32 ? FULL : (1u << (L & 31)) - 1u;
        const uint32_t m0 = __ballot_sync(FULL, lo16(sbs) == bs) >> g & lm;
        const uint32_t m1 = __ballot_sync(FULL, hi16(sbs) == bs) >> g & lm;
        res = make_int4(bs >> 2, bs > 0 ? (int)m0 : 0, bs > 0 ? (int)m1 : 0, bs > 0 ? 1 : 0);
    } else {
        const int rl = has ? (m - 1) % R : -1, h = v_last & 1;
        int hs = 0;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r == rl) hs = half16(H[r], h);
        res.x = __shfl_sync(FULL, hs, (lane & ~(L - 1)) + (t_last > 0 ? t_last : 0)) >> 2;
    }
    return res;
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

// Wait (one lane) until the stripe above has written `need` columns of its
// boundary row.  Stripes are taken in list order, so the one waited for is
// already running or done and the wait ends; after 2^24 polls (seconds) it
// gives up, sets ST_WAIT, and the batch fails with an error.
__device__ __forceinline__ void lin_wait(const uint32_t *p, uint32_t need, int *status)
{
    for (int it = 0; ld_acquire(p) < need; ++it) {
        __nanosleep(64);
        if ((it & 1023) == 1023 && (*(volatile int *)status & ST_WAIT)) return;
        if (it >= (1 << 24)) { atomicOr(status, ST_WAIT); return; }
    }
}

// One stripe of 64 R rows (the last: what is left) of a region on a warp.
// Values are relative to the lane's base B (a multiple of 4, moved every 32 steps
// so that the lane's values lie around LIN_MID, all of them positive).  V: the region's first row; rows rb ..
// of it are this stripe's.  bin / bout: boundary rows (4 H of columns 1..n) of
// the stripe above and of this one (null: none), pin / pout their progress.
template <bool LOCAL, int R>
__device__ __forceinline__ int4 lin_stripe(const uint32_t *tab, uint32_t *prof, const LinConst &c,
                                           const uint8_t *V, int m, int rb, const uint8_t *Hs, int n,
                                           uint8_t *dir, const int *bin, const uint32_t *pin, int *bout,
                                           uint32_t *pout, size_t plane, const LinTrack &tr, int *status)
{
    constexpr int NG = (R + 3) / 4;
    const int lane = threadIdx.x & 31;
    const int rows = min(64 * R, m - rb);
    const int v_last = (rows - 1) / R;
    const int t_last = v_last >> 1;
    const bool on = lane <= t_last;
    const int hi_on = 2 * lane + 1 <= v_last ? 1 : 0;
    const int i_base = rb + 2 * lane * R;
    const unsigned lim = on ? (unsigned)(n + hi_on) : 0u;
    __syncwarp();
    lin_profile<R>(tab, V, i_base, m, on, prof);
    __syncwarp();
    // column 0; the lane's first row there at LIN_MID
    int B = (LOCAL ? 0 : c.go4 * i_base) - LIN_MID;
    uint32_t H[R];
#pragma unroll
    for (int r = 0; r < R; ++r) H[r] = pk16(LIN_MID + (LOCAL ? 0 : c.go4 * (r + 1)), LIN_NEG);
    const int lo0 = LIN_MID + (LOCAL ? 0 : c.go4 * R), hi0 = LIN_MID + (LOCAL ? 0 : c.go4 * 2 * R);
    uint32_t in_h = pk16(LIN_MID, lo0), out_h = pk16(lo0, hi0);
    LinCols cols;
    cols.init(Hs, n, -2 * lane);
    const char *lbase = reinterpret_cast<const char *>(prof + lane * NG);
    const char *pa = lbase + PG_NRES * (128 * NG);
    uint32_t sbs = 0, seen = 0, cid = 0;
    int abs0 = 0, abs1 = 0;                          // best 4 H of the low and high half's rows so far
    uint32_t floor2 = 0, d2 = 0, b2 = 0;
    int bval = 0;
    const int nsteps = n + v_last;
    const int ks = bout ? 64 : 2 * t_last;           // (a stripe with one below has all its lanes)
    uint8_t *dst = dir + lane * 32;
    // one step: the low half's column x (0-based), its residue code
    auto step = [&](const int k, const uint32_t code) {
        const uint32_t rh = v16add(__shfl_up_sync(FULL, out_h, 1), d2);
        const uint32_t bh = (uint32_t)__shfl_sync(FULL, bval, k & 31);
        const uint32_t dgH = in_h;
        const uint32_t th = lane == 0 ? bh : rh;
        in_h = prmt(th, out_h, 0x5432u);
        return dgH;
    };
    auto rows_of = [&](const uint32_t dgH, const uint32_t code) {
        const char *ph = pa + LIN_NC * (128 * NG);
        pa = lbase + code * (128 * NG);
        const uint32_t w = lin_rows<R, LOCAL, true>(H, dgH, in_h, reinterpret_cast<const uint32_t *>(pa),
                                                    reinterpret_cast<const uint32_t *>(ph), c, floor2);
        out_h = H[R - 1];
        if (LOCAL) sbs = lin_max<R>(sbs, H);
        return w;
    };
    // four steps with every lane inside its columns
    auto group = [&](const int k0, const uint32_t res4) {
        uint32_t w[4], e[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t code = (res4 >> (8 * s)) & 0xffu;
            const uint32_t dgH = step(k0 + s, code);
            w[s] = rows_of(dgH, code);
            e[s] = LOCAL ? v16add(out_h, b2) : out_h;
        }
        if (on) {
            uint8_t *d = dst + (size_t)(k0 >> 3) * 1024 + (k0 & 4) * 4;
            *reinterpret_cast<uint4 *>(d) = make_uint4(w[0], w[1], w[2], w[3]);
            if (LOCAL) *reinterpret_cast<uint4 *>(d + plane) = make_uint4(e[0], e[1], e[2], e[3]);
        }
        // the stripe's last row, 64 R - 1: the last lane's high half, columns
        // k0 - 62 and on, two to a store
        if (bout && lane == 31) {
            int v[4];
            // (local: e holds the values mod 2^16)
#pragma unroll
            for (int s = 0; s < 4; ++s)
                v[s] = (LOCAL ? (int)(int16_t)(uint16_t)((e[s] >> 16) - (uint32_t)B) : hi16(e[s])) + B;
            int2 *o = reinterpret_cast<int2 *>(bout + (k0 - 62));
            o[0] = make_int2(v[0], v[1]);
            o[1] = make_int2(v[2], v[3]);
        }
    };
    // four steps, each lane tested: the ramps (a loop, to keep the code small)
    auto ramp = [&](const int k0, const uint32_t res4) {
#pragma unroll 1
        for (int s = 0; s < 4; ++s) {
            const uint32_t code = (res4 >> (8 * s)) & 0xffu;
            const uint32_t dgH = step(k0 + s, code);
            const int x = k0 + s - 2 * lane;
            if ((unsigned)x < lim) {
                uint32_t *d = reinterpret_cast<uint32_t *>(dst + (size_t)(k0 >> 3) * 1024 + ((k0 & 4) + s) * 4);
                *d = rows_of(dgH, code);
                if (LOCAL) *reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>(d) + plane) = v16add(out_h, b2);
                if (bout && lane == 31 && x >= 1) bout[x] = hi16(out_h) + B;
            }
        }
    };
    for (int k0 = 0; k0 < nsteps; k0 += 4) {
        if ((k0 & 31) == 0) {
            if (LOCAL && k0) lin_chunk(sbs, seen, cid, (k0 >> 5) - 1);
            {
                // move the base of the lanes whose two halves hold real columns
                const int sh = k0 - 1 - 2 * lane >= 1 ? (lo16(H[0]) & ~3) - LIN_MID : 0;
                const uint32_t s2 = pk16(-sh, -sh);
                if (LOCAL) {
                    abs0 = max(abs0, lo16(sbs) + B);
                    abs1 = max(abs1, hi16(sbs) + B);
                }
                B += sh;
                b2 = pk16(B, B);
#pragma unroll
                for (int r = 0; r < R; ++r) H[r] = v16add(H[r], s2);
                in_h = v16add(in_h, s2);
                out_h = v16add(out_h, s2);
                if (LOCAL) {
                    const int f = max(-B, LIN_NEG);
                    floor2 = pk16(f, f);
                    // the maximum so far, as far as the new base can tell it: past
                    // int16 no value of the next 32 columns reaches it
                    sbs = pk16(min(max(abs0 - B, LIN_NEG), 32767), min(max(abs1 - B, LIN_NEG), 32767));
                    seen = sbs;
                }
                const int d = __shfl_up_sync(FULL, B, 1) - B;
                d2 = pk16(0, d);                     // the lane above hands its high half down
            }
            if (LOCAL && k0 && on) {
                lin_snap<R>(tr.snap + ((size_t)(k0 >> 5) * 32 + lane) * 32, H);
                tr.base[(k0 >> 5) * 32 + lane] = B;
            }
            const int j = k0 + 1 + lane;             // boundary columns of the next 32 steps
            const int b0 = __shfl_sync(FULL, B, 0);
            int h = LOCAL ? 0 : c.go4 * j;
            if (bin) {
                const int need = min(n, k0 + 32);
                if (lane == 0 && k0 < n) lin_wait(pin, (uint32_t)need, status);
                __syncwarp();
                h = j <= n ? __ldcg(bin + j) : 0;
            }
            bval = (j <= n ? h - b0 : 0) << 16;
        }
        const uint32_t res4 = cols.next();
        if (k0 >= ks && k0 + 4 <= n) {
            group(k0, res4);
        } else {
            ramp(k0, res4);
        }
        if (bout && lane == 31 && (k0 & 28) == 28 && k0 >= 60)
            st_release(pout, (uint32_t)min(n, k0 + 3 - 62));
    }
    if (bout && lane == 31) st_release(pout, (uint32_t)n);
    int4 res = make_int4(0, 0, 0, 0);
    if (LOCAL) {
        lin_chunk(sbs, seen, cid, (nsteps - 1) >> 5);
        tr.ids[lane] = cid;
        abs0 = on ? max(abs0, lo16(sbs) + B) : 0;
        abs1 = on ? max(abs1, hi16(sbs) + B) : 0;
        int bs = max(abs0, abs1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) bs = max(bs, __shfl_xor_sync(FULL, bs, o));
        const uint32_t m0 = __ballot_sync(FULL, abs0 == bs), m1 = __ballot_sync(FULL, abs1 == bs);
        res = make_int4(bs >> 2, bs > 0 ? (int)m0 : 0, bs > 0 ? (int)m1 : 0, bs > 0 ? 1 : 0);
    } else {
        const int rl = (rows - 1) % R, h = v_last & 1;
        int hs = 0;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r == rl) hs = half16(H[r], h) + B;
        res.x = __shfl_sync(FULL, hs, t_last) >> 2;
    }
    return res;
}

// Each class has its own job counter (a job: a group of 32 / L regions, or a
// stripe), its jobs taken in list order.  The global form goes through the classes
// in order.  In the local form, whose loops are larger, an SM starts on the class
// that holds its share of the batch's work and goes on with the classes after it:
// an SM then runs one class's code at a time, and every class's long jobs start
// early (8k uneven pairs: 5.74 ms in class order, where a late class's longest job
// runs alone at the end; 7.35 ms with the longest jobs of all classes first, whose
// loops together do not fit the instruction cache; 4.74 ms this way.  The global
// form lost 6 % by it, its loops fit).
template <bool LOCAL>
__global__ void __launch_bounds__(WARPS * 32, 2) k_lin_dp(const LinParams lp, int nsm)
{
    __shared__ __align__(16) int8_t tab8[LIN_NC * LIN_ROWB];
    __shared__ uint32_t sl[2 * LIN_CLS];
    __shared__ int first;
    lin_table(tab8, lp.kp.sm, LOCAL);
    for (int t = threadIdx.x; t < 2 * LIN_CLS; t += blockDim.x) sl[t] = lp.tot->cls[t];
    if (threadIdx.x < 32) {
        const int k = threadIdx.x;
        const double w = LOCAL && k < LIN_CLS ? (double)lp.tot->work[k] : 0.0;
        double acc = w;                            // inclusive prefix over the classes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(FULL, acc, o);
            if (k >= o) acc += y;
        }
        uint32_t smid;
        asm("mov.u32 %0, %%smid;" : "=r"(smid));
        const double at = __shfl_sync(FULL, acc, 31) * (double)(smid % (uint32_t)nsm) / (double)nsm;
        const uint32_t past = __ballot_sync(FULL, acc > at && w > 0.0);
        if (k == 0) first = past ? __ffs(past) - 1 : 0;
    }
    __syncthreads();
    const uint32_t *tab = reinterpret_cast<const uint32_t *>(tab8);
    const int lane = threadIdx.x & 31;
    uint32_t *prof = reinterpret_cast<uint32_t *>(g_dyn_prof) + (threadIdx.x >> 5) * (LIN_PROF / 4);
    LinConst c;
    c.go4 = 4 * lp.kp.go;
    const int te = (LOCAL ? -3 : 0) + lp.e_first, tf = (LOCAL ? -3 : 0) + 1 - lp.e_first;
    c.goL = pk16(c.go4 + te, c.go4 + te);
    c.goU = pk16(c.go4 + tf, c.go4 + tf);
    c.four = (uint32_t)lp.kp.four;
    c.one = c.four >> 2;
    // lane k: the jobs of class k
    const int mine = lane < LIN_CLS ? lane : 0;
    const uint32_t my_jobs = (sl[LIN_CLS + mine] + (uint32_t)lin_seg_group(mine) - 1) / (uint32_t)lin_seg_group(mine);
    int cls = first;
    for (;;) {
        const int lanes = lin_seg_lanes(cls), group = lin_seg_group(cls);
        const uint32_t jobs = __shfl_sync(FULL, my_jobs, cls);
        uint32_t job = jobs;
        if (lane == 0 && jobs) job = atomicAdd(&lp.tot->next_job[cls], 1u);
        job = __shfl_sync(FULL, job, 0);
        if (job >= jobs) {
            // the next class with jobs left, around from this one
            const bool any = lane < LIN_CLS && *(volatile uint32_t *)&lp.tot->next_job[mine] < my_jobs;
            const uint32_t left = __ballot_sync(FULL, any);
            if (!left) break;
            const uint32_t after = left & ~((2u << cls) - 1u);
            cls = __ffs(after ? after : left) - 1;
            continue;
        }
        const uint32_t q = job * (uint32_t)group + (uint32_t)(lane / lanes);
        const bool has = q < sl[LIN_CLS + cls];
        const uint32_t pos = sl[cls] + q;
        LinReg e;
        e.m = e.n = 0; e.v = e.h = 0; e.off = 0; e.stripe = 0; e.nstripe = 1;
        if (has) {
            const uint4 *src = reinterpret_cast<const uint4 *>(lp.list + pos);
            uint4 *d = reinterpret_cast<uint4 *>(&e);
            d[0] = src[0];
            d[1] = src[1];
        }
        const uint8_t *V = lp.kp.rseq + e.v, *Hs = lp.kp.cseq + e.h;
        uint8_t *dir = lp.arena + (uint64_t)e.off * 32u;
        int4 r;
        const LinPlanes pl(LOCAL, cls, e.n);
        LinTrack tr{nullptr, nullptr, nullptr};
        if (LOCAL) {
            uint8_t *q = dir + (uint64_t)e.nstripe * pl.tile * 64u;
            tr.snap = q + (uint64_t)e.stripe * pl.snap * 32u;
            q += (uint64_t)e.nstripe * pl.snap * 32u;
            tr.base = (int *)(q + (uint64_t)e.stripe * pl.base * 32u);
            q += (uint64_t)e.nstripe * pl.base * 32u;
            tr.ids = (uint32_t *)(q + (uint64_t)e.stripe * pl.ids * 32u);
        }
        if (cls < 4) {
            const uint32_t ru = lin_row_units(e.n);
            const size_t plane = (size_t)e.nstripe * pl.tile * 32u;
            uint8_t *rows = dir + (uint64_t)e.nstripe * pl.stripe(LOCAL) * 32u;
            const int *bin = e.stripe ? (const int *)(rows + (uint64_t)(e.stripe - 1) * ru * 32u) : nullptr;
            int *bout = e.stripe + 1 < e.nstripe ? (int *)(rows + (uint64_t)e.stripe * ru * 32u) : nullptr;
            uint8_t *d = dir + (uint64_t)e.stripe * pl.tile * 32u;
            const uint32_t *pin = lp.prog + pos - (e.stripe ? 1 : 0);
            uint32_t *pout = lp.prog + pos;
#define LIN_STRIPE(R_) lin_stripe<LOCAL, R_>(tab, prof, c, V, e.m, (int)e.stripe * 64 * R_, Hs, e.n, d, bin, pin, bout, pout, plane, tr, lp.kp.status)
            switch (cls) {
            case 0: r = LIN_STRIPE(8); break;
            case 1: r = LIN_STRIPE(7); break;
            case 2: r = LIN_STRIPE(6); break;
            default: r = LIN_STRIPE(5); break;
            }
#undef LIN_STRIPE
        } else {
#define LIN_SUB(L_, R_) lin_sub<LOCAL, L_, R_>(tab, prof, c, V, e.m, Hs, e.n, dir, tr)
            switch (cls) {
            case 4: r = LIN_SUB(32, 8); break;
            case 5: r = LIN_SUB(32, 7); break;
            case 6: r = LIN_SUB(32, 6); break;
            case 7: r = LIN_SUB(32, 5); break;
            case 8: r = LIN_SUB(16, 8); break;
            case 9: r = LIN_SUB(16, 7); break;
            case 10: r = LIN_SUB(16, 6); break;
            case 11: r = LIN_SUB(16, 5); break;
            case 12: r = LIN_SUB(8, 8); break;
            case 13: r = LIN_SUB(8, 7); break;
            case 14: r = LIN_SUB(8, 6); break;
            case 15: r = LIN_SUB(8, 5); break;
            case 16: r = LIN_SUB(8, 4); break;
            default: r = LIN_SUB(8, 2); break;
            }
#undef LIN_SUB
        }
        if (has && (lane & (lanes - 1)) == 0) lp.dp[pos] = r;
    }
}

// -------------------------------------------------- the local form's end cell
// The DP keeps only the running maximum of each virtual lane's R rows (half an
// operation per row; following the cell itself, row by row at every new maximum,
// took as many instructions as the recurrence: 130 a step against 77, 100k pairs
// 5.58 -> 3.51 ms) and the 32-step chunk in which it last rose.  The end cell, the first maximum in column-major order, is found
// here: the R rows of a virtual lane that reached the score are computed again
// over that chunk, from their values at its start (the snapshots) and from the
// row above them (the edge words: 4 H mod 2^16 of both halves' last rows at each
// step), up to the first column that holds the score.  At most 32 columns, so a
// thread does it.  Returns column << 3 | row; ~0: none up to column `last`.
struct LinStrip {
    const uint32_t *edge;   // edge words of the virtual lane above (null: row 0)
    const uint32_t *snap;   // this lane's snapshot of the chunk (null: it starts at column 0)
    int base;               // what that is relative to
    int half;               // of the lane
    int va;                 // the virtual lane above + 1, counted in its stripe
    int col;                // column of the snapshot (0: none)
};
__device__ __forceinline__ uint32_t lin_edge(const LinStrip &s, uint32_t tile_row, int j)
{
    const int u = s.va - 1, k = j - 1 + u;
    const uint32_t w = __ldg(s.edge + (uint32_t)(k >> 3) * tile_row + (uint32_t)((u >> 1) * 8 + (k & 7)));
    return u & 1 ? w >> 16 : w & 0xffffu;
}
__device__ __forceinline__ uint32_t lin_locate(const int8_t *sm, const uint8_t *V, int m, int row0, int R,
                                               const uint8_t *Hs, int last, int score, int go,
                                               uint32_t tile_row, const LinStrip &s)
{
    int a[8], H[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        a[r] = (r < R && row0 + r < m ? (int)__ldg(V + row0 + r) : PG_NRES) * 32;
        H[r] = s.col && r < R ? (half16(__ldg(s.snap + r), s.half) + s.base) >> 2 : 0;
    }
    uint32_t raw = 0;
    int top = 0;
    if (s.edge && s.col) {                             // neighbours differ by at most 62
        raw = lin_edge(s, tile_row, s.col);
        top = H[0] + ((int)(int16_t)(uint16_t)(raw - 4u * (uint32_t)H[0]) >> 2);
    }
    for (int j = s.col + 1; j <= last; ++j) {
        int dg = top;
        if (s.edge) {
            const uint32_t x = lin_edge(s, tile_row, j);
            top += (int)(int16_t)(uint16_t)(x - raw) >> 2;
            raw = x;
        }
        const int b = __ldg(Hs + j - 1);
        int up = top, mx = 0;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int d = dg + sm[a[r] + b];
            dg = H[r];
            H[r] = __viaddmax_s32_relu(max(up, H[r]), go, d);
            up = H[r];
            mx = max(mx, up);
        }
        if (mx == score) {
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if (H[r] == score) return ((uint32_t)j << 3) | (uint32_t)r;
        }
    }
    return ~0u;
}

// ------------------------------------------------------------ the traceback
// Counts what computeAlignmentStats counts (src/align/SeqanFullAligner.cpp:238-246):
// diagonal columns (D), identical ones (M), gap runs (G).  A region's walk is
// one chain of dependent reads, so its latency is what counts, in two forms:
//
//  - a thread per region, for the many short ones: moves have no branch on the
//    tag, and locally the tags of four cells along the diagonal are read at once
//    (100k pairs 0.79 -> 0.56 ms; the global form, with half the registers, ran
//    faster one cell at a time, 1.06 against 1.29 ms on 400k X-drop pairs).  A
//    warp waits for whichever of its 32 walks misses L1, about 400 cycles a move.
//  - a warp per region, for regions of many columns (lin_wide) and for batches too
//    small to fill the chip with threads: 16 lanes read the next 16 cells of the diagonal, a
//    ballot gives the run of diagonal moves, and the other lanes bring the
//    sectors of the 16 cells after those into L1.
struct LinPath {
    int i, j;              // in: the end cell; out: the start cell
    uint32_t M, D, G;
};
struct LinDirs {
    const uint32_t *dirs;  // the region's direction words
    uint32_t tile_row;     // words per 8 steps
    uint32_t stripe_words;
    int rows, R;           // of a stripe; per virtual lane
    const uint8_t *V, *Hs;
    int e_tag, f_tag;
};

template <bool LOCAL>
__device__ __forceinline__ void lin_walk_thread(const LinDirs &x, LinPath &p)
{
    constexpr int RUN = LOCAL ? 4 : 1;
    const uint32_t inv = (65536u + (uint32_t)x.R - 1u) / (uint32_t)x.R;   // q / R for q < 8192
    int st = (p.i - 1) / x.rows;
    int q = p.i - 1 - st * x.rows;                 // row in the stripe
    int j = p.j, last = 0;
    const uint32_t *base = x.dirs + (uint64_t)st * x.stripe_words;
    bool more = true;
    while (j > 0 && more) {
        if (q < 0) {
            if (--st < 0) break;
            q = x.rows - 1;
            base -= x.stripe_words;
        }
        // the tags of the next cells along the diagonal, all loads in flight together
        // (past the first row or column: the last valid cell again, not used)
        const int len = min(RUN, min(q + 1, j));
        uint32_t word[RUN];
        int sh[RUN], ra[RUN], rb[RUN], tag[RUN];
#pragma unroll
        for (int t = 0; t < RUN; ++t) {
            const int tt = RUN > 1 ? min(t, len - 1) : 0, qt = q - tt;
            const int v = (int)((uint32_t)qt * inv >> 16);
            const int k = j - 1 - tt + v;
            word[t] = __ldg(base + (uint32_t)(k >> 3) * x.tile_row + (uint32_t)((v >> 1) * 8 + (k & 7)));
            sh[t] = 16 * (v & 1) + 2 * (x.R - 1 - (qt - v * x.R));
            if (LOCAL) { ra[t] = __ldg(x.V + st * x.rows + qt); rb[t] = __ldg(x.Hs + j - 1 - tt); }
        }
        // the diagonal run, then the gap (or the end) after it
        int run = 0, gap = 0;
        bool on = true;
#pragma unroll
        for (int t = 0; t < RUN; ++t) {
            tag[t] = (int)(word[t] >> sh[t]) & 3;
            on = on && t < len && (LOCAL ? tag[t] == 1 : tag[t] >= 2);
            run += on ? 1 : 0;
            p.M += on && (LOCAL ? ra[t] == rb[t] : tag[t] == 3) ? 1u : 0u;
        }
#pragma unroll
        for (int t = 0; t < RUN; ++t)
            if (t == run && t < len) {
                gap = tag[t] == x.f_tag ? 1 : tag[t] == x.e_tag ? 2 : 0;
                more = gap != 0;
            }
        p.D += (uint32_t)run;
        last = run ? 0 : last;
        p.G += gap && gap != last ? 1u : 0u;
        last = gap ? gap : last;
        q -= run + (gap == 1 ? 1 : 0);
        j -= run + (gap == 2 ? 1 : 0);
    }
    p.i = st < 0 ? 0 : st * x.rows + q + 1;
    p.j = j;
    if (!LOCAL && ((p.i > 0 && last != 1) || (j > 0 && last != 2))) ++p.G;
}

// the same by a warp; dummy: this lane's 4 bytes of shared memory
template <bool LOCAL>
__device__ __forceinline__ void lin_walk_warp(const LinDirs &x, LinPath &p, uint32_t *dummy)
{
    constexpr int RUN = 16;
    const int lane = threadIdx.x & 31;
    const uint32_t inv = (65536u + (uint32_t)x.R - 1u) / (uint32_t)x.R;
    const uint32_t sdummy = (uint32_t)__cvta_generic_to_shared(dummy);
    int st = (p.i - 1) / x.rows;
    int q = p.i - 1 - st * x.rows;
    int j = p.j, last = 0;
    const uint32_t *base = x.dirs + (uint64_t)st * x.stripe_words;
    int ra = 0, rb = 1;                            // local: the residues of the run before, and its cells
    uint32_t ran = 0;
    bool more = true;
    while (j > 0 && more) {
        if (q < 0) {
            if (--st < 0) break;
            q = x.rows - 1;
            base -= x.stripe_words;
        }
        const int len = min(RUN, min(q + 1, j));
        // lane t: the cell t moves along the diagonal (lanes past the run's reach
        // fetch ahead: a copy into shared memory that nothing waits for)
        const int tt = min(lane, min(q, j - 1)), qt = q - tt;
        const int v = (int)((uint32_t)qt * inv >> 16);
        const int k = j - 1 - tt + v;
        const uint32_t *w = base + (uint32_t)(k >> 3) * x.tile_row + (uint32_t)((v >> 1) * 8 + (k & 7));
        uint32_t word = 0;
        if (lane < RUN) {
            word = __ldg(w);
        } else {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(sdummy), "l"(w) : "memory");
        }
        if (LOCAL) {
            p.M += (uint32_t)__popc(__ballot_sync(FULL, ra == rb) & ran);
            ra = __ldg(x.V + st * x.rows + qt);
            rb = __ldg(x.Hs + j - 1 - tt);
        }
        const int tag = (int)(word >> (16 * (v & 1) + 2 * (x.R - 1 - (qt - v * x.R)))) & 3;
        const bool cell = lane < len && (LOCAL ? tag == 1 : tag >= 2);
        const int run = __ffs(~__ballot_sync(FULL, cell)) - 1;     // lane RUN is never one of them
        if (LOCAL) ran = (1u << run) - 1u;
        else p.M += (uint32_t)__popc(__ballot_sync(FULL, cell && tag == 3) & ((1u << run) - 1u));
        p.D += (uint32_t)run;
        last = run ? 0 : last;
        int gap = 0;
        if (run < len) {
            const int g = __shfl_sync(FULL, tag, run);
            gap = g == x.f_tag ? 1 : g == x.e_tag ? 2 : 0;
            more = gap != 0;
        }
        p.G += gap && gap != last ? 1u : 0u;
        last = gap ? gap : last;
        q -= run + (gap == 1 ? 1 : 0);
        j -= run + (gap == 2 ? 1 : 0);
    }
    if (LOCAL) p.M += (uint32_t)__popc(__ballot_sync(FULL, ra == rb) & ran);
    p.i = st < 0 ? 0 : st * x.rows + q + 1;
    p.j = j;
    if (!LOCAL && ((p.i > 0 && last != 1) || (j > 0 && last != 2))) ++p.G;
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// regions per SM up to which every walk has a warp of its own
constexpr uint32_t LIN_WALK_WARPS = 64;

// blocks [0, warp_blocks): a warp for each wide region (all: for each entry of the
// list); the rest: a thread per entry
template <bool LOCAL>
__global__ void __launch_bounds__(256) k_lin_walk(const LinParams lp, uint32_t warp_blocks, bool all)
{
    __shared__ int8_t sm[LIN_NC * 32];
    __shared__ uint32_t dummy[256];
    if (LOCAL) {
        for (int t = threadIdx.x; t < LIN_NC * 32; t += blockDim.x)
            sm[t] = t < PG_NRES * 32 ? ((t & 31) < PG_NRES ? lp.kp.sm[(t >> 5) * PG_NRES + (t & 31)] : (int8_t)0)
                                     : (int8_t)-128;
        __syncthreads();
    }
    const bool warp = blockIdx.x < warp_blocks;
    uint32_t pos = warp ? blockIdx.x * 8u + (threadIdx.x >> 5) : (blockIdx.x - warp_blocks) * 256u + threadIdx.x;
    if (pos >= (warp && !all ? lp.tot->wide : lp.tot->entries)) return;
    if (warp && !all) pos = lp.wlist[pos];
    LinReg e;
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(lp.list + pos);
        uint4 *d = reinterpret_cast<uint4 *>(&e);
        d[0] = src[0];
        d[1] = src[1];
    }
    if (e.stripe || (!warp && e.n >= lin_wide(LOCAL))) return;
    const int m = e.m, n = e.n, ns = e.nstripe;
    const int cls = lin_class(lp, LOCAL, m, n);
    const int L = lin_seg_lanes(cls), R = lin_seg_rows(cls);
    LinDirs x;
    x.V = lp.kp.rseq + e.v; x.Hs = lp.kp.cseq + e.h;
    x.tile_row = (uint32_t)L * 8u;
    x.stripe_words = lin_tile_units(L, n) * 8u;
    x.dirs = reinterpret_cast<const uint32_t *>(lp.arena + (uint64_t)e.off * 32u);
    x.rows = 2 * L * R; x.R = R;
    x.e_tag = LOCAL ? 3 - lp.e_first : lp.e_first;
    x.f_tag = LOCAL ? 2 + lp.e_first : 1 - lp.e_first;
    int4 d = lp.dp[pos + (LOCAL ? 0 : ns - 1)];
    LinPath p{m, n, 0u, 0u, 0u};
    if (LOCAL) {
        for (int s = 1; s < ns; ++s) {
            const int4 o = lp.dp[pos + s];
            if (o.x > d.x) d = o;
        }
        // every virtual lane that reached the score: the smallest column, then row
        const LinPlanes pl(true, cls, n);
        const uint32_t *edges = x.dirs + (uint64_t)ns * x.stripe_words;
        const uint32_t *snaps = edges + (uint64_t)ns * x.stripe_words;
        const int *bases = reinterpret_cast<const int *>(snaps + (uint64_t)ns * pl.snap * 8u);
        const uint32_t *ids = reinterpret_cast<const uint32_t *>(bases) + (uint64_t)ns * pl.base * 8u;
        p.i = 0;
        for (int s = 0; d.w && s < ns; ++s) {
            const int4 o = lp.dp[pos + s];
            if (o.x != d.x) continue;
#pragma unroll 1
            for (uint32_t m0 = (uint32_t)o.y, m1 = (uint32_t)o.z; m0 | m1;) {
                const int f0 = m0 ? __ffs(m0) - 1 : 32, f1 = m1 ? __ffs(m1) - 1 : 32;
                const int v = f0 <= f1 ? 2 * f0 : 2 * f1 + 1;
                if (f0 <= f1) m0 &= m0 - 1; else m1 &= m1 - 1;
                const int row0 = (s * 2 * L + v) * R, t = v >> 1;
                LinStrip q;
                q.half = v & 1;
                // the row above: the virtual lane before, or the last one of the stripe above
                q.edge = edges + (uint64_t)s * x.stripe_words;
                q.va = v;
                if (v == 0) { q.va = 2 * L; q.edge = s ? q.edge - x.stripe_words : nullptr; }
                const int c = (int)((__ldg(ids + (uint64_t)s * pl.ids * 8u + t) >> (16 * q.half)) & 0xffffu);
                const int start = 32 * c - 2 * t - q.half;       // its column before the chunk
                q.col = max(0, start);
                q.snap = snaps + ((uint64_t)s * pl.snap + (uint64_t)(c * L + t)) * 8u;
                q.base = q.col && cls < 4 ? __ldg(bases + (uint64_t)s * pl.base * 8u + (uint64_t)(c * 32 + t)) : 0;
                // an earlier find wins a tie (its rows are above)
                const int lim = min(p.i ? p.j - 1 : n, start + 32);
                const uint32_t z = lin_locate(sm, x.V, m, row0, R, x.Hs, lim, d.x, lp.kp.go, x.tile_row, q);
                if (z != ~0u) { p.j = (int)(z >> 3); p.i = row0 + (int)(z & 7u) + 1; }
            }
        }
        if (d.w && !p.i) {
            // the DP saw the score in one of these lanes: not an empty result
            atomicOr(lp.kp.status, ST_END);
            d.w = 0;
        }
    }
    const int end_i = p.i, end_j = p.j;
    if (!LOCAL || d.w) {
        if (warp) lin_walk_warp<LOCAL>(x, p, dummy + threadIdx.x);
        else lin_walk_thread<LOCAL>(x, p);
    }
    if (warp && (threadIdx.x & 31)) return;
    if (!LOCAL) {
        lp.walk[e.key] = make_int4(d.x, (int)p.M, (int)p.D, (int)p.G);
        return;
    }
    pg_result o = empty_result();
    o.cells = sat_u32((uint64_t)m * (uint64_t)n);
    if (d.w) {
        const uint32_t len = (uint32_t)((end_i - p.i) + (end_j - p.j)) - p.D;
        o.score = d.x;
        o.aln_len = len; o.matches = p.M; o.gap_opens = p.G;
        o.beg_v = (uint16_t)p.i; o.end_v = (uint16_t)end_i;
        o.beg_h = (uint16_t)p.j; o.end_h = (uint16_t)end_j;
        if (len > 0) { o.identity = identity_of(p.M, len); o.flags = 0; }
    }
    apply_filter(o, m, n, lp.kp.cov_thr, lp.kp.ani_thr);
    lp.kp.out[e.key] = o;
}

// X-drop: the record of each pair from its regions' walks (the better seed by
// identity, as SeqanXdropAligner.cpp:303-354), one thread per pair
static __global__ void __launch_bounds__(256) k_lin_finish(const LinParams lp)
{
    const KParams &kp = lp.kp;
    const int gmax = kp.go;                          // go > ge
    for (uint64_t p = lp.p0 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < lp.p1;
         p += (uint64_t)gridDim.x * blockDim.x) {
        const LinPair r = lin_pair<true>(kp, p);
        pg_result best = empty_result();
        if (r.bad) {
            atomicOr(kp.status, ST_BAD_INDEX);
            kp.out[p] = best;
            continue;
        }
        const pg_pair pr = kp.pairs[p];
        const uint64_t ri = (uint64_t)pr.row + kp.roff, ci = (uint64_t)pr.col + kp.coff;
        const XdRec rec0 = kp.xd[2 * p], rec1 = kp.xd[2 * p + 1];
        uint64_t cells = 0;
        bool bad = false, have = false;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const XdRec &rec = s ? rec1 : rec0;
            if (rec.flags & XF_NONE) continue;
            if (rec.flags & XF_SAME) {
                cells += (uint64_t)rec0.cells + (uint64_t)(rec0.ev - rec0.bv) * (uint64_t)(rec0.eh - rec0.bh);
                continue;
            }
            if (rec.flags & XF_BAD) bad = true;
            const int rm = rec.ev - rec.bv, rn = rec.eh - rec.bh;
            cells += rec.cells + (uint64_t)rm * (uint64_t)rn;
            if (s == 1 && !(rec0.flags & XF_NONE) && rec.bv == rec0.bv && rec.ev == rec0.ev &&
                rec.bh == rec0.bh && rec.eh == rec0.eh) continue;   // the first seed's region again
            int score = 0;
            uint32_t M = 0, D = 0, G = 0;
            if (r.dp[s]) {
                const int4 w = lp.walk[2 * p + s];
                score = w.x; M = (uint32_t)w.y; D = (uint32_t)w.z; G = (uint32_t)w.w;
            } else if (rm + rn > 0) {
                score = kp.go + (rm + rn - 1) * gmax;               // one gap run
                G = 1;
            }
            const uint32_t L = (uint32_t)(rm + rn) - D;
            pg_result cur;
            cur.score = score; cur.aln_len = L; cur.matches = M; cur.gap_opens = G;
            cur.beg_v = rec.bv; cur.end_v = rec.ev;
            cur.beg_h = rec.bh; cur.end_h = rec.eh;
            cur.seed_used = (uint8_t)s; cur.pad = 0; cur.cells = 0; cur.score_aln = 0.0f;
            if (L == 0) { cur.identity = 0.0f; cur.flags = PG_RF_EMPTY; }
            else { cur.identity = identity_of(M, L); cur.flags = 0; }
            const bool nan = ((cur.flags | best.flags) & PG_RF_EMPTY) != 0;
            if (!have || (!nan && cur.identity > best.identity)) { best = cur; have = true; }
        }
        best.cells = sat_u32(cells);
        if (bad) best.flags |= PG_RF_BAD_SEED;
        apply_filter(best, (int)(kp.roffs[ri + 1] - kp.roffs[ri]), (int)(kp.coffs[ci + 1] - kp.coffs[ci]),
                     kp.cov_thr, kp.ani_thr);
        kp.out[p] = best;
    }
}

#ifdef PG_LIN_UNIT
// ------------------------------------------------------------ host launches
// (only in the units that instantiate them: a second copy of the kernels would
// come with every other include)
template <bool XDROP>
cudaError_t lin_attributes(int *blocks_per_sm)
{
    cudaError_t e = cudaFuncSetAttribute(k_lin_dp<!XDROP>, cudaFuncAttributeMaxDynamicSharedMemorySize, LIN_DYN);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_lin_dp<!XDROP>, WARPS * 32, LIN_DYN);
    return e;
}
// class sizes and totals of the pairs [p0, p1): 2 launches
template <bool XDROP>
void lin_count(const LinParams &lp, int nsm, cudaStream_t st)
{
    const uint64_t n = lp.p1 - lp.p0;
    const uint64_t grid = (n + LIN_PT - 1) / LIN_PT;
    k_lin_hist<XDROP><<<(int)(grid < (uint64_t)nsm * 8 ? grid : (uint64_t)nsm * 8), LIN_PT, 0, st>>>(lp);
    k_lin_scan<<<1, 1024, 0, st>>>(lp);
}
// list, DP, traceback and results; returns the launches
template <bool XDROP>
int lin_align(const LinParams &lp, uint32_t entries, uint32_t wide, uint32_t jobs, int nsm, int max_blocks,
              cudaStream_t st)
{
    const uint64_t n = lp.p1 - lp.p0;
    const uint64_t gp = (n + LIN_PT * LIN_PP - 1) / (LIN_PT * LIN_PP);
    k_lin_place<XDROP><<<(int)(gp < (uint64_t)nsm * 8 ? gp : (uint64_t)nsm * 8), LIN_PT, 0, st>>>(lp);
    // fewer jobs than resident warps: as few warps per block as hold them, so that
    // they spread over the SMs
    const uint32_t want = (jobs + (uint32_t)max_blocks - 1) / (uint32_t)max_blocks;
    const int warps = want < 1 ? 1 : want < (uint32_t)WARPS ? (int)want : WARPS;
    k_lin_dp<!XDROP><<<max_blocks, warps * 32, warps * LIN_PROF, st>>>(lp, nsm);
    // a warp per wide region, whose walk is long, and per region while that leaves
    // SMs with no more than LIN_WALK_WARPS of them
    const bool all = entries <= (uint32_t)nsm * LIN_WALK_WARPS;
    const uint32_t wb = ((all ? entries : wide) + 7) / 8, tb = all ? 0 : (entries + 255) / 256;
    k_lin_walk<!XDROP><<<wb + tb ? wb + tb : 1, 256, 0, st>>>(lp, wb, all);
    if (XDROP) {
        const uint64_t gf = (n + 255) / 256;
        k_lin_finish<<<(int)(gf < (uint64_t)nsm * 8 ? gf : (uint64_t)nsm * 8), 256, 0, st>>>(lp);
    }
    return XDROP ? 4 : 3;
}
#endif

}  // namespace pg
