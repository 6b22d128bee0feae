// pg_kernels_xd.cuh -- the X-drop extension kernels (one definition: only
// pg_api.cu includes this file): k_xdr, a thread, for the longest a warp, per
// direction of a (pair, seed) with the band window in registers (pg_xdreg.cuh), the
// default; k_xdf and k_xd, thread per (pair, seed) task with the 32-bit band in a shared-memory ring (pg_xdrop.cuh),
// stepping one direction at a time or running each task to its end (tuning
// option xd_stepped); k_xd16, a thread per task on 16-bit lanes (tuning option
// xd_int16); k_xd_wide, warp per task for the bands that overflow a thread's
// window or ring (after k_xdr it also joins the directions into records).
#pragma once
#include <cstdint>

#include "pg_kernels.cuh"
#include "pg_xdreg.cuh"

namespace pg {

// ------------------------------------------------------------------ k_xd
// One thread per (pair, seed) task, run to its end before the thread takes
// the next: fewer registers than k_xdf (7 resident blocks per SM against 5),
// which wins when the residues stream from DRAM (sequence sets larger than
// L2); a warp waits on its longest extension.
__global__ void __launch_bounds__(XT) k_xd(const KParams kp)
{
    __shared__ int ssm[32 * 32];
    __shared__ int ring[3 * XW * XT];
    load_sm(ssm, kp.sm);
    __syncthreads();
    int *base = ring + threadIdx.x;
    const uint64_t ntask = 2 * kp.n;
    unsigned long long exec = 0;
    for (;;) {
        const uint64_t task = atomicAdd(&kp.counter[1], 1u);
        if (task >= ntask) break;
        const uint64_t p = task >> 1;
        const int s = (int)(task & 1);
        const pg_pair pr = kp.pairs[p];
        XdRec rec{0, 0, 0, 0, 0u, 0u};
        const uint8_t *V, *Hs;
        int m, n;
        if (!pair_seqs(kp, pr, V, m, Hs, n)) {
            rec.flags = XF_BADIDX;
        } else if (s >= kp.seed_count ||
                   (s == 1 && (kp.flags & PG_F_SKIP_SPURIOUS_SEED) && pr.count < 2)) {
            rec.flags = XF_NONE;
        } else if (s == 1 && pr.rs1 == pr.rs0 && pr.cs1 == pr.cs0) {
            rec.flags = XF_SAME;
        } else {
            int bv, ev, bh, eh;
            if (seed_region(kp, pr, s, m, n, bv, ev, bh, eh)) rec.flags |= XF_BAD;
            bool ok = true;
            if (bv > 0 && bh > 0) {
                const XdOut x = xdrop_dir_thread<XW, XT>(V + bv - 1, bv, -1, Hs + bh - 1, bh, -1,
                                                         ssm, kp.xg, kp.xdrop, base);
                ok = x.ok;
                rec.cells += x.cells;
                bv -= x.dv; bh -= x.dh;
            }
            if (ok && ev < m && eh < n) {
                const XdOut x = xdrop_dir_thread<XW, XT>(V + ev, m - ev, 1, Hs + eh, n - eh, 1,
                                                         ssm, kp.xg, kp.xdrop, base);
                ok = x.ok;
                rec.cells += x.cells;
                ev += x.dv; eh += x.dh;
            }
            if (ok) {
                rec.bv = (uint16_t)bv; rec.ev = (uint16_t)ev;
                rec.bh = (uint16_t)bh; rec.eh = (uint16_t)eh;
                exec += rec.cells;
            } else {
                rec.flags |= XF_OVF;
                rec.cells = 0;
                const unsigned int slot = atomicAdd(&kp.counter[2], 1u);
                kp.ovf[slot] = (uint32_t)task;
            }
        }
        kp.xd[task] = rec;
    }
    if (exec) atomicAdd(kp.exec_cells, exec);
}

// ------------------------------------------------------------------ k_xdf
// One thread per (pair, seed) task, each thread stepping one extension
// direction at a time: when a direction ends the thread starts the next one
// at once (the task's other direction, or the next task).  Running each task
// to its end before taking the next, as an earlier kernel did, left a warp
// waiting on its longest extension: 6.5 of 32 lanes active per instruction,
// 28.6 ms per 1M pairs against 16.8 ms here (xdrop1m, sequences in L2).  The next tasks' inputs are read ahead
// in three stages (work counter, pair record, sequence offsets), each
// consumed a task later, so starting a task waits on no memory.  A band
// wider than the 16-slot ring sends the task to the overflow list for
// k_xd_wide.
// a task in the read-ahead pipeline: id, then its pair record, then what
// starting it needs (flags, its seed, its sequences' offsets)
constexpr uint32_t XFT_VALID = 1, XFT_IDX = 2, XFT_SAME = 4, XFT_FEW = 8;
struct XfReady {
    uint32_t t, flags, seed;   // seed: rs | cs << 16 of the task's seed
    uint64_t r0, r1, c0, c1;
};

__global__ void __launch_bounds__(XT) k_xdf(const KParams kp)
{
    __shared__ int ssm[32 * 32];
    __shared__ int ring[3 * XW * XT];
    load_sm(ssm, kp.sm);
    __syncthreads();
    int *base = ring + threadIdx.x;
    const uint32_t ntask = (uint32_t)(2 * kp.n);
    unsigned long long exec = 0;
    // read-ahead pipeline: ta (task id), tb + pb (pair record), c (ready)
    uint32_t ta, tb;
    pg_pair pb;
    XfReady c;
    auto load_pair = [&](uint32_t t, pg_pair &pr) {
        if (t < ntask) pr = kp.pairs[t >> 1];
    };
    auto make_ready = [&](uint32_t t, const pg_pair &pr, XfReady &x) {
        x.t = t;
        x.flags = 0;
        if (t >= ntask) return;
        x.flags = XFT_VALID;
        const uint64_t r = (uint64_t)pr.row + kp.roff, cc = (uint64_t)pr.col + kp.coff;
        const int s = (int)(t & 1);
        x.seed = s ? ((uint32_t)pr.rs1 | ((uint32_t)pr.cs1 << 16)) : ((uint32_t)pr.rs0 | ((uint32_t)pr.cs0 << 16));
        if (pr.rs1 == pr.rs0 && pr.cs1 == pr.cs0) x.flags |= XFT_SAME;
        if (pr.count < 2) x.flags |= XFT_FEW;
        if (r >= kp.nr || cc >= kp.nc) return;
        x.flags |= XFT_IDX;
        x.r0 = kp.roffs[r]; x.r1 = kp.roffs[r + 1];
        x.c0 = kp.coffs[cc]; x.c1 = kp.coffs[cc + 1];
    };
    {
        const uint32_t t0 = atomicAdd(&kp.counter[1], 1u);
        pg_pair p0;
        load_pair(t0, p0);
        make_ready(t0, p0, c);
        tb = atomicAdd(&kp.counter[1], 1u);
        load_pair(tb, pb);
        ta = atomicAdd(&kp.counter[1], 1u);
    }

    XdDir<XW, XT> dir;
    XdRec rec{0, 0, 0, 0, 0u, 0u};
    uint32_t task = 0;
    const uint8_t *V = nullptr, *Hs = nullptr;
    int m = 0, n = 0, bv = 0, ev = 0, bh = 0, eh = 0;
    int phase = 0;     // 0: start a task, 1: left direction running, 2: right direction running
    auto write_rec = [&]() {
        if (rec.flags & XF_OVF) {
            rec.cells = 0;
            const unsigned int slot = atomicAdd(&kp.counter[2], 1u);
            kp.ovf[slot] = task;
        } else if (!(rec.flags & (XF_NONE | XF_SAME | XF_BADIDX))) {
            rec.bv = (uint16_t)bv; rec.ev = (uint16_t)ev;
            rec.bh = (uint16_t)bh; rec.eh = (uint16_t)eh;
            exec += rec.cells;
        }
        kp.xd[task] = rec;
    };
    for (;;) {
        while (phase == 0) {
            if (!(c.flags & XFT_VALID)) break;
            // take c, move the pipeline on by one task
            const XfReady cur = c;
            make_ready(tb, pb, c);
            tb = ta;
            load_pair(tb, pb);
            ta = atomicAdd(&kp.counter[1], 1u);
            task = cur.t;
            const int s = (int)(task & 1);
            rec = XdRec{0, 0, 0, 0, 0u, 0u};
            if (!(cur.flags & XFT_IDX)) {
                rec.flags = XF_BADIDX;
            } else if (s >= kp.seed_count ||
                       (s == 1 && (kp.flags & PG_F_SKIP_SPURIOUS_SEED) && (cur.flags & XFT_FEW))) {
                rec.flags = XF_NONE;
            } else if (s == 1 && (cur.flags & XFT_SAME)) {
                rec.flags = XF_SAME;
            } else {
                V = kp.rseq + cur.r0; m = (int)(cur.r1 - cur.r0);
                Hs = kp.cseq + cur.c0; n = (int)(cur.c1 - cur.c0);
                // seed_region for the task's seed
                bv = (int)(cur.seed & 0xffffu); bh = (int)(cur.seed >> 16);
                ev = bv + kp.seed_len; eh = bh + kp.seed_len;
                if (ev > m || eh > n) {
                    bv = min(bv, m); ev = min(ev, m); bh = min(bh, n); eh = min(eh, n);
                    rec.flags |= XF_BAD;
                }
                if (bv > 0 && bh > 0) {
                    dir.init(V + bv - 1, bv, -1, Hs + bh - 1, bh, -1, kp.xg, kp.xdrop, base);
                    phase = 1;
                } else if (ev < m && eh < n) {
                    dir.init(V + ev, m - ev, 1, Hs + eh, n - eh, 1, kp.xg, kp.xdrop, base);
                    phase = 2;
                }
            }
            if (phase == 0) write_rec();
        }
        if (phase == 0) break;          // no task left for this thread
        if (dir.step(ssm, kp.xg, kp.xdrop, base)) continue;
        const XdOut x = dir.finish(base);
        rec.cells += x.cells;
        if (!x.ok) {
            rec.flags |= XF_OVF;
            write_rec();
            phase = 0;
        } else if (phase == 1) {
            bv -= x.dv; bh -= x.dh;
            if (ev < m && eh < n) {
                dir.init(V + ev, m - ev, 1, Hs + eh, n - eh, 1, kp.xg, kp.xdrop, base);
                phase = 2;
            } else {
                write_rec();
                phase = 0;
            }
        } else {
            ev += x.dv; eh += x.dh;
            write_rec();
            phase = 0;
        }
    }
    if (exec) atomicAdd(kp.exec_cells, exec);
}

// --------------------------------------------------------- extension order
// k_xdr's tasks are directions (pair, seed, left or right of the seed), taken
// longest first: a thread that takes a long one late leaves its warp's other
// lanes idle until it ends.  A direction's length is not known beforehand, but the
// shorter of the two sequences' residues on that side bounds it, and ordering by
// that bound (in quarter octaves) gives nearly the ideal finish.  With both
// directions of a seed as one task the kernel took 4.44 ms on 400k pairs and 5.4 on
// 60k of uneven lengths, 4.13 and 4.51 so (and 3.8 with the longest on warps).
// Directions with nothing to extend are not listed.
__device__ __forceinline__ int xdir_bucket(int len)
{
    const uint32_t b = (uint32_t)len + 2u;               // >= 2
    const int e = 31 - __clz(b);
    return min(XBUCKET - 1, 4 * e + (int)((b << 2 >> e) & 3u));
}

// the length in the middle of a bucket, about
__device__ __forceinline__ float xdir_bucket_len(int b)
{
    return exp2f(0.25f * (float)b + 0.125f);
}
// directions shorter than this are a thread's whatever the batch
constexpr float XDR_LONG = 64.0f;

// the buckets of pair p's four directions (-1: not listed)
__device__ __forceinline__ void xdir_buckets(const KParams &kp, uint64_t p, int (&b)[4])
{
    b[0] = b[1] = b[2] = b[3] = -1;
    const pg_pair pr = kp.pairs[p];
    const uint64_t r = (uint64_t)pr.row + kp.roff, c = (uint64_t)pr.col + kp.coff;
    if (r >= kp.nr || c >= kp.nc) return;
    const int m = (int)(kp.roffs[r + 1] - kp.roffs[r]), n = (int)(kp.coffs[c + 1] - kp.coffs[c]);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        int bv, ev, bh, eh;
        if (xd_seed(kp, pr, s, m, n, bv, ev, bh, eh) & (XF_NONE | XF_SAME)) continue;
        if (bv > 0 && bh > 0) b[2 * s] = xdir_bucket(min(bv, bh));
        if (ev < m && eh < n) b[2 * s + 1] = xdir_bucket(min(m - ev, n - eh));
    }
}

__global__ void __launch_bounds__(256) k_xtask_hist(const KParams kp)
{
    __shared__ unsigned int h[XBUCKET];
    for (int b = threadIdx.x; b < XBUCKET; b += blockDim.x) h[b] = 0;
    __syncthreads();
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < kp.n;
         p += (uint64_t)gridDim.x * blockDim.x) {
        int b[4];
        xdir_buckets(kp, p, b);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (b[k] >= 0) atomicAdd(&h[b[k]], 1u);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < XBUCKET; b += blockDim.x)
        if (h[b]) atomicAdd(&kp.xsched[b], h[b]);
}

// xorder[]: direction ids 4 p + 2 s + side, highest bucket first (any order inside
// a bucket)
__global__ void __launch_bounds__(256) k_xtask_bucket(const KParams kp)
{
    __shared__ unsigned int start[XBUCKET], h[XBUCKET], base[XBUCKET];
    if (threadIdx.x == 0) {
        unsigned int acc = 0;
        for (int b = XBUCKET - 1; b >= 0; --b) { start[b] = acc; acc += kp.xsched[b]; }
    }
    uint32_t *order = const_cast<uint32_t *>(kp.xorder);
    const uint64_t ntask = 4 * kp.n;
    for (uint64_t c0 = (uint64_t)blockIdx.x * blockDim.x; c0 < kp.n; c0 += (uint64_t)gridDim.x * blockDim.x) {
        for (int b = threadIdx.x; b < XBUCKET; b += blockDim.x) h[b] = 0;
        __syncthreads();
        const uint64_t p = c0 + threadIdx.x;
        int b[4] = {-1, -1, -1, -1};
        unsigned int r[4] = {0, 0, 0, 0};
        if (p < kp.n) {
            xdir_buckets(kp, p, b);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (b[k] >= 0) r[k] = atomicAdd(&h[b[k]], 1u);
        }
        __syncthreads();
        for (int b = threadIdx.x; b < XBUCKET; b += blockDim.x)
            if (h[b]) base[b] = start[b] + atomicAdd(&kp.xsched[XBUCKET + b], h[b]);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (b[k] < 0) continue;
            const uint64_t q = (uint64_t)base[b[k]] + r[k];
            if (q < ntask) order[q] = (uint32_t)(4 * p + k);
            else atomicOr(kp.status, ST_BAD_SCHED);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ k_xdr
// One thread per direction of a (pair, seed) with the band window in registers
// (XrDirT<NW>): every step computes the 2 NW window columns with packed 16-bit
// operations and no branch on the band, so a warp's threads step together
// whatever their band widths.  Directions are taken (longest length bound first
// when kp.xorder is set) and their inputs read ahead as in k_xdf.  A window wider
// than 2 NW - 1 columns is flagged for k_xd_wide, which also joins the directions
// into the (pair, seed) records.  NW = 8 runs: a 12-slot window (NW = 6) executed
// 15 % fewer instructions on xdrop1m, but the 4 % of tasks that outgrew it, rerun on
// 16 slots in a launch of their own, were long homolog extensions at a tenth of
// the warps, and the extension took 9.85 ms per 1M pairs against 9.3.
// Needs xdr_supported(xg, xdrop) and direction ids in 32 bits (n < 2^30).
//
// MIXED (XDR_MIXED to XDR_MIXED_MAX directions a resident warp): a quarter of the warps starts on
// the threads' directions and helps with the long ones after.  With all warps on the long
// ones first the two kinds run one after the other, the second with the machine half
// empty: 12k pairs of ordinary lengths 0.92 -> 0.75 ms, 20k 1.53 -> 1.09, 60k 2.27 -> 1.51;
// uneven ones 1.47 -> 1.14, 2.3 -> 1.52, 4.1 -> 2.69.  An instance of its own, as the loop
// over the two parts made small batches 8 % slower (256 pairs 0.204 -> 0.220).  In the largest
// the mean load passes nearly every length, so that hardly any is long: 300k uneven pairs
// 7.8 -> 7.1 ms, 400k 7.45 -> 7.55, 400k of ordinary lengths 4.31 -> 4.39.
constexpr uint64_t XDR_MIXED = 12, XDR_MIXED_MAX = 576;
// the first `first` directions of the order, a warp each
__device__ __forceinline__ void xdr_long(const KParams &kp, const int *ssm, uint32_t first)
{
    for (;;) {
        uint32_t i = first;
        if ((threadIdx.x & 31) == 0 && first) i = atomicAdd(&kp.xsched[2 * XBUCKET], 1u);
        i = __shfl_sync(FULL, i, 0);
        if (i >= first) break;
        const uint32_t t = kp.xorder[i];
        const pg_pair pr = kp.pairs[t >> 2];
        const uint8_t *V, *Hs;
        int m, n, bv, ev, bh, eh;
        if (!pair_seqs(kp, pr, V, m, Hs, n)) continue;
        xd_seed(kp, pr, (int)((t >> 1) & 1), m, n, bv, ev, bh, eh);
        const bool right = t & 1;
        const XdOut x = xdrop_dir_regs(right ? V + ev : V + bv - 1, right ? m - ev : bv, right ? 1 : -1,
                                          right ? Hs + eh : Hs + bh - 1, right ? n - eh : bh, right ? 1 : -1,
                                          ssm, kp.xg, kp.xdrop);
        if ((threadIdx.x & 31) == 0) {
            XdSide o;
            o.dv = (uint16_t)x.dv; o.dh = (uint16_t)x.dh;
            o.cells = x.ok ? x.cells : XDIR_OVF;
            kp.xdir[t] = o;
            if (!x.ok) kp.ovf[atomicAdd(&kp.counter[2], 1u)] = t;
        }
    }
}

// the directions after the first `first` ones, a thread each
template <int NW>
__device__ __forceinline__ void xdr_threads(const KParams &kp, const char *tbl, uint32_t ntask, uint32_t first)
{
    uint32_t ta, tb;
    pg_pair pb;
    XfReady c;
    // the next direction: through the longest-first order when there is one
    constexpr uint32_t NONE = 0xffffffffu;
    auto fetch = [&]() -> uint32_t {
        const uint32_t i = first + atomicAdd(&kp.counter[1], 1u);
        return i >= ntask ? NONE : kp.xorder ? kp.xorder[i] : i;
    };
    auto load_pair = [&](uint32_t t, pg_pair &pr) {
        if (t != NONE) pr = kp.pairs[t >> 2];
    };
    auto make_ready = [&](uint32_t t, const pg_pair &pr, XfReady &x) {
        x.t = t;
        x.flags = 0;
        if (t == NONE) return;
        x.flags = XFT_VALID;
        const uint64_t r = (uint64_t)pr.row + kp.roff, cc = (uint64_t)pr.col + kp.coff;
        const int s = (int)((t >> 1) & 1);
        x.seed = s ? ((uint32_t)pr.rs1 | ((uint32_t)pr.cs1 << 16)) : ((uint32_t)pr.rs0 | ((uint32_t)pr.cs0 << 16));
        if (pr.rs1 == pr.rs0 && pr.cs1 == pr.cs0) x.flags |= XFT_SAME;
        if (pr.count < 2) x.flags |= XFT_FEW;
        if (r >= kp.nr || cc >= kp.nc) return;
        x.flags |= XFT_IDX;
        x.r0 = kp.roffs[r]; x.r1 = kp.roffs[r + 1];
        x.c0 = kp.coffs[cc]; x.c1 = kp.coffs[cc + 1];
    };
    {
        const uint32_t t0 = fetch();
        pg_pair p0;
        load_pair(t0, p0);
        make_ready(t0, p0, c);
        tb = fetch();
        load_pair(tb, pb);
        ta = fetch();
    }

    XrDirT<NW> dir;
    uint32_t task = 0;
    bool run = false;
    for (;;) {
        while (!run) {
            if (!(c.flags & XFT_VALID)) break;
            const XfReady cur = c;
            make_ready(tb, pb, c);
            tb = ta;
            load_pair(tb, pb);
            ta = fetch();
            task = cur.t;
            // (with the order every direction listed runs; the tests are for input order)
            const int s = (int)((task >> 1) & 1);
            if (!(cur.flags & XFT_IDX) || s >= kp.seed_count) continue;
            if (s == 1 && ((cur.flags & XFT_SAME) ||
                           ((kp.flags & PG_F_SKIP_SPURIOUS_SEED) && (cur.flags & XFT_FEW)))) continue;
            const uint8_t *V = kp.rseq + cur.r0, *Hs = kp.cseq + cur.c0;
            const int m = (int)(cur.r1 - cur.r0), n = (int)(cur.c1 - cur.c0);
            const int bv = min((int)(cur.seed & 0xffffu), m), bh = min((int)(cur.seed >> 16), n);
            const int ev = min((int)(cur.seed & 0xffffu) + kp.seed_len, m);
            const int eh = min((int)(cur.seed >> 16) + kp.seed_len, n);
            if (!(task & 1)) {
                run = bv > 0 && bh > 0;
                if (run) dir.init(V + bv - 1, bv, -1, Hs + bh - 1, bh, -1, kp.xg, kp.xdrop);
            } else {
                run = ev < m && eh < n;
                if (run) dir.init(V + ev, m - ev, 1, Hs + eh, n - eh, 1, kp.xg, kp.xdrop);
            }
        }
        if (!run) break;
        if (dir.step(tbl, kp.xg, kp.xdrop)) continue;
        const XdOut x = dir.finish();
        XdSide o;
        o.dv = (uint16_t)x.dv; o.dh = (uint16_t)x.dh;
        o.cells = x.ok ? x.cells : XDIR_OVF;
        kp.xdir[task] = o;
        if (!x.ok) kp.ovf[atomicAdd(&kp.counter[2], 1u)] = task;
        run = false;
    }
}

template <int NW, bool MIXED>
__global__ void __launch_bounds__(XT) k_xdr(const KParams kp)
{
    __shared__ int ssm[PG_NRES * XR_STRIDE];
    __shared__ unsigned int total, nlong;
    // where no gap fits into X a direction ends soon after its homology does, far below
    // its bound: fewer long ones, beyond three times the mean load, on half of the warps
    // (12k / 20k / 40k pairs 0.62 / 1.03 / 1.31 ms with the mean load as the line, 0.45 /
    // 0.51 / 0.95 by threads alone, 0.36 / 0.52 / 0.69 so)
    const bool narrow = MIXED && kp.xdrop < -kp.xg;
    load_sm33(ssm, kp.sm);
    if (threadIdx.x < 32) {
        // the directions listed, and the long ones among them (a prefix of the order):
        // those beyond the mean load of a thread, by the length bounds.  None where X
        // lets a band outgrow a warp's window too (X / |g| gap steps to either side)
        unsigned int t = 0, l = 0;
        float load = 0.0f;
        if (kp.xorder)
            for (int b = threadIdx.x; b < XBUCKET; b += 32) {
                t += kp.xsched[b];
                load += (float)kp.xsched[b] * xdir_bucket_len(b);
            }
        t = __reduce_add_sync(FULL, t);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) load += __shfl_xor_sync(FULL, load, o);
        const float lim = fmaxf(XDR_LONG, load / (float)(gridDim.x * blockDim.x) * (narrow ? 3.0f : 1.0f));
        if (kp.xorder && 2 * kp.xdrop <= 20 * -kp.xg)
            for (int b = threadIdx.x; b < XBUCKET; b += 32)
                if (xdir_bucket_len(b) > lim) l += kp.xsched[b];
        l = __reduce_add_sync(FULL, l);
        if (threadIdx.x == 0) { total = kp.xorder ? t : (unsigned int)(4 * kp.n); nlong = l; }
    }
    __syncthreads();
    const char *tbl = reinterpret_cast<const char *>(ssm);
    const uint32_t ntask = total, first = nlong;
    // (a loop over the two parts: with xdr_long called a second time after it, behind the
    // same test, 12k to 40k uneven pairs ran 20 to 50 % slower)
    const bool later = MIXED && (threadIdx.x >> 5) < (narrow ? XT / 64 : XT / 128);
    if constexpr (MIXED) {
        for (int part = 0; part < 2; ++part) {
            if ((part == 0) != later) xdr_long(kp, ssm, first);
            else xdr_threads<NW>(kp, tbl, ntask, first);
            __syncwarp();
        }
    } else {
        xdr_long(kp, ssm, first);
        xdr_threads<NW>(kp, tbl, ntask, first);
    }
}

// ------------------------------------------------------------- k_xd_wide
__device__ __forceinline__ XdOut xdrop_dir_any(const uint8_t *V, int nv, int vstep,
                                               const uint8_t *Hs, int nh, int hstep,
                                               const int *ssm, int g, int X, int *sring,
                                               int *gring, int gring_w)
{
    XdOut o = xdrop_dir_warp(V, nv, vstep, Hs, nh, hstep, ssm, g, X, sring, RING_W);
    if (!o.ok) o = xdrop_dir_warp(V, nv, vstep, Hs, nh, hstep, ssm, g, X, gring, gring_w);
    return o;
}

// ------------------------------------------------------------------ k_xd16
// The extension in 16-bit lanes (xdrop_dir_thread16), a task per thread run to
// its end: two band cells per instruction.
// A task whose band outgrows the ring or whose score passes SAT16 goes to the
// overflow list and k_xd_wide reruns it in 32 bits.
__global__ void __launch_bounds__(XT) k_xd16(const KParams kp)
{
    __shared__ int ssm[32 * 32];
    __shared__ uint32_t ring[3 * 8 * XT];
    load_sm(ssm, kp.sm);
    __syncthreads();
    uint32_t *base = ring + threadIdx.x;
    const uint64_t ntask = 2 * kp.n;
    unsigned long long exec = 0;
    for (;;) {
        const uint64_t task = atomicAdd(&kp.counter[1], 1u);
        if (task >= ntask) break;
        const uint64_t p = task >> 1;
        const int s = (int)(task & 1);
        const pg_pair pr = kp.pairs[p];
        XdRec rec{0, 0, 0, 0, 0u, 0u};
        const uint8_t *V, *Hs;
        int m, n;
        if (!pair_seqs(kp, pr, V, m, Hs, n)) {
            rec.flags = XF_BADIDX;
        } else if (s >= kp.seed_count ||
                   (s == 1 && (kp.flags & PG_F_SKIP_SPURIOUS_SEED) && pr.count < 2)) {
            rec.flags = XF_NONE;
        } else if (s == 1 && pr.rs1 == pr.rs0 && pr.cs1 == pr.cs0) {
            rec.flags = XF_SAME;
        } else {
            int bv, ev, bh, eh;
            if (seed_region(kp, pr, s, m, n, bv, ev, bh, eh)) rec.flags |= XF_BAD;
            bool ok = true;
            if (bv > 0 && bh > 0) {
                const XdOut x = xdrop_dir_thread16<XT>(V + bv - 1, bv, -1, Hs + bh - 1, bh, -1,
                                                       ssm, kp.xg, kp.xdrop, base);
                ok = x.ok; rec.cells += x.cells; bv -= x.dv; bh -= x.dh;
            }
            if (ok && ev < m && eh < n) {
                const XdOut x = xdrop_dir_thread16<XT>(V + ev, m - ev, 1, Hs + eh, n - eh, 1,
                                                       ssm, kp.xg, kp.xdrop, base);
                ok = x.ok; rec.cells += x.cells; ev += x.dv; eh += x.dh;
            }
            if (ok) {
                rec.bv = (uint16_t)bv; rec.ev = (uint16_t)ev; rec.bh = (uint16_t)bh; rec.eh = (uint16_t)eh;
                exec += rec.cells;
            } else {
                rec.flags |= XF_OVF;
                rec.cells = 0;
                const unsigned int slot = atomicAdd(&kp.counter[2], 1u);
                kp.ovf[slot] = (uint32_t)task;
            }
        }
        kp.xd[task] = rec;
    }
    if (exec) atomicAdd(kp.exec_cells, exec);   // index 0 = X-drop cells
}

// ------------------------------------------------------------------ k_xda
// The affine gap model of the extension (PG_F_XDROP_AFFINE): a warp per
// (pair, seed) task taken from the work counter, both directions by
// xdrop_dir_warp_affine on the warp's ring of 7 x gring_w ints in global
// memory (L2-resident; gring_w covers the longest sequence, so no band
// overflows).
__global__ void __launch_bounds__(WARPS * 32) k_xda(const KParams kp)
{
    __shared__ int ssm[32 * 32];
    load_sm(ssm, kp.sm);
    __syncthreads();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint64_t gw = (uint64_t)blockIdx.x * WARPS + wib;
    int *ring = kp.gring + gw * (uint64_t)XDA_ARRAYS * (uint64_t)kp.gring_w;
    const uint64_t ntask = 2 * kp.n;
    unsigned long long exec = 0;
    for (;;) {
        unsigned int tk = 0;
        if (lane == 0) tk = atomicAdd(&kp.counter[1], 1u);
        const uint64_t task = __shfl_sync(FULL, tk, 0);
        if (task >= ntask) break;
        const uint64_t p = task >> 1;
        const int s = (int)(task & 1);
        const pg_pair pr = kp.pairs[p];
        XdRec rec{0, 0, 0, 0, 0u, 0u};
        const uint8_t *V, *Hs;
        int m, n;
        if (!pair_seqs(kp, pr, V, m, Hs, n)) {
            rec.flags = XF_BADIDX;
        } else if (s >= kp.seed_count ||
                   (s == 1 && (kp.flags & PG_F_SKIP_SPURIOUS_SEED) && pr.count < 2)) {
            rec.flags = XF_NONE;
        } else if (s == 1 && pr.rs1 == pr.rs0 && pr.cs1 == pr.cs0) {
            rec.flags = XF_SAME;
        } else {
            int bv, ev, bh, eh;
            if (seed_region(kp, pr, s, m, n, bv, ev, bh, eh)) rec.flags |= XF_BAD;
            if (bv > 0 && bh > 0) {
                const XdOut x = xdrop_dir_warp_affine(V + bv - 1, bv, -1, Hs + bh - 1, bh, -1, ssm,
                                                      kp.go, kp.ge, kp.xdrop, ring, kp.gring_w);
                rec.cells += x.cells;
                bv -= x.dv; bh -= x.dh;
            }
            if (ev < m && eh < n) {
                const XdOut x = xdrop_dir_warp_affine(V + ev, m - ev, 1, Hs + eh, n - eh, 1, ssm,
                                                      kp.go, kp.ge, kp.xdrop, ring, kp.gring_w);
                rec.cells += x.cells;
                ev += x.dv; eh += x.dh;
            }
            rec.bv = (uint16_t)bv; rec.ev = (uint16_t)ev; rec.bh = (uint16_t)bh; rec.eh = (uint16_t)eh;
            exec += rec.cells;
        }
        if (lane == 0) kp.xd[task] = rec;
        __syncwarp();
    }
    if (lane == 0 && exec) atomicAdd(kp.exec_cells, exec);
}

// The (pair, seed) records from k_xdr's directions: first the tasks with a direction
// that outgrew its window (listed by direction in kp.ovf), a warp each, then the
// rest, a lane each.
__device__ __forceinline__ void xd_join(const KParams &kp, const int *ssm, int *sring, int *gring,
                                        uint64_t gw, uint64_t nw)
{
    const int lane = threadIdx.x & 31;
    const uint64_t ntask = 2 * kp.n;
    const uint32_t novf = kp.counter[2];
    unsigned long long exec = 0;
    auto load = [&](uint64_t task, XdRec &rec, const uint8_t *&V, int &m, const uint8_t *&Hs, int &n, int &bv,
                    int &ev, int &bh, int &eh, XdSide &a, XdSide &b) {
        const pg_pair pr = kp.pairs[task >> 1];
        a = b = XdSide{0, 0, 0u};
        bv = ev = bh = eh = 0;
        if (!pair_seqs(kp, pr, V, m, Hs, n)) { rec.flags = XF_BADIDX; return; }
        rec.flags = xd_seed(kp, pr, (int)(task & 1), m, n, bv, ev, bh, eh);
        if (rec.flags & (XF_NONE | XF_SAME)) return;
        if (bv > 0 && bh > 0) a = kp.xdir[2 * task];
        if (ev < m && eh < n) b = kp.xdir[2 * task + 1];
    };
    for (;;) {
        uint32_t q = 0;
        if (lane == 0 && novf) q = atomicAdd(&kp.xsched[2 * XBUCKET + 1], 1u);
        q = __shfl_sync(FULL, q, 0);
        if (q >= novf) break;
        const uint32_t id = kp.ovf[q];
        const uint64_t task = id >> 1;
        XdRec rec{0, 0, 0, 0, 0u, 0u};
        const uint8_t *V, *Hs;
        int m, n, bv, ev, bh, eh;
        XdSide a, b;
        load(task, rec, V, m, Hs, n, bv, ev, bh, eh, a, b);
        const bool wl = (a.cells & XDIR_OVF) != 0, wr = (b.cells & XDIR_OVF) != 0;
        if ((id & 1) && wl) continue;                // its other direction's entry does both
        if (wl) {
            const XdOut x = xdrop_dir_any(V + bv - 1, bv, -1, Hs + bh - 1, bh, -1, ssm, kp.xg, kp.xdrop,
                                          sring, gring, kp.gring_w);
            a.dv = (uint16_t)x.dv; a.dh = (uint16_t)x.dh; a.cells = x.cells;
        }
        if (wr) {
            const XdOut x = xdrop_dir_any(V + ev, m - ev, 1, Hs + eh, n - eh, 1, ssm, kp.xg, kp.xdrop,
                                          sring, gring, kp.gring_w);
            b.dv = (uint16_t)x.dv; b.dh = (uint16_t)x.dh; b.cells = x.cells;
        }
        rec.bv = (uint16_t)(bv - a.dv); rec.bh = (uint16_t)(bh - a.dh);
        rec.ev = (uint16_t)(ev + b.dv); rec.eh = (uint16_t)(eh + b.dh);
        rec.cells = a.cells + b.cells;
        if (lane == 0) { kp.xd[task] = rec; exec += rec.cells; }
    }
    for (uint64_t task = gw * 32 + lane; task < ntask; task += nw * 32) {
        XdRec rec{0, 0, 0, 0, 0u, 0u};
        const uint8_t *V, *Hs;
        int m, n, bv, ev, bh, eh;
        XdSide a, b;
        load(task, rec, V, m, Hs, n, bv, ev, bh, eh, a, b);
        if ((a.cells | b.cells) & XDIR_OVF) continue;
        rec.bv = (uint16_t)(bv - a.dv); rec.bh = (uint16_t)(bh - a.dh);
        rec.ev = (uint16_t)(ev + b.dv); rec.eh = (uint16_t)(eh + b.dh);
        rec.cells = a.cells + b.cells;
        kp.xd[task] = rec;
        exec += rec.cells;
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) exec += __shfl_xor_sync(FULL, exec, o);
    if (lane == 0 && exec) atomicAdd(kp.exec_cells, exec);
}

__global__ void __launch_bounds__(WARPS * 32) k_xd_wide(const KParams kp)
{
    __shared__ int ssm[32 * 32];
    __shared__ int sring[WARPS][3 * RING_W];
    load_sm(ssm, kp.sm);
    __syncthreads();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint64_t gw = (uint64_t)blockIdx.x * WARPS + wib;
    const uint64_t nw = (uint64_t)gridDim.x * WARPS;
    int *gring = kp.gring + gw * 3ull * (uint64_t)kp.gring_w;
    if (kp.xdir) { xd_join(kp, ssm, sring[wib], gring, gw, nw); return; }
    const unsigned int novf = kp.counter[2];
    unsigned long long exec = 0;
    for (uint64_t q = gw; q < novf; q += nw) {
        const uint32_t task = kp.ovf[q];
        const uint64_t p = task >> 1;
        const int s = (int)(task & 1);
        const pg_pair pr = kp.pairs[p];
        const uint8_t *V, *Hs;
        int m, n;
        pair_seqs(kp, pr, V, m, Hs, n);
        XdRec rec{0, 0, 0, 0, 0u, 0u};
        int bv, ev, bh, eh;
        if (seed_region(kp, pr, s, m, n, bv, ev, bh, eh)) rec.flags |= XF_BAD;
        if (bv > 0 && bh > 0) {
            const XdOut x = xdrop_dir_any(V + bv - 1, bv, -1, Hs + bh - 1, bh, -1, ssm, kp.xg,
                                          kp.xdrop, sring[wib], gring, kp.gring_w);
            rec.cells += x.cells;
            bv -= x.dv; bh -= x.dh;
        }
        if (ev < m && eh < n) {
            const XdOut x = xdrop_dir_any(V + ev, m - ev, 1, Hs + eh, n - eh, 1, ssm, kp.xg,
                                          kp.xdrop, sring[wib], gring, kp.gring_w);
            rec.cells += x.cells;
            ev += x.dv; eh += x.dh;
        }
        rec.bv = (uint16_t)bv; rec.ev = (uint16_t)ev; rec.bh = (uint16_t)bh; rec.eh = (uint16_t)eh;
        exec += rec.cells;
        if (lane == 0) kp.xd[task] = rec;
    }
    if (lane == 0 && exec) atomicAdd(kp.exec_cells, exec);
}

}  // namespace pg
