// pg_dptag.cuh -- the affine traceback-form DP with the decisions in the values
// (sm_103a).
//
// dp_warp_dir16 and dp_pair_dir16 (pg_dpdir16.cuh) find a cell's decisions by
// comparing the packed values again, 17 ALU operations per row and two cells.
// Here values are scaled by 4 and a decision rides in the two low bits, as in
// the linear form (pg_lin.cuh): a maximum then picks the larger value and on a
// tie the preferred source, and says which it was.  E and F are kept less the
// first gap score (E~ = E - go), so that each is one DPX add-max:
//     E~'= max(E~ + ge [+ tag], H)         bit 0: extended or opened
//     X  = max(E~' + go + tag, diag + tag)
//     H  = max(F~' + go + tag, X [, 0])    bits 1-0: diagonal, E or F
// Stored H carries the tag that an opened gap has (the logic operation that
// clears H sets it at no cost).  Per row and two cells: prmt, add, four add-max,
// three logic operations, 9 on the ALU pipe, which bounds the DP (two cycles a
// warp instruction); the tags are gathered by six multiply-adds on the FMA pipe
// (sums of the tagged less the cleared values).
//
// Scaled values: H of a region lies between -(2 |go| + (m + n) |max(go, ge)|)
// (global, a path of gaps; local: 0) and smax min(m, n).  tag_sum and tag_min
// (pg_api.cu) are the m + n and min(m, n) up to which these, times 4, fit int16.
// A whole-warp region past tag_min, up to tag_try, runs too, keeps its largest H and
// reports sat when that left the range.  Those and the larger ones run in a pass of
// their own with BASE: a lane's values are relative to a base that follows them (moved
// every 32 steps, as in lin_stripe), so that no region is too large and none is done
// on wider lanes.  Without it long homologs ran here to the end and then once more
// through the checked form: uneven Smith-Waterman batches of 1000 and 6000 pairs took
// 32.9 and 38.6 ms, 23.4 and 31.8 by the checked form alone, 16.1 and 21.2 so (X-drop
// 41.6 and 48.4, 32.0 and 35.0 so).
// The words' layout is that of the untagged forms.
//
// Measured (k_sw_dir, 40k Smith-Waterman pairs of 250 residues, gaps -11 / -2):
// 3.15 -> 2.28 ms, 0.77 instructions issued a cycle and scheduler, the ALU pipe
// busy three quarters of the time.
#pragma once
#include <cstdint>

#include "pg_lin.cuh"

namespace pg {

constexpr int TAG_SMAX = 31;                       // 4 * 31 + 3 fits the int8 profile
constexpr int TAG_MAX = 31000;                     // scaled H provably up to here

// what the tagged form adds to a diagonal term besides 4 s: its tag (the largest
// of the three) less the one its H carries
template <int TIE>
__host__ __device__ __forceinline__ constexpr int tag_diag()
{
    return ((TIE & TIE_E_BEFORE_F) ? 2 : 3) - ((TIE & TIE_OPEN_FIRST) ? 1 : 0);
}

template <int TIE>
__device__ __forceinline__ void tag_table(int8_t *t, const int8_t *sm)
{
    for (int k = threadIdx.x; k < LIN_NC * LIN_ROWB; k += blockDim.x) {
        const int a = k / LIN_ROWB, b = k - a * LIN_ROWB;
        t[k] = a < PG_NRES && b < PG_NRES ? (int8_t)(4 * (int)sm[a * PG_NRES + b] + tag_diag<TIE>()) : (int8_t)-128;
    }
}

// L = 32: a region on a warp, in stripes of 64 R rows; L = 16: each half of the
// warp its own region of at most 32 R rows (m = 0: none).  prof: this warp's
// profile; bnd: its row scratch (L = 32, n + 1 entries); four: a 4 the compiler
// cannot see, so that the multiply-adds stay on the FMA pipe.  The result is
// that of the lane's region.
template <int TIE, int R, bool LOCAL, int L, bool BASE>
__device__ DirOut dp_tag16(const uint8_t *__restrict__ V, int m, const uint8_t *__restrict__ Hs, int n,
                           const uint32_t *tab, uint32_t *prof, int go, int ge, uint32_t four,
                           uint2 *__restrict__ bnd, uint32_t *__restrict__ dir)
{
    static_assert(R >= 1 && R <= 8 && (L == 32 || L == 16), "a direction word holds 8 rows");
    static_assert(!BASE || L == 32, "lanes with a base have a warp");
    constexpr bool E_FIRST = (TIE & TIE_E_BEFORE_F) != 0, OPEN_FIRST = (TIE & TIE_OPEN_FIRST) != 0;
    constexpr int BH = OPEN_FIRST ? 1 : 0;         // the tag stored H carries
    constexpr uint32_t BH2 = BH * ONE2;
    constexpr bool TRACK = LOCAL || (L == 32 && !BASE);
    constexpr int NG = (R + 3) / 4;
    // nibble: bit 0 E rather than F, bit 1 not the diagonal, bits 2, 3 opened
    constexpr uint32_t FLIP = 0x11111111u * ((E_FIRST ? 2u : 3u) | (OPEN_FIRST ? 0u : 12u));
    constexpr uint32_t NEG2 = (uint32_t)(NEG16 & 0xffff) * ONE2;
    const int lane = threadIdx.x & 31, sl = lane & (L - 1);
    const int gmax = go > ge ? go : ge;
    const int te = E_FIRST ? 1 : 0;
    const uint32_t geT = pk16(4 * ge + 1 - BH, 4 * ge + 1 - BH);
    const uint32_t goE = pk16(4 * go + te, 4 * go + te), goF = pk16(4 * go + 1 - te, 4 * go + 1 - te);
    const uint32_t c4 = four, c8 = four + four;
    const uint32_t mul[4] = {1u, four * four, four * four * four * four, four * four * four * four * four * four};
    const bool has = m > 0 && n > 0;
    // scaled H and F~ of row i in column 0
    auto h0 = [&](int i) { return (LOCAL || i == 0 ? 0 : 4 * (go + (i - 1) * gmax)) + BH; };
    auto f0 = [&](int i) { return LOCAL || i == 0 ? NEG16 : 4 * (i - 1) * gmax; };
    int bs = 0, bi = 0, bj = 0;
    int score = 0;
    uint32_t top = 0;                              // largest stored H (TRACK)
    const int m_all = L == 32 ? m : 1;
    for (int rb = 0, stripe = 0; rb < m_all; rb += 64 * R, ++stripe) {
        const int rows = L == 32 ? min(64 * R, m - rb) : m;
        const int v_last = has ? (rows - 1) / R : -1;
        const int t_last = v_last >> 1;
        const bool last_block = L == 16 || rb + rows >= m;
        const bool on = has && sl <= t_last;
        const int hi_on = 2 * sl + 1 <= v_last ? 1 : 0;
        const int i_base = rb + 2 * sl * R;        // row above the low half
        const int own = has ? n + v_last : 0;
        const unsigned lim = on ? (unsigned)(n + hi_on) : 0u;
        __syncwarp();
        lin_profile<R>(tab, V, i_base, m, on, prof);
        __syncwarp();
        // column 0 of the low half's rows, column -1 (sentinels) of the high half's.  BASE:
        // less B, a multiple of 4, which puts the row above the lane's first at LIN_MID
        uint32_t H[R], E[R], S[R];
        const int iu = min(i_base, m), il = min(i_base + R, m), ih = min(i_base + 2 * R, m);
        int B = BASE ? h0(iu) - BH - LIN_MID : 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            H[r] = pk16(h0(min(i_base + r + 1, m)) - B, NEG16);
            E[r] = NEG2;
            S[r] = 0;
        }
        auto fb = [&](int i) { return BASE && !(LOCAL || i == 0) ? f0(i) - B : f0(i); };
        uint32_t in_h = pk16(h0(iu) - B, h0(il) - B), out_h = pk16(h0(il) - B, h0(ih) - B);
        uint32_t in_f = pk16(fb(iu), fb(il)), out_f = pk16(fb(il), fb(ih));
        // H(0, j) of the first lane, in the high half
        uint32_t bord = (uint32_t)(LOCAL ? BH : 4 * go + BH) << 16;
        const uint32_t bstep = LOCAL ? 0u : (uint32_t)(4 * gmax) << 16;
        uint2 brow = make_uint2(0u, 0u);           // 32 columns of the row above the stripe
        uint32_t floor2 = 0u, d2 = 0u;             // BASE: 0, and what a value from the lane above gains
        int top0 = BH, top1 = BH;                  // BASE: largest stored H of the halves, whole
        LinCols cols;
        cols.init(Hs, has ? n : 0, -2 * sl);
        const char *lbase = reinterpret_cast<const char *>(prof + lane * NG);
        const char *pa = lbase + PG_NRES * (128 * NG);
        uint32_t sbs = on ? BH2 : 0x7fff7fffu, seen = sbs, sj = 0;
        const int nsteps = L == 32 ? own : max(own, __shfl_xor_sync(FULL, own, 16));
        uint4 *dst = reinterpret_cast<uint4 *>(dir) +
                     (size_t)stripe * (size_t)(dir16_steps(n) >> 2) * (2 * L) + sl * 2;
        // one column of the lane's 2R rows; returns its direction words
        auto rows_of = [&](const uint32_t dgH, const uint32_t code) {
            const char *ph = pa + LIN_NC * (128 * NG);
            pa = lbase + code * (128 * NG);
            uint32_t lo[NG], hi[NG];
            if (NG == 2) {
                const uint2 a = *reinterpret_cast<const uint2 *>(pa), b = *reinterpret_cast<const uint2 *>(ph);
                lo[0] = a.x; lo[NG - 1] = a.y; hi[0] = b.x; hi[NG - 1] = b.y;
            } else {
                lo[0] = *reinterpret_cast<const uint32_t *>(pa);
                hi[0] = *reinterpret_cast<const uint32_t *>(ph);
            }
            uint32_t wt[2] = {0u, 0u}, wc[2] = {0u, 0u};   // sums of the tagged and of the cleared values
            uint32_t dH = dgH, cH = in_h, cF = in_f;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int g = r >> 2, q = r & 3;
                uint32_t dg = v16add(dH, prmt(lo[g], hi[g], sx_sel(q)));
                if (LOCAL && BASE) dg = v16max(dg, floor2);
                const uint32_t et = __viaddmax_s16x2(E[r], geT, H[r]);
                const uint32_t ec = et & LIN_CLR;
                const uint32_t x = __viaddmax_s16x2(ec, goE, dg);
                const uint32_t ft = __viaddmax_s16x2(cF, geT, cH);
                const uint32_t fc = ft & LIN_CLR;
                const uint32_t ht = LOCAL && !BASE ? __viaddmax_s16x2_relu(fc, goF, x) : __viaddmax_s16x2(fc, goF, x);
                const uint32_t hc = (ht & LIN_CLR) | BH2;
                const uint32_t a = ft * c8 + (et * c4 + ht), b = fc * c8 + (ec * c4 + hc);
                if (q == 0) { wt[g] = a; wc[g] = b; }
                else { wt[g] = a * mul[q] + wt[g]; wc[g] = b * mul[q] + wc[g]; }
                dH = H[r];
                H[r] = hc; E[r] = ec; cH = hc; cF = fc;
            }
            out_h = cH;
            out_f = cF;
            if (TRACK) sbs = lin_max<R>(sbs, H);
            // cleared H carries BH: add it back to each nibble
            const uint32_t W0 = (wt[0] - wc[0] + BH * 0x11111111u) ^ FLIP;
            const uint32_t W1 = R > 4 ? (wt[1] - wc[1] + BH * 0x11111111u) ^ FLIP : 0u;
            return make_uint2(prmt(W0, W1, 0x5410u), prmt(W0, W1, 0x7632u));
        };
        // Two steps a turn, each lane tested at each: the warps of an SM are at
        // different row counts, and with four steps a turn, or with a copy of the
        // steps that need no test, their loops together outgrew the instruction
        // cache (40k Smith-Waterman pairs: 4.2 ms with both, three of four issue
        // slots lost to it; one step a turn with both copies 2.5; two steps, one
        // copy 2.3)
        uint32_t res4 = 0;
        for (int k0 = 0; k0 < nsteps; k0 += 2) {
            if (BASE && (k0 & 31) == 0) {
                // move the base of the lanes whose two halves hold real columns
                const int sh = k0 - 1 - 2 * sl >= 1 ? (lo16(H[0]) & ~3) - LIN_MID : 0;
                const uint32_t s2 = pk16(-sh, -sh);
                if (LOCAL) {
                    top0 = max(top0, lo16(sbs) + B);
                    top1 = max(top1, hi16(sbs) + B);
                }
                B += sh;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    H[r] = v16add(H[r], s2);
                    E[r] = v16add(E[r], s2);
                    if (LOCAL) S[r] = v16add(S[r], s2);    // modulo 2^16
                }
                in_h = v16add(in_h, s2);
                out_h = v16add(out_h, s2);
                in_f = v16add(in_f, s2);
                out_f = v16add(out_f, s2);
                if (LOCAL) {
                    const int f = max(-B, NEG16);
                    floor2 = pk16(f, f);
                    // the maximum so far, as far as the new base can tell it: past int16 no
                    // value of the next 32 columns reaches it
                    if (on) sbs = seen = pk16(min(max(top0 - B, NEG16), 32767), min(max(top1 - B, NEG16), 32767));
                }
                d2 = pk16(0, __shfl_up_sync(FULL, B, 1) - B);
                const int b0 = __shfl_sync(FULL, B, 0);
                if (rb > 0) {
                    // (past the last column, where the low half's step is in vain: far below)
                    brow = make_uint2(0u, 0u);
                    if (k0 + lane + 1 <= n) {
                        brow = bnd[k0 + lane + 1];
                        brow = make_uint2((brow.x - (uint32_t)b0) << 16, (brow.y - (uint32_t)b0) << 16);
                    }
                } else {
                    bord = (uint32_t)(LOCAL ? BH - b0 : 4 * (go + k0 * gmax) + BH - b0) << 16;
                }
            }
            if (!BASE && L == 32 && rb > 0 && (k0 & 31) == 0 && k0 + lane + 1 <= n) brow = bnd[k0 + lane + 1];
            if ((k0 & 3) == 0) res4 = cols.next();
            else res4 >>= 16;
            uint2 w[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int k = k0 + s;
                uint32_t rh = __shfl_up_sync(FULL, out_h, 1, L), rf = __shfl_up_sync(FULL, out_f, 1, L);
                if (BASE) { rh = v16add(rh, d2); rf = v16add(rf, d2); }
                const uint32_t dgH = in_h;
                uint32_t bh = bord, bf = NEG2;
                if (L == 32 && rb > 0) {
                    bh = __shfl_sync(FULL, brow.x, k & 31);
                    bf = __shfl_sync(FULL, brow.y, k & 31);
                }
                bord += bstep;
                in_h = prmt(sl == 0 ? bh : rh, out_h, 0x5432u);
                in_f = prmt(sl == 0 ? bf : rf, out_f, 0x5432u);
                w[s] = make_uint2(0u, 0u);
                if ((unsigned)(k - 2 * sl) < lim) {
                    w[s] = rows_of(dgH, (res4 >> (8 * s)) & 0xffu);
                    const int j = k - 2 * sl + 1;  // low half's column; high half: j - 1
                    // the row under the stripe (a stripe with one below it has all
                    // its rows): its last lane's high half
                    if (L == 32 && !last_block && lane == 31 && j >= 2 && j <= n + 1)
                        bnd[j - 1] = BASE ? make_uint2((uint32_t)(hi16(out_h) + B), (uint32_t)(hi16(out_f) + B))
                                          : make_uint2(out_h, out_f);
                    if (LOCAL && sbs != seen) {
                        // a half's maximum rose: keep its rows and the column
                        const uint32_t mask = v16ne(sbs, seen) * 0xffffu;
#pragma unroll
                        for (int r = 0; r < R; ++r) S[r] = (H[r] & mask) | (S[r] & ~mask);
                        sj = (pk16(j, j - 1) & mask) | (sj & ~mask);
                        seen = sbs;
                    }
                }
            }
            if (on && k0 < own)
                dst[(size_t)(k0 >> 2) * (2 * L) + ((k0 >> 1) & 1)] = make_uint4(w[0].x, w[0].y, w[1].x, w[1].y);
        }
        __syncwarp();
        if (TRACK && !BASE && on) top = v16max(top, sbs);
        if (LOCAL && on) {
            // first maximum in column-major order: the low half's rows before the
            // high half's in a column; against earlier stripes a tie goes to the
            // smaller column
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int st = BASE ? max(h ? top1 : top0, half16(sbs, h) + B) : half16(sbs, h);
                const int s = st >> 2, c = (int)(h ? sj >> 16 : sj & 0xffffu);
                if (s > 0 && (s > bs || (s == bs && c < bj))) {
                    int rr = R - 1;
#pragma unroll
                    for (int r = R - 1; r >= 0; --r)
                        if (((half16(S[r], h) ^ (st - B)) & 0xffff) == 0) rr = r;
                    bs = s; bj = c; bi = i_base + h * R + rr + 1;
                }
            }
        }
        if (!LOCAL && last_block) {
            const int rl = has ? (rows - 1) % R : -1, h = v_last & 1;
            int hs = 0;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r == rl) hs = half16(H[r], h) + B;
            score = __shfl_sync(FULL, hs, (lane & ~(L - 1)) + (t_last > 0 ? t_last : 0)) >> 2;
        }
    }
    DirOut res;
    res.have = 0; res.ei = 0; res.ej = 0; res.score = score;
    if (LOCAL) {
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) {
            const int os = __shfl_xor_sync(FULL, bs, o);
            const int oi = __shfl_xor_sync(FULL, bi, o);
            const int oj = __shfl_xor_sync(FULL, bj, o);
            const bool take = os > bs || (os == bs && (oj < bj || (oj == bj && oi < bi)));
            if (take) { bs = os; bi = oi; bj = oj; }
        }
        res.score = bs;
        res.have = bs > 0;
        res.ei = bi; res.ej = bj;
    }
    if (L == 32 && !BASE) res.sat = __any_sync(FULL, lo16(top) > SAT16_DP || hi16(top) > SAT16_DP) ? 1 : 0;
    return res;
}

}  // namespace pg
