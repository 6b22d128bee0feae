// pg_kmer.cu -- candidate generation on the GPU: the k-mer SpGEMM C = A·Aᵀ of
// PASTIS (src/kmer/KmerOps.cpp:31-245, src/sim_search.cpp:154-187) with the
// KmerIntersectLoc semiring (inc/sr.hpp:30-117), restated as sort and join.
//
//   1. k-mers of every row sequence of the block: code over the alphabet
//      (Horner, base = alphabet size, as KmerOps.cpp:60-62), offset; one warp per
//      sequence, lanes across positions.
//   2. radix sort of the row occurrences by a bijection of the code (a
//      multiplication modulo a power of two, so that a table indexed by its top
//      bits is evenly filled), and that table: first occurrence of each value.
//   3. a block per column sequence: each of its k-mers finds its run of equal
//      codes on the row side through the table; the occurrence pairs that survive
//      the symmetric prune are counted per row in a hash table in shared memory.
//      The rows whose count passes ckthr (few from ckthr = 1 on: most pairs share one
//      k-mer by chance) get their first / second seed (smallest / largest seed value) and
//      score (largest k-mer self score) in a second sweep over the same runs, are
//      ranked by row and written out.
//   4. the columns' records are moved into place, column-major.
// The product of a block is never written out or sorted: for 200k proteins that
// was 58M 16-byte products through a 7-pass radix sort, a run-length encoding and
// a reduction, 28.5 ms a call with the allocation of their buffers; 10.3 ms now (even/odd
// prune, ckthr = 1).  A column that outgrows the tables of step 3, the usual one without
// a threshold (ckthr = 0) or from about 500k rows on, goes through k_cand_parts.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "../../include/pastis_gb300.h"

int pg_internal_seqs(const pg_ctx *c, const uint8_t **rseq, const uint64_t **roffs, uint64_t *nr,
                     const uint8_t **cseq, const uint64_t **coffs, uint64_t *nc, int *device,
                     void **stream, int *mode);
int pg_internal_fail(int code, const char *msg);
int pg_internal_score(const pg_ctx *c, const int8_t **d_sm);
int pg_internal_pool(pg_ctx *c, cudaMemPool_t *pool);

namespace {

#define KCU(call)                                                                  \
    do {                                                                           \
        cudaError_t e_ = (call);                                                   \
        if (e_ != cudaSuccess)                                                     \
            return pg_internal_fail(e_ == cudaErrorMemoryAllocation ? PG_ERR_OOM : PG_ERR_CUDA, \
                                    cudaGetErrorString(e_));                       \
    } while (0)

// murphy10 code of each residue code (ARNDCQEGHILKMFPSTWYVBZX*J): codes in the
// order Alphabet::init assigns them (src/Alphabet.cpp:31-51) to the groups of
// inc/Alphabet.hpp:83-104; the representative residue of each murphy10 code.
constexpr uint8_t kMurphy[PG_NRES] = {0, 1, 2, 2, 3, 2, 2, 4, 5, 6, 6, 1, 6, 7, 8, 9, 9, 7, 7, 6,
                                      10, 11, 12, 13, 14};
constexpr uint8_t kMurphyRep[15] = {0, 11, 3, 4, 7, 8, 9, 13, 14, 15, 20, 21, 22, 23, 24};

struct KmerTab {
    uint8_t map[32];     // residue code -> alphabet code
    int16_t cost[32];    // alphabet code -> self score of its letter
    uint32_t base;
    int k;
    int bits;            // of the k-mer universe
};

// the bijection of a code the row side is sorted by
__device__ __forceinline__ uint32_t kmer_mix(uint32_t code, int bits)
{
    return (code * 0x9E3779B1u) & (bits < 32 ? (1u << bits) - 1u : 0xffffffffu);
}

// k-mers of sequences [s0, s0 + ns) of one side; one warp per sequence
__global__ void k_kmer_fill(const uint8_t *seq, const uint64_t *offs, uint64_t s0, uint64_t ns,
                            int stride, const uint64_t *start, KmerTab tab, uint32_t *codes,
                            uint64_t *vals)
{
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    for (uint64_t s = warp; s < ns; s += nwarps) {
        const uint64_t b = offs[s0 + s];
        const int len = (int)(offs[s0 + s + 1] - b);
        if (len < tab.k) continue;
        const int nk = (len - tab.k) / stride + 1;
        const uint64_t o = start[s];
        for (int q = lane; q < nk; q += 32) {
            const int pos = q * stride;
            uint32_t code = 0;
            for (int j = 0; j < tab.k; ++j) code = code * tab.base + tab.map[seq[b + pos + j] & 31];
            codes[o + q] = kmer_mix(code, tab.bits);
            vals[o + q] = (s << 16) | (uint64_t)pos;
        }
    }
}

__global__ void k_kmer_count(const uint64_t *offs, uint64_t s0, uint64_t ns, int k, int stride,
                             uint64_t *cnt)
{
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < ns;
         s += (uint64_t)gridDim.x * blockDim.x) {
        const int len = (int)(offs[s0 + s + 1] - offs[s0 + s]);
        cnt[s] = len < k ? 0 : (uint64_t)((len - k) / stride + 1);
    }
}

// PG_PRUNE_* on global indices (sim_search.cpp:172-186 and :403-412)
__device__ __forceinline__ bool keep_pair(int prune, uint64_t r, uint64_t c)
{
    if (prune == PG_PRUNE_EVEN_ODD) {
        if (r == c) return false;
        const bool odd = ((r ^ c) & 1) != 0;
        return r > c ? !odd : odd;
    }
    if (prune == PG_PRUNE_UPPER) return r < c;
    return true;
}

// the distinct values of the sorted codes: their number per block of RB codes,
// then (after a scan of those) their value and first occurrence (one entry more:
// the end), for each value of their top bits the first distinct one (table, ~0:
// none), and the occurrences' rows and offsets in arrays of their own (the sweeps
// over a run read rows only)
constexpr int RB = 2048;
template <class I>
struct KmerRun {
    uint32_t h;
    I start;
};
__global__ void __launch_bounds__(256) k_runs_count(const uint32_t *h, uint64_t n, uint32_t *cnt)
{
    const uint64_t i0 = (uint64_t)blockIdx.x * RB;
    uint32_t c = 0;
    for (uint64_t i = i0 + threadIdx.x; i < min(i0 + RB, n); i += 256)
        c += i == 0 || h[i - 1] != h[i] ? 1u : 0u;
    c = __reduce_add_sync(0xffffffffu, c);
    __shared__ uint32_t w[8];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) c += w[k];
        cnt[blockIdx.x] = c;
    }
}
template <class I>
__global__ void __launch_bounds__(256) k_runs_write(const uint32_t *h, const uint64_t *val, uint64_t n,
                                                    const uint64_t *first, int shift, KmerRun<I> *run, I *table,
                                                    uint32_t *rrow, uint16_t *rpos)
{
    __shared__ uint32_t w[8];
    const uint64_t i0 = (uint64_t)blockIdx.x * RB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t o = first[blockIdx.x];
    for (uint64_t q = i0; q < min(i0 + RB, n); q += 256) {
        const uint64_t i = q + threadIdx.x;
        const uint32_t v = i < n ? h[i] : 0u, u = i < n && i ? h[i - 1] : 0u;
        const bool head = i < n && (i == 0 || u != v);
        const uint32_t m = __ballot_sync(0xffffffffu, head);
        if (lane == 0) w[warp] = (uint32_t)__popc(m);
        __syncthreads();
        uint32_t before = 0, all = 0;
        for (int k = 0; k < 8; ++k) { before += k < warp ? w[k] : 0u; all += w[k]; }
        if (head) {
            const uint64_t x = o + before + (uint32_t)__popc(m & ((1u << lane) - 1u));
            run[x] = KmerRun<I>{v, (I)i};
            if (i == 0 || (u >> shift) != (v >> shift)) table[v >> shift] = (I)x;
        }
        if (i < n) {
            const uint64_t rv = val[i];
            rrow[i] = (uint32_t)(rv >> 16);
            rpos[i] = (uint16_t)rv;
        }
        if (i == n - 1) run[o + all] = KmerRun<I>{0u, (I)n};
        o += all;
        __syncthreads();
    }
}

// the run of each column k-mer on the row side (length 0: none), in the order of
// the columns; a warp per column, lanes across positions.  own: the columns are the
// rows and a k-mer of its own sequence alone makes no pair.  nu: the distinct values;
// bound: the sum of the lengths, the block's occurrence pairs before the prune.
template <class I>
__global__ void k_col_runs(const uint8_t *seq, const uint64_t *offs, uint64_t s0, uint64_t ns, int stride,
                           const uint64_t *kstart, KmerTab tab, const I *table, int shift, const KmerRun<I> *run,
                           const uint64_t *nu_, bool own, I *first, I *len, unsigned long long *bound)
{
    __shared__ uint8_t map[32];
    if (threadIdx.x < 32) map[threadIdx.x] = tab.map[threadIdx.x];
    __syncthreads();
    const uint64_t nu = *nu_;
    unsigned long long sum = 0;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    for (uint64_t s = warp; s < ns; s += nwarps) {
        const uint64_t b = offs[s0 + s], o = kstart[s];
        const int nk = (int)(kstart[s + 1] - o);
        for (int q = lane; q < nk; q += 32) {
            const uint8_t *p = seq + b + (uint64_t)q * (uint64_t)stride;
            uint32_t code = 0;
            for (int j = 0; j < tab.k; ++j) code = code * tab.base + map[__ldg(p + j) & 31];
            const uint32_t h = kmer_mix(code, tab.bits);
            I lo = 0, hi = 0;
            const I t = __ldg(table + (h >> shift));
            if (t != (I)~(I)0) {
                uint64_t u = t;
                KmerRun<I> e = run[u];
                while (e.h < h && ++u < nu) e = run[u];
                if (u < nu && e.h == h) { lo = e.start; hi = run[u + 1].start; }
            }
            if (own && hi - lo == 1) hi = lo;
            first[o + q] = lo;
            len[o + q] = hi - lo;
            sum += hi - lo;
        }
    }
    __syncwarp();
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (lane == 0 && sum) atomicAdd(bound, sum);
}

// first index of run [lo, hi) whose row is r or more (rows ascend within a run: the
// occurrences were written by sequence and the sort is stable)
template <class I>
__device__ __forceinline__ I run_split(const uint32_t *rrow, I lo, I hi, uint64_t r)
{
    while (lo < hi) {
        const I mid = lo + ((hi - lo) >> 1);
        if (__ldg(rrow + mid) < r) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// 1 for the occurrences of odd rows (counted from the set's first), and a 0 at the end
template <class I>
__global__ void k_odd_rows(const uint32_t *rrow, uint64_t n, uint64_t row_begin, I *odd)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += (uint64_t)gridDim.x * blockDim.x)
        odd[i] = i < n ? (I)((rrow[i] + row_begin) & 1) : (I)0;
}

// The block's occurrence pairs after the prune, without a visit to each: from where
// the column stands in each of its runs and, for the even/odd prune, the odd rows
// before every occurrence (before: their exclusive prefix sum).  A block of a few
// hundred low-complexity sequences has 1e11 pairs, which must be refused and not
// walked.  The upper prune keeps the front of a run, which becomes its length.
template <class I>
__global__ void k_pairs_count(uint64_t col_begin, uint64_t ns, uint64_t row_begin, int prune, const uint64_t *kstart,
                              const uint32_t *rrow, const I *before, const I *first, I *len, unsigned long long *tot)
{
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    unsigned long long sum = 0;
    for (uint64_t c = warp; c < ns; c += nwarps) {
        const uint64_t gc = c + col_begin, o = kstart[c];
        const uint64_t at = gc > row_begin ? gc - row_begin : 0;       // the row below which r < c
        for (uint64_t x = o + lane; x < kstart[c + 1]; x += 32) {
            const I lo = first[x], hi = lo + len[x];
            if (lo == hi) continue;
            const I s = run_split(rrow, lo, hi, at);
            if (prune == PG_PRUNE_UPPER) {
                len[x] = s - lo;
                sum += s - lo;
            } else {
                // odd rows below and even ones above an even column, the others about an odd one
                const I e = gc >= row_begin ? run_split(rrow, s, hi, at + 1) : s;
                const uint64_t below = before[s] - before[lo], above = before[hi] - before[e];
                sum += gc & 1 ? (uint64_t)(s - lo) - below + above : below + (uint64_t)(hi - e) - above;
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (lane == 0 && sum) atomicAdd(tot, sum);
}

constexpr int CT = 128;              // threads per column block
constexpr int CSLOT = 2048;          // hash slots: 6 blocks per SM with their tables
constexpr int CLIST = 896;           // pairs kept for the second sweep
constexpr int CROWS = 1536;          // distinct rows a block takes (CT inserts may be under way beyond)
constexpr int CSURV = 320;           // rows that pass ckthr
constexpr uint32_t CHEAVY = 1u << 17;  // pairs of a column that one block takes
constexpr uint32_t CRUN = 1024;     // rows of a run that is expanded with its warp's others
constexpr uint32_t CEMPTY = 0xffffffffu;
constexpr uint32_t CMARK = 0x80000000u;

// what the column kernels share
template <class I>
struct CandArgs {
    const uint8_t *cseq;
    const uint64_t *coffs;
    uint64_t col_begin, ncols, row_begin, nrows;
    KmerTab tab;
    int stride, prune, ckthr, mosthr;
    const uint32_t *rrow;            // row occurrences by mixed code: sequence, offset
    const uint16_t *rpos;
    const uint64_t *kstart;          // first k-mer of each column, and of its k-mers:
    const I *first;                  // first row occurrence,
    const I *len;                    // their number
    pg_pair *tmp;                    // records in any column order, tmp_cap of them
    uint64_t tmp_cap;
    uint64_t *start;                 // per column: its records in tmp, their number
    uint32_t *cnt;
    unsigned long long *tot;         // [0] pairs before the prune, or after it (k_pairs_count),
                                     // [1] places in tmp, [2] overflowed columns, [3] next column,
                                     // [4] next part, [5] records
    uint32_t *ovf;                   // overflowed columns
    // parts of the overflowed columns: column, first row, end row, its column's first part
    const uint4 *part;
    uint64_t nparts;
    uint64_t *pstart;                // per part: its records in tmp, their number
    uint32_t *pcnt;
};
constexpr uint64_t CPARTS = ~0ull;   // start of a column whose records its parts hold

// Visits every occurrence pair of column c that survives the prune, in no order:
// visit(valid, row, row occurrence j, k-mer number), called by whole warps (the
// lanes without a pair pass valid = false); false, the same in all lanes, ends the
// warp's visits.  The block's threads take the column's k-mers, CQ each at a time,
// their reads in flight together.
constexpr int CQ = 3;
template <class I, class F>
__device__ __forceinline__ void cand_visit(const CandArgs<I> &A, uint64_t c, F visit)
{
    const uint64_t o = A.kstart[c];
    const int nk = (int)(A.kstart[c + 1] - o);
    const int lane = threadIdx.x & 31;
    const uint64_t gc = c + A.col_begin;
    auto one = [&](bool in, uint64_t j, int q) {
        const uint32_t r = in ? __ldg(A.rrow + j) : 0u;
        return visit(in && keep_pair(A.prune, r + A.row_begin, gc), r, j, q);
    };
    bool on = true;
    for (int q0 = 0; q0 < nk && on; q0 += (int)blockDim.x * CQ) {
        __syncwarp();
        I lo[CQ], ln[CQ];
#pragma unroll
        for (int r = 0; r < CQ; ++r) {
            const int q = q0 + r * (int)blockDim.x + (int)threadIdx.x;
            lo[r] = 0; ln[r] = 0;
            if (q < nk) { lo[r] = __ldg(A.first + o + q); ln[r] = __ldg(A.len + o + q); }
        }
        // (not unrolled: with three copies of the visits four of eighteen stall cycles an
        // issue were waits for instructions, 0.3 so; reading the rows of two or three
        // groups of pairs together was slower, 11.2 and 13.7 ms a call against 11.1)
#pragma unroll 1
        for (int r = 0; r < CQ && on; ++r) {
            // the warp's runs end to end, a lane per occurrence pair (a lane per run left
            // 3 of 32 lanes busy: a family's k-mer has tens of rows, a chance one one or
            // two); runs of more than CRUN rows one at a time
            const int q = q0 + r * (int)blockDim.x + (int)threadIdx.x;
            I lor = lo[0], lnr = ln[0];
#pragma unroll
            for (int x = 1; x < CQ; ++x)
                if (r == x) { lor = lo[x]; lnr = ln[x]; }
            const bool big = lnr > CRUN;
            const uint32_t n = big ? 0u : (uint32_t)lnr;
            uint32_t inc = n;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += y;
            }
            const uint32_t all = __shfl_sync(0xffffffffu, inc, 31);
            const I l0 = lor - (I)(inc - n);     // run start less the pairs before it
            for (uint32_t i0 = 0; i0 < all && on; i0 += 32) {
                const uint32_t i = i0 + lane;
                int src = 0;                       // the lane whose run holds pair i
#pragma unroll
                for (int d = 16; d > 0; d >>= 1)
                    if (__shfl_sync(0xffffffffu, inc, src + d - 1) <= i) src += d;
                src = min(src, 31);
                const I l = __shfl_sync(0xffffffffu, l0, src);
                on = one(i < all, (uint64_t)(I)(l + (I)i), q - lane + src);
            }
            for (uint32_t m = __ballot_sync(0xffffffffu, big); m && on; m &= m - 1) {
                const int src = __ffs(m) - 1;
                const uint64_t l = __shfl_sync(0xffffffffu, lor, src);
                const uint64_t u = __shfl_sync(0xffffffffu, lnr, src);
                for (uint64_t j = 0; j < u && on; j += 32) on = one(j + lane < u, l + j + lane, q - lane + src);
            }
        }
    }
}

// code and self score of the k-mer at p
__device__ __forceinline__ uint32_t kmer_at(const uint8_t *p, const uint8_t *map, const int *cost, const KmerTab &tab,
                                            int &score)
{
    uint32_t code = 0;
    score = 0;
    for (int j = 0; j < tab.k; ++j) {
        const uint32_t a = map[__ldg(p + j) & 31];
        code = code * tab.base + a;
        score += cost[a];
    }
    return code;
}
__device__ __forceinline__ uint64_t seed_value(uint32_t code, uint32_t rpos, int cpos)
{
    return ((uint64_t)code << 32) | ((uint64_t)rpos << 16) | (uint64_t)cpos;
}

__device__ __forceinline__ pg_pair cand_record(uint32_t row, uint64_t c, uint32_t len, uint64_t mn, uint64_t mx,
                                               int score)
{
    pg_pair p;
    p.row = row;
    p.col = (uint32_t)c;
    p.rs0 = (uint16_t)((mn >> 16) & 0xffff);
    p.cs0 = (uint16_t)(mn & 0xffff);
    p.rs1 = len >= 2 ? (uint16_t)((mx >> 16) & 0xffff) : 0;
    p.cs1 = len >= 2 ? (uint16_t)(mx & 0xffff) : 0;
    p.count = (uint16_t)len;         // ushort arithmetic of the semiring
    p.score = (int16_t)score;
    return p;
}
__device__ __forceinline__ bool cand_count_ok(uint32_t len, int ckthr) { return (int)(uint16_t)len > ckthr; }

// What bounds it: the latency of a column's chain of reads (table, code, run, row
// values, all at random places in HBM or L2), hidden by the other columns of an
// SM; hence small blocks, a hash table just large enough for the long proteins'
// columns, and the second sweep from a list of the pairs kept in shared memory
// (from the runs again where a column has more than CLIST of them).
template <class I>
__global__ void __launch_bounds__(CT, 6) k_cand(const CandArgs<I> A)
{
    __shared__ uint32_t key[CSLOT], num[CSLOT];
    __shared__ I list_j[CLIST];
    __shared__ uint32_t list_qs[CLIST];          // k-mer number << 11 | hash slot
    __shared__ uint16_t used[CROWS + CT];        // the slots in use
    __shared__ unsigned long long smin[CSURV], smax[CSURV];
    __shared__ uint32_t srow[CSURV], slen[CSURV];
    __shared__ int sscore[CSURV], cost[32];
    __shared__ uint8_t map[32];
    __shared__ uint32_t ndist, nsurv, nkeep, nlist, over;
    __shared__ unsigned long long base, next;
    static_assert(CSLOT == 2048, "11 bits of a list word");
    const int t = threadIdx.x;
    // without a threshold every row survives, so that more than CSURV are too many
    const uint32_t limit = A.ckthr <= 0 ? CSURV + 1 : CROWS;
    if (t < 32) { map[t] = A.tab.map[t]; cost[t] = A.tab.cost[t]; }
    if (t == 0) { ndist = 0; next = atomicAdd(&A.tot[3], 1ull); }
    for (int k = t; k < CSLOT; k += CT) { key[k] = CEMPTY; num[k] = 0; }
    for (;;) {
        // the next column: one counter for all blocks, columns differ in length.  The
        // one after it is taken below, so that no column waits for the counter
        // (with the rounds of cand_visit not unrolled 6.50 -> 6.35 ms for 200k proteins)
        __syncthreads();
        const uint64_t c = next;
        if (c >= A.ncols) break;
        for (uint32_t x = t; x < ndist; x += CT) { key[used[x]] = CEMPTY; num[used[x]] = 0; }
        __syncthreads();
        if (t == 0) {
            ndist = 0; nsurv = 0; nkeep = 0; nlist = 0; over = 0; base = 0;
            next = atomicAdd(&A.tot[3], 1ull);
        }
        __syncthreads();
        cand_visit(A, c, [&](bool valid, uint32_t r, uint64_t j, int q) {
            // a column that outgrows the block is left to k_cand_parts: one lane's reading
            // decides for the warp, which stays together for the ballots below
            if (__shfl_sync(0xffffffffu, *(volatile uint32_t *)&over, 0)) return false;
            uint32_t s = (r * 0x9E3779B1u) >> 21;
            bool fresh = false;
            while (valid) {
                uint32_t k = *(volatile uint32_t *)&key[s];
                if (k == CEMPTY) { k = atomicCAS(&key[s], CEMPTY, r); fresh = k == CEMPTY; }
                if (fresh || k == r) break;
                s = (s + 1) & (CSLOT - 1);
            }
            __syncwarp();
            if (valid) atomicAdd(&num[s], 1u);
            // one atomic a warp for the places in the two lists
            const uint32_t mf = __ballot_sync(0xffffffffu, fresh), mv = __ballot_sync(0xffffffffu, valid);
            const uint32_t below = (1u << (t & 31)) - 1u;
            uint32_t bf = 0, bv = 0;
            if ((t & 31) == 0) {
                if (mf) bf = atomicAdd(&ndist, (uint32_t)__popc(mf));
                if (mv) bv = atomicAdd(&nlist, (uint32_t)__popc(mv));
                if (bf + (uint32_t)__popc(mf) >= limit || bv >= CHEAVY) over = 1;
            }
            bf = __shfl_sync(0xffffffffu, bf, 0);
            bv = __shfl_sync(0xffffffffu, bv, 0) + (uint32_t)__popc(mv & below);
            if (fresh) used[bf + (uint32_t)__popc(mf & below)] = (uint16_t)s;
            if (valid && bv < CLIST) { list_j[bv] = (I)j; list_qs[bv] = ((uint32_t)q << 11) | s; }
            return true;
        });
        __syncthreads();
        for (uint32_t x = t; x < ndist && !over; x += CT) {
            const int s = used[x];
            const uint32_t len = num[s];
            uint32_t mark = 0;
            if (cand_count_ok(len, A.ckthr)) {
                const uint32_t u = atomicAdd(&nsurv, 1u);
                if (u < CSURV) {
                    srow[u] = key[s]; slen[u] = len;
                    smin[u] = ~0ull; smax[u] = 0; sscore[u] = -32768;
                    mark = CMARK | u;
                }
            }
            num[s] = mark;
        }
        __syncthreads();
        if (over || nsurv > CSURV) {
            if (t == 0) { A.ovf[atomicAdd(&A.tot[2], 1ull)] = (uint32_t)c; A.start[c] = CPARTS; }
            continue;
        }
        const uint32_t ns = nsurv;
        if (ns) {
            const uint8_t *p = A.cseq + A.coffs[A.col_begin + c];
            auto update = [&](uint32_t u, uint64_t j, int q) {
                int sc;
                const uint32_t code = kmer_at(p + (uint64_t)q * (uint64_t)A.stride, map, cost, A.tab, sc);
                const uint64_t sv = seed_value(code, __ldg(A.rpos + j), q * A.stride);
                if (sv < *(volatile unsigned long long *)&smin[u]) atomicMin(&smin[u], (unsigned long long)sv);
                if (sv > *(volatile unsigned long long *)&smax[u]) atomicMax(&smax[u], (unsigned long long)sv);
                if (sc > *(volatile int *)&sscore[u]) atomicMax(&sscore[u], sc);
            };
            if (nlist <= CLIST) {
                for (uint32_t x = t; x < nlist; x += CT) {
                    const uint32_t w = list_qs[x], mark = num[w & (CSLOT - 1)];
                    if (mark & CMARK) update(mark & ~CMARK, list_j[x], (int)(w >> 11));
                }
            } else {
                cand_visit(A, c, [&](bool valid, uint32_t r, uint64_t j, int q) {
                    if (!valid) return true;
                    uint32_t s = (r * 0x9E3779B1u) >> 21;
                    while (key[s] != r) s = (s + 1) & (CSLOT - 1);
                    const uint32_t mark = num[s];
                    if (mark & CMARK) update(mark & ~CMARK, j, q);
                    return true;
                });
            }
            __syncthreads();
            for (uint32_t u = t; u < ns; u += CT)
                if (sscore[u] > A.mosthr) atomicAdd(&nkeep, 1u);
            __syncthreads();
            if (t == 0 && nkeep) {
                base = atomicAdd(&A.tot[1], (unsigned long long)nkeep);
                atomicAdd(&A.tot[5], (unsigned long long)nkeep);
            }
            __syncthreads();
            const bool fits = base + nkeep <= A.tmp_cap;
            for (uint32_t u = t; u < ns && fits; u += CT) {
                if (sscore[u] <= A.mosthr) continue;
                uint32_t rank = 0;
                for (uint32_t v = 0; v < ns; ++v)
                    rank += srow[v] < srow[u] && sscore[v] > A.mosthr ? 1u : 0u;
                A.tmp[base + rank] = cand_record(srow[u], c, slen[u], smin[u], smax[u], sscore[u]);
            }
        }
        if (t == 0) { A.start[c] = base; A.cnt[c] = nkeep; }
    }
}

// -------------------------------------------------- columns that outgrow a block
// A column with more rows than k_cand's table, survivors than its list or pairs than
// one block should walk is done in parts of the row range.  Rows ascend within a run,
// so a part is a contiguous piece of each of the column's runs, found by a search, and
// goes through a table in shared memory that holds the seeds and the score of every
// row it meets (a part visits its pairs once).  Parts are as many as give about WPART
// rows and at most WWORK pairs each; a part that meets more than WROWS rows all the
// same is done again in narrower ones, down to one row.  Against a dense array over
// all rows of the block, 24 bytes a row to clear and to read twice: 200k proteins
// without threshold or prune 855 -> 21 ms a call, 800k with ckthr = 1 and the even/odd
// prune 7450 -> 170 ms (63 and 295 ms when the whole product was sorted).
constexpr int WT = 256;              // threads of a block
constexpr int WSLOT = 2048;          // hash slots: 3 blocks per SM
constexpr int WROWS = 1536;          // distinct rows (WT inserts may be under way beyond)
constexpr uint64_t WPART = 1000;
constexpr uint64_t WWORK = 1u << 18;
constexpr int WB = WT;               // buckets of the row order

// parts of the x-th overflowed column: their number, and (EMIT) themselves from first[x] on
template <class I, bool EMIT>
__global__ void __launch_bounds__(256) k_parts(const CandArgs<I> A, uint64_t novf, uint32_t *num, const uint64_t *first,
                                               uint4 *part)
{
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    for (uint64_t x = warp; x < novf; x += nwarps) {
        const uint64_t c = A.ovf[x], gc = c + A.col_begin;
        // rows that the prune may keep
        uint64_t nr = A.nrows;
        if (A.prune == PG_PRUNE_UPPER) nr = min(nr, gc > A.row_begin ? gc - A.row_begin : (uint64_t)0);
        uint64_t n;
        if (EMIT) {
            n = num[x];
        } else {
            uint64_t pairs = 0;
            for (uint64_t q = A.kstart[c] + lane; q < A.kstart[c + 1]; q += 32) pairs += A.len[q];
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, d);
            if (A.prune == PG_PRUNE_EVEN_ODD) pairs = (pairs + 1) / 2;
            if (A.prune == PG_PRUNE_UPPER) pairs = (uint64_t)((double)pairs * (double)nr / (double)A.nrows);
            n = max((min(pairs, nr) + WPART - 1) / WPART, (pairs + WWORK - 1) / WWORK);
            n = max(min(n, nr), (uint64_t)1);
            if (lane == 0) num[x] = (uint32_t)n;
        }
        if (EMIT) {
            const uint64_t f = first[x];
            for (uint64_t k = lane; k < n; k += 32)
                part[f + k] = make_uint4((uint32_t)c, (uint32_t)(nr * k / n), (uint32_t)(nr * (k + 1) / n), (uint32_t)f);
        }
    }
}

struct PartSmem {
    unsigned long long mn[WSLOT], mx[WSLOT];
    uint32_t key[WSLOT], num[WSLOT];
    int score[WSLOT];
    uint16_t used[WROWS + WT];       // the slots in use, in no order
    uint16_t place[WROWS + WT];      // their places in their buckets (0xffff: not kept)
    uint16_t grouped[WROWS + WT];    // the kept ones by bucket
    uint16_t sorted[WROWS + WT];     // and by row
    uint32_t hist[WB], bstart[WB + 1], wsum[WB / 32];
    int cost[32];
    uint8_t map[32];
    uint32_t ndist, over;
    unsigned long long next, base, pairs;
    uint4 part;
};

template <class I>
__global__ void __launch_bounds__(WT, 3) k_cand_parts(const CandArgs<I> A)
{
    extern __shared__ __align__(16) unsigned char part_smem[];
    PartSmem &S = *reinterpret_cast<PartSmem *>(part_smem);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t < 32) { S.map[t] = A.tab.map[t]; S.cost[t] = A.tab.cost[t]; }
    auto clear = [&](int s) {
        S.key[s] = CEMPTY; S.num[s] = 0; S.mn[s] = ~0ull; S.mx[s] = 0; S.score[s] = -32768;
    };
    auto take = [&]() {              // thread 0
        S.next = atomicAdd(&A.tot[4], 1ull);
        if (S.next < A.nparts) S.part = A.part[S.next];
    };
    for (int s = t; s < WSLOT; s += WT) clear(s);
    if (t == 0) { S.ndist = 0; S.over = 0; S.pairs = 0; take(); }
    __syncthreads();
    for (;;) {
        const uint64_t id = S.next;
        if (id >= A.nparts) break;
        const uint64_t c = S.part.x, gc = c + A.col_begin;
        const uint32_t r0 = S.part.y, r1 = S.part.z;
        const uint64_t o = A.kstart[c];
        const int nk = (int)(A.kstart[c + 1] - o);
        const uint8_t *p = A.cseq + A.coffs[gc];
        __syncthreads();
        if (t == 0) take();          // the next part's, early
        uint32_t kept = 0;           // records of the part so far
        uint64_t base = 0;
        bool room = true, whole = true;
        uint32_t a = r0, width = r1 - r0;
        while (a < r1) {
            const uint32_t b = width < r1 - a ? a + width : r1;
            const bool split = a != 0 || b != A.nrows;
            // the pairs of rows [a, b)
            bool on = true;
            for (int q0 = 0; q0 < nk && on; q0 += WT) {
                __syncwarp();
                const int q = q0 + t;
                I lo = 0, ln = 0;
                uint32_t code = 0;
                int sc = 0;
                if (q < nk) { lo = __ldg(A.first + o + q); ln = __ldg(A.len + o + q); }
                if (ln && split) {
                    const I hi = run_split(A.rrow, lo, (I)(lo + ln), (uint64_t)b);
                    lo = run_split(A.rrow, lo, hi, (uint64_t)a);
                    ln = hi - lo;
                }
                if (ln) code = kmer_at(p + (uint64_t)q * (uint64_t)A.stride, S.map, S.cost, A.tab, sc);
                // runs end to end, as in cand_visit
                auto one = [&](bool in, uint64_t j, int src) {
                    if (__shfl_sync(0xffffffffu, *(volatile uint32_t *)&S.over, 0)) return false;
                    const uint32_t r = in ? __ldg(A.rrow + j) : 0u;
                    const bool valid = in && keep_pair(A.prune, r + A.row_begin, gc);
                    const uint32_t cd = __shfl_sync(0xffffffffu, code, src);
                    const int s1 = __shfl_sync(0xffffffffu, sc, src);
                    const int qs = q - lane + src;
                    uint32_t s = (r * 0x9E3779B1u) >> 21;
                    bool fresh = false;
                    while (valid) {
                        uint32_t k = *(volatile uint32_t *)&S.key[s];
                        if (k == CEMPTY) { k = atomicCAS(&S.key[s], CEMPTY, r); fresh = k == CEMPTY; }
                        if (fresh || k == r) break;
                        s = (s + 1) & (WSLOT - 1);
                    }
                    __syncwarp();
                    if (valid) {
                        const uint64_t sv = seed_value(cd, __ldg(A.rpos + j), qs * A.stride);
                        atomicAdd(&S.num[s], 1u);
                        if (sv < *(volatile unsigned long long *)&S.mn[s]) atomicMin(&S.mn[s], (unsigned long long)sv);
                        if (sv > *(volatile unsigned long long *)&S.mx[s]) atomicMax(&S.mx[s], (unsigned long long)sv);
                        if (s1 > *(volatile int *)&S.score[s]) atomicMax(&S.score[s], s1);
                    }
                    const uint32_t mf = __ballot_sync(0xffffffffu, fresh);
                    if (mf) {
                        uint32_t bf = 0;
                        if (lane == 0) {
                            bf = atomicAdd(&S.ndist, (uint32_t)__popc(mf));
                            if (bf + (uint32_t)__popc(mf) >= WROWS) S.over = 1;
                        }
                        bf = __shfl_sync(0xffffffffu, bf, 0);
                        if (fresh) S.used[bf + (uint32_t)__popc(mf & ((1u << lane) - 1u))] = (uint16_t)s;
                    }
                    return true;
                };
                const bool big = ln > CRUN;
                const uint32_t n = big ? 0u : (uint32_t)ln;
                uint32_t inc = n;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
                    if (lane >= d) inc += y;
                }
                const uint32_t all = __shfl_sync(0xffffffffu, inc, 31);
                const I l0 = lo - (I)(inc - n);
                for (uint32_t i0 = 0; i0 < all && on; i0 += 32) {
                    const uint32_t i = i0 + lane;
                    int src = 0;
#pragma unroll
                    for (int d = 16; d > 0; d >>= 1)
                        if (__shfl_sync(0xffffffffu, inc, src + d - 1) <= i) src += d;
                    src = min(src, 31);
                    const I l = __shfl_sync(0xffffffffu, l0, src);
                    on = one(i < all, (uint64_t)(I)(l + (I)i), src);
                }
                for (uint32_t m = __ballot_sync(0xffffffffu, big); m && on; m &= m - 1) {
                    const int src = __ffs(m) - 1;
                    const uint64_t l = __shfl_sync(0xffffffffu, lo, src), u = __shfl_sync(0xffffffffu, ln, src);
                    for (uint64_t j = 0; j < u && on; j += 32) on = one(j + lane < u, l + j + lane, src);
                }
            }
            __syncthreads();
            const uint32_t nd = S.ndist;
            if (S.over && b - a > 1) {
                // too many rows: again in narrower ones.  The part's records stay together, in
                // room for as many as it can have, one to a row and to ckthr + 1 pairs
                if (whole) {
                    uint64_t mine = 0;
                    for (int q = t; q < nk; q += WT) {
                        const I lo = __ldg(A.first + o + q);
                        mine += run_split(A.rrow, lo, (I)(lo + __ldg(A.len + o + q)), (uint64_t)b) -
                                run_split(A.rrow, lo, (I)(lo + __ldg(A.len + o + q)), (uint64_t)a);
                    }
                    atomicAdd(&S.pairs, (unsigned long long)mine);
                    __syncthreads();
                    const uint64_t most = min((uint64_t)(r1 - r0), (uint64_t)S.pairs / (uint64_t)(max(A.ckthr, 0) + 1));
                    if (t == 0) S.base = atomicAdd(&A.tot[1], (unsigned long long)most);
                    __syncthreads();
                    base = S.base;
                    room = base + most <= A.tmp_cap;
                    whole = false;
                }
                width = (b - a) / 2;
            } else {
                // the rows that stay, ranked by row: grouped by its high bits first
                const int sh = max(0, 24 - __clz((int)(b - a - 1)));
                S.hist[t] = 0;
                __syncthreads();
                for (uint32_t x = t; x < nd; x += WT) {
                    const int s = S.used[x];
                    const bool keep = cand_count_ok(S.num[s], A.ckthr) && S.score[s] > A.mosthr;
                    S.place[x] = keep ? (uint16_t)atomicAdd(&S.hist[(S.key[s] - a) >> sh], 1u) : (uint16_t)0xffff;
                }
                __syncthreads();
                uint32_t inc = S.hist[t];
                const uint32_t own = inc;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
                    if (lane >= d) inc += y;
                }
                if (lane == 31) S.wsum[warp] = inc;
                __syncthreads();
                for (int k = 0; k < warp; ++k) inc += S.wsum[k];
                S.bstart[t] = inc - own;
                if (t == WT - 1) {
                    S.bstart[WB] = inc;
                    if (whole) S.base = inc ? atomicAdd(&A.tot[1], (unsigned long long)inc) : 0;
                }
                __syncthreads();
                const uint32_t nkeep = S.bstart[WB];
                if (whole) { base = S.base; room = base + nkeep <= A.tmp_cap; }
                for (uint32_t x = t; x < nd; x += WT)
                    if (S.place[x] != 0xffff) {
                        const int s = S.used[x];
                        S.grouped[S.bstart[(S.key[s] - a) >> sh] + S.place[x]] = (uint16_t)s;
                    }
                __syncthreads();
                for (uint32_t x = t; x < nkeep; x += WT) {
                    const int s = S.grouped[x];
                    const uint32_t r = S.key[s], g = (r - a) >> sh;
                    uint32_t rank = S.bstart[g];
                    for (uint32_t y = S.bstart[g]; y < S.bstart[g + 1]; ++y) rank += S.key[S.grouped[y]] < r ? 1u : 0u;
                    S.sorted[rank] = (uint16_t)s;
                }
                __syncthreads();
                for (uint32_t x = t; x < nkeep && room; x += WT) {
                    const int s = S.sorted[x];
                    A.tmp[base + kept + x] = cand_record(S.key[s], c, S.num[s], S.mn[s], S.mx[s], S.score[s]);
                }
                kept += nkeep;
                a = b;
            }
            __syncthreads();
            for (uint32_t x = t; x < nd; x += WT) clear(S.used[x]);
            if (t == 0) { S.ndist = 0; S.over = 0; S.pairs = 0; }
            __syncthreads();
        }
        if (t == 0) {
            A.pstart[id] = base;
            A.pcnt[id] = kept;
            if (kept) { atomicAdd(&A.cnt[c], kept); atomicAdd(&A.tot[5], (unsigned long long)kept); }
        }
        __syncthreads();
    }
}

// the columns' records into place, a warp per column or part (poff: the parts' records
// before each), as 32-bit words
template <class I>
__global__ void k_cand_place(const CandArgs<I> A, const uint64_t *pos, const uint64_t *poff, pg_pair *out)
{
    constexpr int W = sizeof(pg_pair) / 4;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t x = warp; x < A.ncols + A.nparts; x += nwarps) {
        uint64_t from, to, n;
        if (x < A.ncols) {
            from = A.start[x];
            if (from == CPARTS) continue;
            to = pos[x];
            n = A.cnt[x];
        } else {
            const uint64_t id = x - A.ncols;
            const uint4 p = A.part[id];
            from = A.pstart[id];
            to = pos[p.x] + poff[id] - poff[p.w];
            n = A.pcnt[id];
        }
        const uint32_t *src = reinterpret_cast<const uint32_t *>(A.tmp + from);
        uint32_t *dst = reinterpret_cast<uint32_t *>(out + to);
        for (uint64_t k = threadIdx.x & 31; k < n * W; k += 32) dst[k] = src[k];
    }
}

__global__ void k_triple_flags(const pg_result *res, uint64_t n, uint32_t *keep)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n;
         i += (uint64_t)gridDim.x * blockDim.x)
        keep[i] = (i < n && res[i].score_aln != 0.0f) ? 1u : 0u;
}

__global__ void k_triple_write(const pg_pair *pairs, const pg_result *res, uint64_t n,
                               const uint32_t *keep, const uint64_t *pos, uint64_t roff,
                               uint64_t coff, uint64_t *rows, uint64_t *cols, float *vals)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        if (!keep[i]) continue;
        const uint64_t o = pos[i];
        rows[o] = (uint64_t)pairs[i].row + roff;
        cols[o] = (uint64_t)pairs[i].col + coff;
        vals[o] = res[i].score_aln;
    }
}

// device buffers of one call, freed on every exit path
struct Bufs {
    std::vector<void *> ptrs;
    cudaStream_t st = nullptr;
    cudaMemPool_t pool = nullptr;    // the context's; null: the device's default pool
    ~Bufs()
    {
        for (void *p : ptrs) cudaFreeAsync(p, st);
    }
    template <class T>
    cudaError_t get(T **p, size_t count)
    {
        void *q = nullptr;
        const size_t bytes = std::max<size_t>(count * sizeof(T), 16);
        const cudaError_t e = pool ? cudaMallocFromPoolAsync(&q, bytes, pool, st) : cudaMallocAsync(&q, bytes, st);
        if (e == cudaSuccess) ptrs.push_back(q);
        *p = (T *)q;
        return e;
    }
};

uint64_t pow_u(uint64_t b, int k)
{
    uint64_t r = 1;
    for (int i = 0; i < k; ++i) r *= b;
    return r;
}

struct SideKmers {
    uint32_t *code = nullptr;
    uint64_t *val = nullptr;
    uint64_t *start = nullptr;       // first k-mer of each sequence (one more: n)
    uint64_t *spare = nullptr;       // n + 1 words that the sort is done with
    uint64_t n = 0;
};

// k-mers of one side: how many per sequence, and (sorted) the occurrences by mixed code
int side_kmers(Bufs &B, const uint8_t *seq, const uint64_t *offs, uint64_t s0, uint64_t ns,
               const pg_kmer_config &kc, const KmerTab &tab, int nsm, bool sorted, SideKmers &out)
{
    cudaStream_t st = B.st;
    uint64_t *cnt, *start;
    KCU(B.get(&cnt, ns + 1));
    KCU(B.get(&start, ns + 1));
    const int grid = nsm * 8;
    KCU(cudaMemsetAsync(cnt + ns, 0, sizeof(uint64_t), st));
    k_kmer_count<<<grid, 256, 0, st>>>(offs, s0, ns, kc.k, kc.stride, cnt);
    size_t tb = 0;
    KCU(cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, start, ns + 1, st));
    void *tmp;
    KCU(B.get((char **)&tmp, tb));
    KCU(cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, start, ns + 1, st));
    uint64_t total = 0;
    KCU(cudaMemcpyAsync(&total, start + ns, sizeof total, cudaMemcpyDeviceToHost, st));
    KCU(cudaStreamSynchronize(st));
    out.n = total;
    out.start = start;
    if (!sorted) return PG_OK;
    uint32_t *c0, *c1;
    uint64_t *v0, *v1;
    KCU(B.get(&c0, total)); KCU(B.get(&c1, total));
    KCU(B.get(&v0, total + 1)); KCU(B.get(&v1, total + 1));
    if (total) k_kmer_fill<<<grid, 256, 0, st>>>(seq, offs, s0, ns, kc.stride, start, tab, c0, v0);
    KCU(cudaGetLastError());
    cub::DoubleBuffer<uint32_t> kb(c0, c1);
    cub::DoubleBuffer<uint64_t> vb(v0, v1);
    size_t sb = 0;
    KCU(cub::DeviceRadixSort::SortPairs(nullptr, sb, kb, vb, (int64_t)total, 0, tab.bits, st));
    void *stmp;
    KCU(B.get((char **)&stmp, sb));
    KCU(cub::DeviceRadixSort::SortPairs(stmp, sb, kb, vb, (int64_t)total, 0, tab.bits, st));
    out.code = kb.Current();
    out.val = vb.Current();
    out.spare = vb.Alternate();
    return PG_OK;
}

// steps 2 (the table) to 4 on the sorted row occurrences; I holds their indices
template <class I>
int candidates_of(Bufs &B, const SideKmers &R, const pg_kmer_config &kc, const KmerTab &tab, int nsm,
                  const uint8_t *cseq, const uint64_t *coffs, const SideKmers &C, uint64_t row_begin,
                  uint64_t nrows, bool same, uint64_t col_begin, uint64_t ncols, uint64_t maxp, pg_pair *d_out, uint64_t cap,
                  uint64_t *n_out)
{
    cudaStream_t st = B.st;
    const int grid = nsm * 8;
    // about two occurrences per table entry, at most 2^24 entries (64 MB: inside L2)
    int tb = 1;
    while (tb < 24 && tb < tab.bits && ((uint64_t)2 << tb) < R.n) ++tb;
    const uint64_t rblocks = (R.n + RB - 1) / RB;
    uint32_t *rcnt;
    uint64_t *rfirst;
    KCU(B.get(&rcnt, rblocks + 1));
    KCU(B.get(&rfirst, rblocks + 1));
    KCU(cudaMemsetAsync(rcnt + rblocks, 0, sizeof(uint32_t), st));
    k_runs_count<<<(unsigned)rblocks, 256, 0, st>>>(R.code, R.n, rcnt);
    size_t rb = 0;
    KCU(cub::DeviceScan::ExclusiveSum(nullptr, rb, rcnt, rfirst, (int64_t)(rblocks + 1), st));
    void *rtmp;
    KCU(B.get((char **)&rtmp, rb));
    KCU(cub::DeviceScan::ExclusiveSum(rtmp, rb, rcnt, rfirst, (int64_t)(rblocks + 1), st));
    KmerRun<I> *run;
    uint32_t *rrow;
    uint16_t *rpos;
    I *cfirst, *clen;
    if (sizeof(KmerRun<I>) <= sizeof *R.spare) run = reinterpret_cast<KmerRun<I> *>(R.spare);
    else KCU(B.get(&run, std::min<uint64_t>(R.n, pow_u(tab.base, tab.k)) + 1));
    KCU(B.get(&rrow, R.n));
    KCU(B.get(&rpos, R.n));
    KCU(B.get(&cfirst, C.n));
    KCU(B.get(&clen, C.n));
    CandArgs<I> A;
    A.cseq = cseq; A.coffs = coffs;
    A.col_begin = col_begin; A.ncols = ncols; A.row_begin = row_begin; A.nrows = nrows;
    A.tab = tab;
    A.stride = kc.stride; A.prune = kc.prune; A.ckthr = kc.ckthr; A.mosthr = kc.mosthr;
    A.rrow = rrow; A.rpos = rpos; A.kstart = C.start; A.first = cfirst; A.len = clen;
    const int shift = tab.bits - tb;
    I *table;
    KCU(B.get(&table, (size_t)1 << tb));
    KCU(cudaMemsetAsync(table, 0xff, sizeof(I) << tb, st));
    k_runs_write<I><<<(unsigned)rblocks, 256, 0, st>>>(R.code, R.val, R.n, rfirst, shift, run, table, rrow, rpos);
    KCU(B.get(&A.tot, 6));
    KCU(cudaMemsetAsync(A.tot, 0, sizeof(unsigned long long) * 6, st));
    k_col_runs<I><<<grid, 256, 0, st>>>(cseq, coffs, col_begin, ncols, kc.stride, C.start, tab, table, shift, run,
                                        rfirst + rblocks, same && kc.prune != PG_PRUNE_NONE, cfirst, clen, A.tot);
    KCU(cudaGetLastError());
    unsigned long long pairs = 0;
    KCU(cudaMemcpyAsync(&pairs, A.tot, sizeof pairs, cudaMemcpyDeviceToHost, st));
    KCU(cudaStreamSynchronize(st));
    if (pairs > maxp && kc.prune != PG_PRUNE_NONE) {
        // more than the caller allows before the prune: how many after it
        I *before = nullptr;
        if (kc.prune == PG_PRUNE_EVEN_ODD) {
            KCU(B.get(&before, R.n + 1));
            k_odd_rows<I><<<grid, 256, 0, st>>>(rrow, R.n, row_begin, before);
            size_t ob = 0;
            KCU(cub::DeviceScan::ExclusiveSum(nullptr, ob, before, before, (int64_t)(R.n + 1), st));
            void *otmp;
            KCU(B.get((char **)&otmp, ob));
            KCU(cub::DeviceScan::ExclusiveSum(otmp, ob, before, before, (int64_t)(R.n + 1), st));
        }
        KCU(cudaMemsetAsync(A.tot, 0, sizeof pairs, st));
        k_pairs_count<I><<<grid, 256, 0, st>>>(col_begin, ncols, row_begin, kc.prune, C.start, rrow, before, cfirst, clen,
                                               A.tot);
        KCU(cudaGetLastError());
        KCU(cudaMemcpyAsync(&pairs, A.tot, sizeof pairs, cudaMemcpyDeviceToHost, st));
        KCU(cudaStreamSynchronize(st));
    }
    if (pairs > maxp)
        return pg_internal_fail(PG_ERR_RANGE, "pg_candidates: too many k-mer occurrence pairs for one block");
    if (!pairs) return PG_OK;
    KCU(B.get(&A.start, ncols));
    KCU(B.get(&A.cnt, ncols + 1));
    KCU(B.get(&A.ovf, ncols));
    // room for the records: as many as the caller takes, or as the pairs may give (one to
    // ckthr + 1 of them; of the pairs before a prune about half are left)
    const uint64_t most = (kc.prune == PG_PRUNE_NONE ? pairs : pairs / 2 + pairs / 16) / (uint64_t)(std::max(kc.ckthr, 0) + 1);
    A.tmp_cap = std::min<uint64_t>(cap, most + 1024);
    unsigned long long tot[6] = {};
    uint64_t *poff = nullptr;
    for (;;) {
        KCU(B.get(&A.tmp, A.tmp_cap));
        KCU(cudaMemsetAsync(A.cnt, 0, (ncols + 1) * sizeof(uint32_t), st));
        KCU(cudaMemsetAsync(A.tot, 0, sizeof tot, st));
        A.part = nullptr; A.nparts = 0; A.pstart = nullptr; A.pcnt = nullptr;
        const uint64_t blocks = std::min<uint64_t>(ncols, (uint64_t)nsm * 6);
        k_cand<I><<<(unsigned)blocks, CT, 0, st>>>(A);
        KCU(cudaGetLastError());
        KCU(cudaMemcpyAsync(tot, A.tot, sizeof tot, cudaMemcpyDeviceToHost, st));
        KCU(cudaStreamSynchronize(st));
        if (const uint64_t novf = tot[2]) {
            uint32_t *pnum;
            uint64_t *pfirst;
            KCU(B.get(&pnum, novf + 1));
            KCU(B.get(&pfirst, novf + 1));
            KCU(cudaMemsetAsync(pnum + novf, 0, sizeof(uint32_t), st));
            k_parts<I, false><<<grid, 256, 0, st>>>(A, novf, pnum, nullptr, nullptr);
            size_t pb = 0;
            KCU(cub::DeviceScan::ExclusiveSum(nullptr, pb, pnum, pfirst, (int64_t)(novf + 1), st));
            void *ptmp;
            KCU(B.get((char **)&ptmp, pb));
            KCU(cub::DeviceScan::ExclusiveSum(ptmp, pb, pnum, pfirst, (int64_t)(novf + 1), st));
            KCU(cudaMemcpyAsync(&A.nparts, pfirst + novf, sizeof A.nparts, cudaMemcpyDeviceToHost, st));
            KCU(cudaStreamSynchronize(st));
            uint4 *part;
            KCU(B.get(&part, A.nparts));
            KCU(B.get(&A.pstart, A.nparts));
            KCU(B.get(&A.pcnt, A.nparts + 1));
            KCU(B.get(&poff, A.nparts + 1));
            KCU(cudaMemsetAsync(A.pcnt + A.nparts, 0, sizeof(uint32_t), st));
            k_parts<I, true><<<grid, 256, 0, st>>>(A, novf, pnum, pfirst, part);
            A.part = part;
            KCU(cudaFuncSetAttribute(k_cand_parts<I>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PartSmem)));
            k_cand_parts<I><<<(unsigned)std::min<uint64_t>(A.nparts, (uint64_t)nsm * 3), WT, sizeof(PartSmem), st>>>(A);
            KCU(cudaGetLastError());
            KCU(cudaMemcpyAsync(tot, A.tot, sizeof tot, cudaMemcpyDeviceToHost, st));
            KCU(cudaStreamSynchronize(st));
        }
        *n_out = tot[5];
        if (tot[5] > cap) return pg_internal_fail(PG_ERR_RANGE, "pg_candidates: output capacity too small");
        if (tot[1] <= A.tmp_cap) break;
        A.tmp_cap = tot[1] + tot[1] / 8;     // more places than room: once more with room for them
    }
    if (!tot[5]) return PG_OK;
    uint64_t *pos;
    KCU(B.get(&pos, ncols + 1));
    size_t xb = 0;
    KCU(cub::DeviceScan::ExclusiveSum(nullptr, xb, A.cnt, pos, (int64_t)(ncols + 1), st));
    void *xtmp;
    KCU(B.get((char **)&xtmp, xb));
    KCU(cub::DeviceScan::ExclusiveSum(xtmp, xb, A.cnt, pos, (int64_t)(ncols + 1), st));
    if (A.nparts) {
        size_t ob = 0;
        KCU(cub::DeviceScan::ExclusiveSum(nullptr, ob, A.pcnt, poff, (int64_t)(A.nparts + 1), st));
        void *otmp;
        KCU(B.get((char **)&otmp, ob));
        KCU(cub::DeviceScan::ExclusiveSum(otmp, ob, A.pcnt, poff, (int64_t)(A.nparts + 1), st));
    }
    k_cand_place<I><<<grid, 256, 0, st>>>(A, pos, poff, d_out);
    KCU(cudaGetLastError());
    KCU(cudaStreamSynchronize(st));
    return PG_OK;
}

}  // namespace

extern "C" {

void pg_kmer_config_default(pg_kmer_config *kc)
{
    if (!kc) return;
    std::memset(kc, 0, sizeof *kc);
    kc->k = 6;
    kc->stride = 1;
    kc->alphabet = PG_ALPH_PROTEIN;
    kc->prune = PG_PRUNE_NONE;
    kc->ckthr = 0;          // src/main.cpp:104-105
    kc->mosthr = -1;
    kc->max_products = 0;
}

int pg_candidates(pg_ctx *ctx, const pg_kmer_config *kc, uint64_t row_begin, uint64_t row_end,
                  uint64_t col_begin, uint64_t col_end, pg_pair *d_out, uint64_t cap,
                  uint64_t *n_out, void *stream)
{
    if (!ctx || !kc || !n_out || (cap && !d_out))
        return pg_internal_fail(PG_ERR_ARG, "pg_candidates: bad argument");
    *n_out = 0;
    if (kc->k < 1 || kc->k > 16 || kc->stride < 1 || (kc->alphabet != PG_ALPH_PROTEIN &&
        kc->alphabet != PG_ALPH_MURPHY10) || kc->prune < 0 || kc->prune > 2)
        return pg_internal_fail(PG_ERR_ARG, "pg_candidates: bad k-mer configuration");
    const uint8_t *rseq, *cseq;
    const uint64_t *roffs, *coffs;
    uint64_t nr, nc;
    int dev, mode;
    void *cst;
    int rc = pg_internal_seqs(ctx, &rseq, &roffs, &nr, &cseq, &coffs, &nc, &dev, &cst, &mode);
    if (rc) return rc;
    if (row_begin > row_end || row_end > nr || col_begin > col_end || col_end > nc)
        return pg_internal_fail(PG_ERR_ARG, "pg_candidates: block out of range");
    if (row_end - row_begin >= (1ull << 32) || col_end - col_begin >= (1ull << 32))
        return pg_internal_fail(PG_ERR_ARG, "pg_candidates: block wider than 2^32 sequences");
    const int8_t *d_sm = nullptr;
    rc = pg_internal_score(ctx, &d_sm);
    if (rc) return rc;
    KmerTab tab;
    std::memset(&tab, 0, sizeof tab);
    tab.k = kc->k;
    int8_t sm[PG_NRES * PG_NRES];
    KCU(cudaSetDevice(dev));
    KCU(cudaMemcpy(sm, d_sm, sizeof sm, cudaMemcpyDeviceToHost));
    if (kc->alphabet == PG_ALPH_PROTEIN) {
        tab.base = PG_NRES;
        for (int a = 0; a < PG_NRES; ++a) { tab.map[a] = (uint8_t)a; tab.cost[a] = sm[a * PG_NRES + a]; }
    } else {
        tab.base = 15;
        for (int a = 0; a < PG_NRES; ++a) tab.map[a] = kMurphy[a];
        for (int m = 0; m < 15; ++m) tab.cost[m] = sm[kMurphyRep[m] * PG_NRES + kMurphyRep[m]];
    }
    for (int a = PG_NRES; a < 32; ++a) tab.map[a] = tab.map[22];   // out-of-table codes read as X
    // the reference asserts the k-mer universe fits an int (KmerOps.cpp:117-120)
    if (pow_u(tab.base, tab.k) > (uint64_t)0x7fffffff)
        return pg_internal_fail(PG_ERR_ARG, "pg_candidates: alphabet^k exceeds 2^31");
    tab.bits = 1;
    while (tab.bits < 32 && ((uint64_t)1 << tab.bits) < pow_u(tab.base, tab.k)) ++tab.bits;
    int nsm = 0;
    KCU(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    Bufs B;
    B.st = stream ? (cudaStream_t)stream : (cudaStream_t)cst;
    rc = pg_internal_pool(ctx, &B.pool);
    if (rc) return rc;
    const bool same = rseq == cseq && roffs == coffs && row_begin == col_begin && row_end == col_end;
    SideKmers R, C;
    rc = side_kmers(B, rseq, roffs, row_begin, row_end - row_begin, *kc, tab, nsm, true, R);
    if (rc) return rc;
    if (same) C = R;
    else {
        rc = side_kmers(B, cseq, coffs, col_begin, col_end - col_begin, *kc, tab, nsm, false, C);
        if (rc) return rc;
    }
    if (!R.n || !C.n) return PG_OK;
    const uint64_t maxp = kc->max_products ? kc->max_products : (1ull << 31);
    if (R.n < 0xffffffffull)
        return candidates_of<uint32_t>(B, R, *kc, tab, nsm, cseq, coffs, C, row_begin, row_end - row_begin, same,
                                       col_begin, col_end - col_begin, maxp, d_out, cap, n_out);
    return candidates_of<uint64_t>(B, R, *kc, tab, nsm, cseq, coffs, C, row_begin, row_end - row_begin, same,
                                   col_begin, col_end - col_begin, maxp, d_out, cap, n_out);
}

int pg_triples(const pg_pair *d_pairs, const pg_result *d_res, uint64_t n, uint64_t bl_roffset,
               uint64_t bl_coffset, uint64_t *d_rows, uint64_t *d_cols, float *d_vals,
               uint64_t *n_out, void *stream)
{
    if (!n_out || (n && (!d_pairs || !d_res || !d_rows || !d_cols || !d_vals)))
        return pg_internal_fail(PG_ERR_ARG, "pg_triples: bad argument");
    *n_out = 0;
    if (!n) return PG_OK;
    int dev = 0, nsm = 0;
    KCU(cudaGetDevice(&dev));
    KCU(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    Bufs B;
    B.st = (cudaStream_t)stream;
    uint32_t *keep;
    uint64_t *pos;
    KCU(B.get(&keep, n + 1));
    KCU(B.get(&pos, n + 1));
    const int grid = nsm * 8;
    k_triple_flags<<<grid, 256, 0, B.st>>>(d_res, n, keep);
    size_t tb = 0;
    KCU(cub::DeviceScan::ExclusiveSum(nullptr, tb, keep, pos, n + 1, B.st));
    void *tmp;
    KCU(B.get((char **)&tmp, tb));
    KCU(cub::DeviceScan::ExclusiveSum(tmp, tb, keep, pos, n + 1, B.st));
    k_triple_write<<<grid, 256, 0, B.st>>>(d_pairs, d_res, n, keep, pos, bl_roffset, bl_coffset,
                                            d_rows, d_cols, d_vals);
    KCU(cudaGetLastError());
    uint64_t cnt = 0;
    KCU(cudaMemcpyAsync(&cnt, pos + n, sizeof cnt, cudaMemcpyDeviceToHost, B.st));
    KCU(cudaStreamSynchronize(B.st));
    *n_out = cnt;
    return PG_OK;
}

}  // extern "C"
