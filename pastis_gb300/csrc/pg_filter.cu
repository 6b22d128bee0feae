// pg_filter.cu -- learned candidate-pair filter (sm_103a).
//
// PASTIS prunes candidate pairs before alignment by their k-mer overlap only:
// count <= ckthr or score <= mosthr drops a pair (src/DistPWRunner.cpp:48-54).
// This file adds a learned version of that prune: a 16 -> 64 -> 64 -> 1 ReLU
// network over k-mer overlap features of each pair, with BF16 weights and FP32
// accumulation on the tensor cores (mma.sync m16n8k16), trained by the
// hand-written forward / backward / Adam kernels below on pairs labelled by
// this library's own aligner.  pg_align_filtered aligns only the pairs the
// network keeps; the plain aligner stays the reference and judges its recall.
//
// Features of a pair (row sequence length m, column length n, L = max(m, n),
// k-mer count c, k-mer score s, seeds (r0, c0), (r1, c1)), fixed scaling:
//   0 log2(1+c)/4       1 s/32             2 [c >= 2]
//   3 (c0-r0)/L         4 (c1-r1)/L*[c>=2]  5 |(c0-r0)-(c1-r1)|/L*[c>=2]
//   6 r0/m              7 c0/n             8 best seed diagonal window (below)
//   9 log2(m)/12       10 log2(n)/12      11 |log2(m/n)|
//  12..15 |fraction difference| of the two sequences in four residue groups:
//         hydrophobic AVLIMFWC, polar NQSTYGP, positive RKH, negative DE
// Seed diagonal window: the mean substitution score over the 64 positions of
// a seed's diagonal from 32 before its start (positions outside either
// sequence skipped), divided by 4; the larger of the two seeds when the pair
// has two different ones.  It is the ungapped check BLAST-style seeders make
// before a gapped extension.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/pastis_gb300.h"

int pg_internal_seqs(const pg_ctx *c, const uint8_t **rseq, const uint64_t **roffs, uint64_t *nr,
                     const uint8_t **cseq, const uint64_t **coffs, uint64_t *nc, int *device,
                     void **stream, int *mode);
int pg_internal_fail(int code, const char *msg);
int pg_internal_score(const pg_ctx *c, const int8_t **d_sm);

namespace {

constexpr int NF = PG_FILTER_FEATURES;   // 16
constexpr int NH = 64;
// parameter block (FP32 master copy); weights stored output-major
constexpr int P_W1 = 0;                  // [64][16]
constexpr int P_B1 = P_W1 + NH * NF;     // [64]
constexpr int P_W2 = P_B1 + NH;          // [64][64]
constexpr int P_B2 = P_W2 + NH * NH;     // [64]
constexpr int P_W3 = P_B2 + NH;          // [64]
constexpr int P_B3 = P_W3 + NH;          // [1]
constexpr int NPARAM = P_B3 + 1;

constexpr int FWARPS = 4;                // warps per block in the MLP kernels

#define FCU(call)                                                                  \
    do {                                                                           \
        cudaError_t e_ = (call);                                                   \
        if (e_ != cudaSuccess)                                                     \
            return pg_internal_fail(e_ == cudaErrorMemoryAllocation ? PG_ERR_OOM : PG_ERR_CUDA, \
                                    cudaGetErrorString(e_));                       \
    } while (0)

// ------------------------------------------------------------ tensor cores
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ uint32_t ld_u32(const __nv_bfloat16 *p) { return *reinterpret_cast<const uint32_t *>(p); }
__device__ __forceinline__ void st_bf16x2(__nv_bfloat16 *p, float lo, float hi)
{
    *reinterpret_cast<uint32_t *>(p) = pack_bf16(lo, hi);
}

// four 8x8 BF16 matrices; lanes 8i..8i+7 give the row addresses of matrix i
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16 *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const __nv_bfloat16 *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}

// Weights as the MLP kernels read them from shared memory.  The rows are
// padded to an odd number of 16-byte units, so that the eight rows of an
// ldmatrix tile (and the rows of a tile's accumulator stores) meet eight
// different bank groups.  The backward pass reads w2t transposed, so one copy
// serves both directions.
constexpr int LD1 = NF + 8, LD2 = NH + 8;
struct SmemW {
    alignas(16) __nv_bfloat16 w1t[NH * LD1];   // [out][in]
    alignas(16) __nv_bfloat16 w2t[NH * LD2];   // [out][in]
    float b1[NH], b2[NH], w3[NH], b3;
};

// Every load is issued before the first conversion: a block does one or two
// tiles a warp, so the way of the weights through L2 is a good part of it.
__device__ __forceinline__ void load_weights(SmemW &s, const float *P)
{
    static_assert(FWARPS * 32 == 128 && NH * NF == 2 * 512 && P_W2 % 4 == 0, "weight load split");
    const int k = threadIdx.x;
    float4 v1[2], v2[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v2[u] = reinterpret_cast<const float4 *>(P + P_W2)[k + u * 128];
#pragma unroll
    for (int u = 0; u < 2; ++u) v1[u] = reinterpret_cast<const float4 *>(P + P_W1)[k + u * 128];
    if (k < NH) {
        s.b1[k] = P[P_B1 + k];
        s.b2[k] = P[P_B2 + k];
        s.w3[k] = P[P_W3 + k];
    }
    if (k == 0) s.b3 = P[P_B3];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int e = (k + u * 128) * 4;
        uint2 q = make_uint2(pack_bf16(v2[u].x, v2[u].y), pack_bf16(v2[u].z, v2[u].w));
        *reinterpret_cast<uint2 *>(s.w2t + (e / NH) * LD2 + e % NH) = q;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int e = (k + u * 128) * 4;
        uint2 q = make_uint2(pack_bf16(v1[u].x, v1[u].y), pack_bf16(v1[u].z, v1[u].w));
        *reinterpret_cast<uint2 *>(s.w1t + (e / NF) * LD1 + e % NF) = q;
    }
}

// Forward pass of 16 samples.  Thread (g = lane/4, t = lane%4) ends up with
// the rows g and g+8 of h1 / h2 in the mma accumulator layout, and the logits
// of those two rows.
struct Tile {
    float h1[8][4];   // relu(x W1 + b1), fp32
    float h2[8][4];   // relu(h1_bf16 W2 + b2)
    float z0, z1;     // logits of rows g, g+8
};

// the A fragment of 16 rows of X (bf16 [n][16]) from row `base`; rows past n are 0
__device__ __forceinline__ void load_x(uint32_t (&a)[4], const __nv_bfloat16 *X, uint64_t n, uint64_t base)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint64_t r0 = base + g, r1 = base + g + 8;
    a[0] = r0 < n ? ld_u32(X + r0 * NF + 2 * t) : 0u;
    a[1] = r1 < n ? ld_u32(X + r1 * NF + 2 * t) : 0u;
    a[2] = r0 < n ? ld_u32(X + r0 * NF + 2 * t + 8) : 0u;
    a[3] = r1 < n ? ld_u32(X + r1 * NF + 2 * t + 8) : 0u;
}

__device__ __forceinline__ void load_labels(float (&v)[4], const float *label, const float *wts, uint64_t n,
                                            uint64_t base)
{
    const uint64_t r0 = base + ((threadIdx.x & 31) >> 2), r1 = r0 + 8;
    v[0] = r0 < n ? label[r0] : 0.f;
    v[1] = r1 < n ? label[r1] : 0.f;
    v[2] = r0 < n ? wts[r0] : 0.f;
    v[3] = r1 < n ? wts[r1] : 0.f;
}

__device__ __forceinline__ void forward_tile(const SmemW &s, const uint32_t (&a)[4], Tile &T)
{
    const int lane = threadIdx.x & 31, t = lane & 3;
#pragma unroll
    for (int np = 0; np < 4; ++np) {   // a pair of 8-unit tiles an ldmatrix
        uint32_t b[4];
        ldsm4(b, s.w1t + (np * 16 + (lane & 7) + (lane >> 4) * 8) * LD1 + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int nt = 2 * np + q, c = nt * 8 + 2 * t;
            float d[4] = {0.f, 0.f, 0.f, 0.f};
            mma16816(d, a, b[2 * q], b[2 * q + 1]);
            T.h1[nt][0] = fmaxf(d[0] + s.b1[c], 0.f);
            T.h1[nt][1] = fmaxf(d[1] + s.b1[c + 1], 0.f);
            T.h1[nt][2] = fmaxf(d[2] + s.b1[c], 0.f);
            T.h1[nt][3] = fmaxf(d[3] + s.b1[c + 1], 0.f);
        }
    }
    uint32_t a2[4][4];
#pragma unroll
    for (int kc = 0; kc < 4; ++kc) {
        a2[kc][0] = pack_bf16(T.h1[2 * kc][0], T.h1[2 * kc][1]);
        a2[kc][1] = pack_bf16(T.h1[2 * kc][2], T.h1[2 * kc][3]);
        a2[kc][2] = pack_bf16(T.h1[2 * kc + 1][0], T.h1[2 * kc + 1][1]);
        a2[kc][3] = pack_bf16(T.h1[2 * kc + 1][2], T.h1[2 * kc + 1][3]);
    }
    float z0 = 0.f, z1 = 0.f;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int kp = 0; kp < 2; ++kp) {
            uint32_t b[4];
            ldsm4(b, s.w2t + (nt * 8 + (lane & 7)) * LD2 + kp * 32 + (lane >> 3) * 8);
            mma16816(d, a2[2 * kp], b[0], b[1]);
            mma16816(d, a2[2 * kp + 1], b[2], b[3]);
        }
        const int c = nt * 8 + 2 * t;
        T.h2[nt][0] = fmaxf(d[0] + s.b2[c], 0.f);
        T.h2[nt][1] = fmaxf(d[1] + s.b2[c + 1], 0.f);
        T.h2[nt][2] = fmaxf(d[2] + s.b2[c], 0.f);
        T.h2[nt][3] = fmaxf(d[3] + s.b2[c + 1], 0.f);
        z0 += T.h2[nt][0] * s.w3[c] + T.h2[nt][1] * s.w3[c + 1];
        z1 += T.h2[nt][2] * s.w3[c] + T.h2[nt][3] * s.w3[c + 1];
    }
    z0 += __shfl_xor_sync(0xffffffffu, z0, 1);
    z0 += __shfl_xor_sync(0xffffffffu, z0, 2);
    z1 += __shfl_xor_sync(0xffffffffu, z1, 1);
    z1 += __shfl_xor_sync(0xffffffffu, z1, 2);
    T.z0 = z0 + s.b3;
    T.z1 = z1 + s.b3;
}

// ----------------------------------------------------------------- kernels
// Residue-group fractions of every sequence, a warp a sequence: 16 bytes a
// lane and load, counts in packed bytes of a 32-bit word (at most 16 of a group
// a load, so they are unpacked after each).  Bound by instruction issue, two a
// residue: 15 us for 30 thousand proteins of 280 residues (125 us with a thread
// a sequence, whose byte loads shared no sector with its neighbours').
__global__ void k_composition(const uint8_t *seq, const uint64_t *offs, uint64_t nseq, float4 *comp)
{
    // residue group of each code in ARNDCQEGHILKMFPSTWYVBZX*J as its counter's
    // byte (hydrophobic, polar, positive, negative); codes past J have none
    __shared__ uint32_t inc[32];
    if (threadIdx.x < 32) {
        const uint8_t grp[25] = {0, 2, 1, 3, 0, 1, 3, 1, 2, 0, 0, 2, 0, 0, 1, 1, 1, 0, 1, 0, 4, 4, 4, 4, 4};
        const int g = threadIdx.x < 25 ? grp[threadIdx.x] : 4;
        inc[threadIdx.x] = g < 4 ? 1u << (8 * g) : 0u;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; i < nseq; i += nw) {
        const uint64_t b = offs[i], e = offs[i + 1];
        uint32_t c[4] = {0, 0, 0, 0};
        // whole aligned 16-byte units inside [b, e); the ends by bytes
        const uint64_t base = (uint64_t)(uintptr_t)seq;
        const uint64_t ab = (base + b + 15) & ~15ull, ae = (base + e) & ~15ull;
        const uint64_t hb = ab > base + e ? e : ab - base;        // end of the head
        const uint64_t tb = ae < ab ? e : ae - base;              // start of the tail
        uint32_t acc = 0;
        if (b + lane < hb) { const uint8_t r = seq[b + lane]; acc += r < 32 ? inc[r] : 0u; }
        if (tb + lane < e) { const uint8_t r = seq[tb + lane]; acc += r < 32 ? inc[r] : 0u; }
        c[0] = acc & 0xff; c[1] = acc >> 8 & 0xff; c[2] = acc >> 16 & 0xff; c[3] = acc >> 24;
        for (uint64_t q = ab + 16 * lane; q < ae; q += 512) {
            const uint4 v = *reinterpret_cast<const uint4 *>((uintptr_t)q);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            acc = 0;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const uint32_t r = w[k >> 2] >> (8 * (k & 3)) & 0xff;
                acc += r < 32 ? inc[r] : 0u;
            }
            c[0] += acc & 0xff; c[1] += acc >> 8 & 0xff; c[2] += acc >> 16 & 0xff; c[3] += acc >> 24;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k] = __reduce_add_sync(0xffffffffu, c[k]);
        const float inv = e > b ? 1.f / (float)(e - b) : 0.f;
        if (lane == 0)
            comp[i] = make_float4((float)c[0] * inv, (float)c[1] * inv, (float)c[2] * inv, (float)c[3] * inv);
    }
}

constexpr int WIN_BEFORE = 32, WIN_LEN = 64;

// Features of 32 pairs a warp.  The two seeds' diagonal windows are summed by
// the whole warp for one pair after the other (lanes 0-15 the first seed, 16-31
// the second; position t of the window on lane t % 16), so that a window is
// four coalesced loads of each sequence; then every lane forms its own pair's
// row.  Bound by instruction issue, 180 a pair: 37 us for 150 thousand pairs (55
// us with a thread a pair walking its windows by bytes).
__global__ void __launch_bounds__(256) k_features(const pg_pair *pairs, uint64_t n, uint64_t roff, uint64_t coff,
                           const uint8_t *rseq, const uint64_t *roffs, uint64_t nr,
                           const uint8_t *cseq, const uint64_t *coffs, uint64_t nc,
                           const int8_t *sm, const float4 *rcomp, const float4 *ccomp,
                           __nv_bfloat16 *X, int *status)
{
    __shared__ int8_t ssm[PG_NRES * PG_NRES];
    for (int k = threadIdx.x; k < PG_NRES * PG_NRES; k += blockDim.x) ssm[k] = sm[k];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5), groups = (n + 31) / 32;
    for (uint64_t grp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; grp < groups; grp += nw) {
        const uint64_t p = grp * 32 + lane;
        pg_pair pr = {};
        uint64_t r = 0, c = 0, rb = 0, cb = 0;
        int mi = 0, ni = 0;
        float4 ca = make_float4(0.f, 0.f, 0.f, 0.f), cc = ca;
        bool ok = false;
        if (p < n) {
            pr = pairs[p];
            r = pr.row + roff;
            c = pr.col + coff;
            ok = r < nr && c < nc;
            if (ok) {
                rb = roffs[r];
                cb = coffs[c];
                mi = (int)(roffs[r + 1] - rb);
                ni = (int)(coffs[c + 1] - cb);
                ca = rcomp[r];
                cc = ccomp[c];
            } else atomicOr(status, 1);
        }
        const bool two = pr.count >= 2;
        const bool win2 = two && (pr.rs1 != pr.rs0 || pr.cs1 != pr.cs0);
        float win = 0.f;
        const unsigned live = __ballot_sync(0xffffffffu, ok);
        const int h = lane >> 4, l16 = lane & 15;
        for (unsigned rest = live; rest; rest &= rest - 1) {
            const int src = __ffs(rest) - 1;
            const uint8_t *V = rseq + __shfl_sync(0xffffffffu, rb, src);
            const uint8_t *H = cseq + __shfl_sync(0xffffffffu, cb, src);
            const int m = __shfl_sync(0xffffffffu, mi, src), nn = __shfl_sync(0xffffffffu, ni, src);
            const int a0 = __shfl_sync(0xffffffffu, (int)pr.rs0, src), a1 = __shfl_sync(0xffffffffu, (int)pr.rs1, src);
            const int b0 = __shfl_sync(0xffffffffu, (int)pr.cs0, src), b1 = __shfl_sync(0xffffffffu, (int)pr.cs1, src);
            const bool both = __shfl_sync(0xffffffffu, (int)win2, src);
            int sum = 0, cnt = 0;
            if (h == 0 || both) {
                const int i0 = (h ? a1 : a0) - WIN_BEFORE + l16, j0 = (h ? b1 : b0) - WIN_BEFORE + l16;
                uint8_t v[WIN_LEN / 16], w[WIN_LEN / 16];
                bool in[WIN_LEN / 16];
#pragma unroll
                for (int q = 0; q < WIN_LEN / 16; ++q) {
                    const int i = i0 + 16 * q, j = j0 + 16 * q;
                    in[q] = i >= 0 && j >= 0 && i < m && j < nn;
                    v[q] = in[q] ? V[i] : 0;
                    w[q] = in[q] ? H[j] : 0;
                }
#pragma unroll
                for (int q = 0; q < WIN_LEN / 16; ++q) {
                    sum += in[q] ? (int)ssm[v[q] * PG_NRES + w[q]] : 0;
                    cnt += in[q];
                }
            }
            // |sum| <= 64 * 128 and cnt <= 64 of a half: both in one word
            int pk = (sum << 8) + cnt;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) pk += __shfl_xor_sync(0xffffffffu, pk, o);
            const int c1 = pk & 0xff, s1 = (pk - c1) >> 8;
            const float mine = c1 ? (float)s1 / (4.f * (float)c1) : 0.f;
            const float x0 = __shfl_sync(0xffffffffu, mine, 0), x1 = __shfl_sync(0xffffffffu, mine, 16);
            if (lane == src) win = both ? fmaxf(x0, x1) : x0;
        }
        if (p >= n) continue;
        float f[NF];
#pragma unroll
        for (int k = 0; k < NF; ++k) f[k] = 0.f;
        if (ok) {
            const float m = (float)(uint64_t)(unsigned)mi, nn = (float)(uint64_t)(unsigned)ni;
            const float mm = fmaxf(m, 1.f), n1 = fmaxf(nn, 1.f), L = fmaxf(mm, n1);
            const float d0 = ((float)pr.cs0 - (float)pr.rs0) / L;
            const float d1 = ((float)pr.cs1 - (float)pr.rs1) / L;
            f[0] = log2f(1.f + (float)pr.count) * 0.25f;
            f[1] = (float)pr.score * (1.f / 32.f);
            f[2] = two ? 1.f : 0.f;
            f[3] = d0;
            f[4] = two ? d1 : 0.f;
            f[5] = two ? fabsf(d0 - d1) : 0.f;
            f[6] = (float)pr.rs0 / mm;
            f[7] = (float)pr.cs0 / n1;
            f[8] = win;
            f[9] = log2f(mm) * (1.f / 12.f);
            f[10] = log2f(n1) * (1.f / 12.f);
            f[11] = fabsf(log2f(mm / n1));
            f[12] = fabsf(ca.x - cc.x);
            f[13] = fabsf(ca.y - cc.y);
            f[14] = fabsf(ca.z - cc.z);
            f[15] = fabsf(ca.w - cc.w);
        }
        uint32_t o[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = pack_bf16(f[2 * k], f[2 * k + 1]);
        uint32_t *dst = reinterpret_cast<uint32_t *>(X + p * NF);
#pragma unroll
        for (int k = 0; k < 8; ++k) dst[k] = o[k];
    }
}

// Logits, 16 rows a warp and step.  Bound by the latency of the weights' way into
// shared memory for a mini-batch and by issue above it: 8192 rows 4.4 us, 150
// thousand 10 us (10 and 60 us with strided weight reads, eight to a bank, and
// scalar conversions into two layouts).
__global__ void __launch_bounds__(FWARPS * 32) k_mlp_forward(const float *P, const __nv_bfloat16 *X,
                                                              uint64_t n, float *logits)
{
    __shared__ SmemW s;
    load_weights(s, P);
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint64_t tiles = (n + 15) / 16;
    for (uint64_t tile = blockIdx.x * (uint64_t)FWARPS + (threadIdx.x >> 5); tile < tiles;
         tile += (uint64_t)gridDim.x * FWARPS) {
        uint32_t a[4];
        load_x(a, X, n, tile * 16);
        Tile T;
        forward_tile(s, a, T);
        if (t == 0) {
            const uint64_t r0 = tile * 16 + g, r1 = r0 + 8;
            if (r0 < n) logits[r0] = T.z0;
            if (r1 < n) logits[r1] = T.z1;
        }
    }
}

// A block's 64 samples as the weight-gradient products read them, [sample][unit]
constexpr int FROWS = FWARPS * 16;
struct Stage {
    alignas(16) __nv_bfloat16 dh2[FROWS * LD2];   // dL/d(pre-activation 2)
    alignas(16) __nv_bfloat16 h1[FROWS * LD2];    // h1 as layer 2 saw it
    alignas(16) __nv_bfloat16 dh1[FROWS * LD2];   // dL/d(pre-activation 1)
    alignas(16) __nv_bfloat16 x[FROWS * LD1];
};

// Sum N values a lane over the eight lanes with the same t: each step sends
// half of what is left, so N/8 values remain: those from index g * N/8 on.
template <int N> __device__ __forceinline__ void sum_rows(float (&v)[N], int lane)
{
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const int o = 16 >> s, half = N >> (s + 1);
        const bool up = lane & o;
#pragma unroll
        for (int k = 0; k < half; ++k) {
            const float send = up ? v[k] : v[k + half], keep = up ? v[k + half] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
}

// four neighbouring gradients from a pair of lanes' accumulators: the even lane
// takes row g, the odd one row g + 8
__device__ __forceinline__ void add_tile(float *G, int ld, const float (&d)[4], int lane)
{
    const int g = lane >> 2, t = lane & 3;
    const bool odd = t & 1;
    const float s0 = odd ? d[0] : d[2], s1 = odd ? d[1] : d[3];
    const float r0 = __shfl_xor_sync(0xffffffffu, s0, 1), r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
    const float4 v = odd ? make_float4(r0, r1, d[2], d[3]) : make_float4(d[0], d[1], r0, r1);
    atomicAdd(reinterpret_cast<float4 *>(G + (g + 8 * odd) * ld + 4 * (t >> 1)), v);
}

// One pass over a mini-batch: forward, binary cross-entropy with logits
// (weighted by wts, averaged by inv_norm), backward, and gradient
// accumulation into G (same layout as P) and the loss after it.
//
// Bound by latency: at 8192 rows a block has one 64-row step.  The four warps
// take 16 rows each through both layers and back; then the block's activations
// stand in shared memory as [sample][unit], and warp w forms rows 16w..16w+15
// of both weight gradients over all 64 samples, in registers that live as long
// as the block.  Nothing is added in shared memory (an FP32 add there is a
// compare-and-swap loop): a block ends in one vector reduction to G.
// 8192 rows: 6.9 us (30 us with every 16x8 product added to shared memory).
__global__ void __launch_bounds__(FWARPS * 32) k_mlp_backward(const float *P, const __nv_bfloat16 *X,
                                                               const float *label, const float *wts,
                                                               uint64_t n, float inv_norm, float *G)
{
    __shared__ SmemW s;
    __shared__ Stage st;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, wib = threadIdx.x >> 5;
    uint64_t base = blockIdx.x * (uint64_t)FROWS + wib * 16;
    uint32_t a[4];
    float lw[4];   // labels and weights of rows g, g + 8
    load_x(a, X, n, base);
    load_labels(lw, label, wts, n, base);
    load_weights(s, P);
    float dw2[8][4] = {}, dw1[2][4] = {};
    float pw3[16] = {}, pb2[16] = {}, pb1[16] = {}, pb3 = 0.f, ploss = 0.f;
    __syncthreads();
    const uint64_t steps = (n + FROWS - 1) / FROWS;
    for (uint64_t step = blockIdx.x; step < steps; step += gridDim.x) {
        const uint64_t r0 = base + g, r1 = r0 + 8;
        const float y0 = lw[0], y1 = lw[1], w0 = lw[2], w1 = lw[3];
        __nv_bfloat16 *sx = st.x + (wib * 16 + g) * LD1 + 2 * t;
        *reinterpret_cast<uint32_t *>(sx) = a[0];
        *reinterpret_cast<uint32_t *>(sx + 8 * LD1) = a[1];
        *reinterpret_cast<uint32_t *>(sx + 8) = a[2];
        *reinterpret_cast<uint32_t *>(sx + 8 * LD1 + 8) = a[3];
        Tile T;
        forward_tile(s, a, T);
        const float p0 = 1.f / (1.f + __expf(-T.z0)), p1 = 1.f / (1.f + __expf(-T.z1));
        const float dz0 = r0 < n ? w0 * (p0 - y0) * inv_norm : 0.f;
        const float dz1 = r1 < n ? w1 * (p1 - y1) * inv_norm : 0.f;
        if (t == 0) {
            const float l0 = fmaxf(T.z0, 0.f) - T.z0 * y0 + log1pf(__expf(-fabsf(T.z0)));
            const float l1 = fmaxf(T.z1, 0.f) - T.z1 * y1 + log1pf(__expf(-fabsf(T.z1)));
            ploss += ((r0 < n ? w0 * l0 : 0.f) + (r1 < n ? w1 * l1 : 0.f)) * inv_norm;
            pb3 += dz0 + dz1;
        }
        // layer 3 and the pre-activation gradient of layer 2
        float dh2[8][4];
        __nv_bfloat16 *sh = st.h1 + (wib * 16 + g) * LD2 + 2 * t;
        __nv_bfloat16 *s2 = st.dh2 + (wib * 16 + g) * LD2 + 2 * t;
        __nv_bfloat16 *s1 = st.dh1 + (wib * 16 + g) * LD2 + 2 * t;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int c = nt * 8 + 2 * t;
            pw3[2 * nt] += dz0 * T.h2[nt][0] + dz1 * T.h2[nt][2];
            pw3[2 * nt + 1] += dz0 * T.h2[nt][1] + dz1 * T.h2[nt][3];
            dh2[nt][0] = T.h2[nt][0] > 0.f ? dz0 * s.w3[c] : 0.f;
            dh2[nt][1] = T.h2[nt][1] > 0.f ? dz0 * s.w3[c + 1] : 0.f;
            dh2[nt][2] = T.h2[nt][2] > 0.f ? dz1 * s.w3[c] : 0.f;
            dh2[nt][3] = T.h2[nt][3] > 0.f ? dz1 * s.w3[c + 1] : 0.f;
            pb2[2 * nt] += dh2[nt][0] + dh2[nt][2];
            pb2[2 * nt + 1] += dh2[nt][1] + dh2[nt][3];
            st_bf16x2(sh + nt * 8, T.h1[nt][0], T.h1[nt][1]);
            st_bf16x2(sh + 8 * LD2 + nt * 8, T.h1[nt][2], T.h1[nt][3]);
        }
        // dh1 = dh2 W2 (tensor cores), masked by the layer-1 ReLU
        uint32_t a2[4][4];
#pragma unroll
        for (int kc = 0; kc < 4; ++kc) {
            a2[kc][0] = pack_bf16(dh2[2 * kc][0], dh2[2 * kc][1]);
            a2[kc][1] = pack_bf16(dh2[2 * kc][2], dh2[2 * kc][3]);
            a2[kc][2] = pack_bf16(dh2[2 * kc + 1][0], dh2[2 * kc + 1][1]);
            a2[kc][3] = pack_bf16(dh2[2 * kc + 1][2], dh2[2 * kc + 1][3]);
            *reinterpret_cast<uint32_t *>(s2 + kc * 16) = a2[kc][0];
            *reinterpret_cast<uint32_t *>(s2 + 8 * LD2 + kc * 16) = a2[kc][1];
            *reinterpret_cast<uint32_t *>(s2 + kc * 16 + 8) = a2[kc][2];
            *reinterpret_cast<uint32_t *>(s2 + 8 * LD2 + kc * 16 + 8) = a2[kc][3];
        }
        // rows of a transposed tile pair: unit (lane & 7) + 8 * bit 3, columns 8 * bit 4
        const int trow = (lane & 7) + (lane & 8), tcol = (lane >> 4) * 8;
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            float d[2][4] = {};
#pragma unroll
            for (int kc = 0; kc < 4; ++kc) {
                uint32_t b[4];
                ldsm4t(b, s.w2t + (kc * 16 + trow) * LD2 + np * 16 + tcol);
                mma16816(d[0], a2[kc], b[0], b[1]);
                mma16816(d[1], a2[kc], b[2], b[3]);
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int nt = 2 * np + q;
                const float e0 = T.h1[nt][0] > 0.f ? d[q][0] : 0.f, e1 = T.h1[nt][1] > 0.f ? d[q][1] : 0.f;
                const float e2 = T.h1[nt][2] > 0.f ? d[q][2] : 0.f, e3 = T.h1[nt][3] > 0.f ? d[q][3] : 0.f;
                pb1[2 * nt] += e0 + e2;
                pb1[2 * nt + 1] += e1 + e3;
                st_bf16x2(s1 + nt * 8, e0, e1);
                st_bf16x2(s1 + 8 * LD2 + nt * 8, e2, e3);
            }
        }
        base += (uint64_t)gridDim.x * FROWS;
        load_x(a, X, n, base);   // the next step's rows
        load_labels(lw, label, wts, n, base);
        __syncthreads();
        // dW2[o][i] = sum_s dh2[s][o] h1[s][i], dW1[o][f] = sum_s dh1[s][o] x[s][f]:
        // M = this warp's 16 o, N = i or f, K = the samples
        const int arow = (lane & 7) + (lane >> 4) * 8, acol = wib * 16 + (lane & 8);
#pragma unroll
        for (int kc = 0; kc < FWARPS; ++kc) {
            uint32_t am[4], b[4];
            ldsm4t(am, st.dh2 + (kc * 16 + arow) * LD2 + acol);
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                ldsm4t(b, st.h1 + (kc * 16 + trow) * LD2 + np * 16 + tcol);
                mma16816(dw2[2 * np], am, b[0], b[1]);
                mma16816(dw2[2 * np + 1], am, b[2], b[3]);
            }
            ldsm4t(am, st.dh1 + (kc * 16 + arow) * LD2 + acol);
            ldsm4t(b, st.x + (kc * 16 + trow) * LD1 + tcol);
            mma16816(dw1[0], am, b[0], b[1]);
            mma16816(dw1[1], am, b[2], b[3]);
        }
        __syncthreads();
    }
    float *G2 = G + P_W2 + wib * 16 * NH, *G1 = G + P_W1 + wib * 16 * NF;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) add_tile(G2 + nt * 8, NH, dw2[nt], lane);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) add_tile(G1 + nt * 8, NF, dw1[nt], lane);
    // the vectors: over the warp's rows, then over the warps
    float *sum = reinterpret_cast<float *>(st.dh2);          // [warp][w3, b2, b1][unit], b3, loss
    sum_rows(pw3, lane);
    sum_rows(pb2, lane);
    sum_rows(pb1, lane);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
        pb3 += __shfl_xor_sync(0xffffffffu, pb3, o);
        ploss += __shfl_xor_sync(0xffffffffu, ploss, o);
    }
    // values 2g and 2g + 1 of the 16 are units 8g + 2t and the next
    const int unit = g * 8 + 2 * t;
    constexpr int WS = 3 * NH + 2;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        sum[wib * WS + unit + k] = pw3[k];
        sum[wib * WS + NH + unit + k] = pb2[k];
        sum[wib * WS + 2 * NH + unit + k] = pb1[k];
    }
    if (lane == 0) {
        sum[wib * WS + 3 * NH] = pb3;
        sum[wib * WS + 3 * NH + 1] = ploss;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < WS; k += FWARPS * 32) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < FWARPS; ++w) v += sum[w * WS + k];
        const int at = k < NH ? P_W3 + k : k < 2 * NH ? P_B2 + k - NH : k < 3 * NH ? P_B1 + k - 2 * NH
                     : k == 3 * NH ? P_B3 : NPARAM;
        atomicAdd(G + at, v);
    }
}

// Adam (Kingma & Ba 2015) on the FP32 master copy; clears the gradients.
__global__ void k_adam(float *P, float *G, float *M1, float *M2, float lr, float b1, float b2,
                       float eps, float c1, float c2)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= NPARAM) return;
    const float gk = G[k];
    const float m = b1 * M1[k] + (1.f - b1) * gk;
    const float v = b2 * M2[k] + (1.f - b2) * gk * gk;
    M1[k] = m;
    M2[k] = v;
    P[k] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
    G[k] = 0.f;
}

__global__ void k_compact(const float *logits, uint64_t n, float thr, unsigned int *count,
                          uint32_t *kept_idx)
{
    for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; p < n;
         p += (uint64_t)gridDim.x * blockDim.x) {
        if (logits[p] >= thr) {
            const unsigned int slot = atomicAdd(count, 1u);
            kept_idx[slot] = (uint32_t)p;
        }
    }
}

__global__ void k_gather(const pg_pair *pairs, const uint32_t *kept_idx, const unsigned int *count,
                         pg_pair *out)
{
    const unsigned int n = *count;
    for (unsigned int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
        out[q] = pairs[kept_idx[q]];
}

// pruned pairs get an empty result with PG_RF_FILTERED; kept ones their alignment
__global__ void k_scatter(const pg_result *kept_res, const uint32_t *kept_idx, const unsigned int *count,
                          const float *logits, uint64_t n, float thr, pg_result *out)
{
    const unsigned int nk = *count;
    for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; p < n;
         p += (uint64_t)gridDim.x * blockDim.x) {
        if (logits[p] < thr) {
            pg_result o;
            o.score = 0; o.aln_len = 0; o.matches = 0; o.gap_opens = 0;
            o.beg_h = o.end_h = o.beg_v = o.end_v = 0;
            o.identity = 0.f; o.score_aln = 0.f; o.seed_used = 0;
            o.flags = PG_RF_EMPTY | PG_RF_FILTERED; o.pad = 0; o.cells = 0;
            out[p] = o;
        }
    }
    for (unsigned int q = blockIdx.x * blockDim.x + threadIdx.x; q < nk; q += gridDim.x * blockDim.x)
        out[kept_idx[q]] = kept_res[q];
}

}  // namespace

struct pg_filter {
    int device = 0;
    float *d_P = nullptr, *d_G = nullptr, *d_M1 = nullptr, *d_M2 = nullptr;  // G has NPARAM+1 (loss)
    int step = 0;
    int nsm = 0;
    // per-call scratch
    float4 *d_rcomp = nullptr, *d_ccomp = nullptr;
    uint64_t comp_cap_r = 0, comp_cap_c = 0;
    __nv_bfloat16 *d_X = nullptr;
    float *d_logit = nullptr;
    uint32_t *d_idx = nullptr;
    unsigned int *d_cnt = nullptr;
    pg_pair *d_kept = nullptr;
    pg_result *d_kres = nullptr;
    int *d_status = nullptr;
    uint64_t cap = 0;
};

extern "C" {

int pg_filter_create(int device, uint64_t seed, pg_filter **out)
{
    if (!out) return pg_internal_fail(PG_ERR_ARG, "pg_filter_create: null output");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
        return pg_internal_fail(PG_ERR_NODEV, "pg_filter_create: no such device");
    FCU(cudaSetDevice(device));
    pg_filter *f = new pg_filter();
    f->device = device;
    cudaDeviceGetAttribute(&f->nsm, cudaDevAttrMultiProcessorCount, device);
    // He-uniform initialisation from a fixed-seed generator (splitmix64)
    std::vector<float> P(NPARAM, 0.f);
    uint64_t x = seed ^ 0x9e3779b97f4a7c15ull;
    auto unif = [&x]() {
        uint64_t z = (x += 0x9e3779b97f4a7c15ull);
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    };
    const double a1 = std::sqrt(6.0 / NF), a2 = std::sqrt(6.0 / NH), a3 = std::sqrt(3.0 / NH);
    for (int k = 0; k < NH * NF; ++k) P[P_W1 + k] = (float)(a1 * unif());
    for (int k = 0; k < NH * NH; ++k) P[P_W2 + k] = (float)(a2 * unif());
    for (int k = 0; k < NH; ++k) P[P_W3 + k] = (float)(a3 * unif());
    cudaError_t e = cudaMalloc(&f->d_P, NPARAM * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&f->d_G, (NPARAM + 1) * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&f->d_M1, NPARAM * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&f->d_M2, NPARAM * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&f->d_status, sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpy(f->d_P, P.data(), NPARAM * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(f->d_G, 0, (NPARAM + 1) * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(f->d_M1, 0, NPARAM * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(f->d_M2, 0, NPARAM * sizeof(float));
    if (e != cudaSuccess) {
        pg_filter_destroy(f);
        return pg_internal_fail(e == cudaErrorMemoryAllocation ? PG_ERR_OOM : PG_ERR_CUDA,
                                cudaGetErrorString(e));
    }
    *out = f;
    return PG_OK;
}

void pg_filter_destroy(pg_filter *f)
{
    if (!f) return;
    cudaSetDevice(f->device);
    cudaFree(f->d_P); cudaFree(f->d_G); cudaFree(f->d_M1); cudaFree(f->d_M2);
    cudaFree(f->d_rcomp); cudaFree(f->d_ccomp); cudaFree(f->d_X); cudaFree(f->d_logit);
    cudaFree(f->d_idx); cudaFree(f->d_cnt); cudaFree(f->d_kept); cudaFree(f->d_kres);
    cudaFree(f->d_status);
    delete f;
}

int pg_filter_params(pg_filter *f, float *host, int get)
{
    if (!f || !host) return pg_internal_fail(PG_ERR_ARG, "pg_filter_params: null argument");
    FCU(cudaSetDevice(f->device));
    if (get) FCU(cudaMemcpy(host, f->d_P, NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
    else FCU(cudaMemcpy(f->d_P, host, NPARAM * sizeof(float), cudaMemcpyHostToDevice));
    return PG_OK;
}

int pg_filter_features(pg_filter *f, pg_ctx *ctx, const pg_pair *d_pairs, uint64_t n,
                       uint64_t bl_roffset, uint64_t bl_coffset, void *d_features, void *stream)
{
    if (!f || !ctx || (n && (!d_pairs || !d_features)))
        return pg_internal_fail(PG_ERR_ARG, "pg_filter_features: bad argument");
    const uint8_t *rseq, *cseq;
    const uint64_t *roffs, *coffs;
    uint64_t nr, nc;
    int dev, mode;
    void *cst;
    int rc = pg_internal_seqs(ctx, &rseq, &roffs, &nr, &cseq, &coffs, &nc, &dev, &cst, &mode);
    if (rc) return rc;
    const int8_t *d_sm = nullptr;
    rc = pg_internal_score(ctx, &d_sm);
    if (rc) return rc;
    FCU(cudaSetDevice(f->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : (cudaStream_t)cst;
    if (nr > f->comp_cap_r) {
        cudaFree(f->d_rcomp); f->d_rcomp = nullptr; f->comp_cap_r = 0;
        FCU(cudaMalloc(&f->d_rcomp, nr * sizeof(float4)));
        f->comp_cap_r = nr;
    }
    if (nc > f->comp_cap_c) {
        cudaFree(f->d_ccomp); f->d_ccomp = nullptr; f->comp_cap_c = 0;
        FCU(cudaMalloc(&f->d_ccomp, nc * sizeof(float4)));
        f->comp_cap_c = nc;
    }
    const int grid = f->nsm * 8;
    k_composition<<<grid, 256, 0, st>>>(rseq, roffs, nr, f->d_rcomp);
    // a block of the search against itself has one set on both sides
    const bool same = rseq == cseq && roffs == coffs && nr == nc;
    if (!same) k_composition<<<grid, 256, 0, st>>>(cseq, coffs, nc, f->d_ccomp);
    FCU(cudaMemsetAsync(f->d_status, 0, sizeof(int), st));
    if (n) k_features<<<grid, 256, 0, st>>>(d_pairs, n, bl_roffset, bl_coffset, rseq, roffs, nr,
                                           cseq, coffs, nc, d_sm, f->d_rcomp, same ? f->d_rcomp : f->d_ccomp,
                                           (__nv_bfloat16 *)d_features, f->d_status);
    FCU(cudaGetLastError());
    int status = 0;
    FCU(cudaMemcpyAsync(&status, f->d_status, sizeof status, cudaMemcpyDeviceToHost, st));
    FCU(cudaStreamSynchronize(st));
    if (status) return pg_internal_fail(PG_ERR_ARG, "pg_filter_features: pair index out of range");
    return PG_OK;
}

int pg_filter_predict(pg_filter *f, const void *d_features, uint64_t n, float *d_logits, void *stream)
{
    if (!f || (n && (!d_features || !d_logits))) return pg_internal_fail(PG_ERR_ARG, "pg_filter_predict: bad argument");
    if (!n) return PG_OK;
    FCU(cudaSetDevice(f->device));
    const uint64_t tiles = (n + 15) / 16;
    const uint64_t blocks = std::min<uint64_t>((tiles + FWARPS - 1) / FWARPS, (uint64_t)f->nsm * 8);
    k_mlp_forward<<<(unsigned)blocks, FWARPS * 32, 0, (cudaStream_t)stream>>>(
        f->d_P, (const __nv_bfloat16 *)d_features, n, d_logits);
    FCU(cudaGetLastError());
    return PG_OK;
}

int pg_filter_gradients(pg_filter *f, const void *d_features, const float *d_labels,
                        const float *d_weights, uint64_t n, float *host_grad_and_loss, void *stream)
{
    if (!f || !n || !d_features || !d_labels || !d_weights)
        return pg_internal_fail(PG_ERR_ARG, "pg_filter_gradients: bad argument");
    FCU(cudaSetDevice(f->device));
    cudaStream_t st = (cudaStream_t)stream;
    FCU(cudaMemsetAsync(f->d_G, 0, (NPARAM + 1) * sizeof(float), st));
    const uint64_t blocks = std::min<uint64_t>((n + FROWS - 1) / FROWS, (uint64_t)f->nsm * 2);
    k_mlp_backward<<<(unsigned)blocks, FWARPS * 32, 0, st>>>(
        f->d_P, (const __nv_bfloat16 *)d_features, d_labels, d_weights, n, 1.0f / (float)n, f->d_G);
    FCU(cudaGetLastError());
    if (host_grad_and_loss) {
        FCU(cudaMemcpyAsync(host_grad_and_loss, f->d_G, (NPARAM + 1) * sizeof(float),
                            cudaMemcpyDeviceToHost, st));
        FCU(cudaStreamSynchronize(st));
    }
    return PG_OK;
}

int pg_filter_train_step(pg_filter *f, const void *d_features, const float *d_labels,
                         const float *d_weights, uint64_t n, float lr, float *loss, void *stream)
{
    int rc = pg_filter_gradients(f, d_features, d_labels, d_weights, n, nullptr, stream);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    float l = 0.f;
    if (loss) FCU(cudaMemcpyAsync(&l, f->d_G + NPARAM, sizeof(float), cudaMemcpyDeviceToHost, st));
    f->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)f->step), c2 = 1.f - std::pow(b2, (float)f->step);
    k_adam<<<(NPARAM + 255) / 256, 256, 0, st>>>(f->d_P, f->d_G, f->d_M1, f->d_M2, lr, b1, b2, 1e-8f, c1, c2);
    FCU(cudaGetLastError());
    if (loss) {
        FCU(cudaStreamSynchronize(st));
        *loss = l;
    }
    return PG_OK;
}

int pg_align_filtered(pg_ctx *ctx, pg_filter *f, float threshold, const pg_pair *d_pairs, uint64_t n,
                      uint64_t bl_roffset, uint64_t bl_coffset, pg_result *d_out, void *stream,
                      uint64_t *kept)
{
    if (!ctx || !f || (n && (!d_pairs || !d_out))) return pg_internal_fail(PG_ERR_ARG, "pg_align_filtered: bad argument");
    if (kept) *kept = 0;
    if (!n) return PG_OK;
    FCU(cudaSetDevice(f->device));
    if (n > f->cap) {
        cudaFree(f->d_X); cudaFree(f->d_logit); cudaFree(f->d_idx); cudaFree(f->d_kept); cudaFree(f->d_kres);
        f->d_X = nullptr; f->d_logit = nullptr; f->d_idx = nullptr; f->d_kept = nullptr; f->d_kres = nullptr;
        f->cap = 0;
        FCU(cudaMalloc(&f->d_X, n * NF * sizeof(__nv_bfloat16)));
        FCU(cudaMalloc(&f->d_logit, n * sizeof(float)));
        FCU(cudaMalloc(&f->d_idx, n * sizeof(uint32_t)));
        FCU(cudaMalloc(&f->d_kept, n * sizeof(pg_pair)));
        FCU(cudaMalloc(&f->d_kres, n * sizeof(pg_result)));
        f->cap = n;
    }
    if (!f->d_cnt) FCU(cudaMalloc(&f->d_cnt, sizeof(unsigned int)));
    cudaStream_t st = (cudaStream_t)stream;
    int rc = pg_filter_features(f, ctx, d_pairs, n, bl_roffset, bl_coffset, f->d_X, stream);
    if (rc) return rc;
    rc = pg_filter_predict(f, f->d_X, n, f->d_logit, stream);
    if (rc) return rc;
    FCU(cudaMemsetAsync(f->d_cnt, 0, sizeof(unsigned int), st));
    const int grid = f->nsm * 8;
    k_compact<<<grid, 256, 0, st>>>(f->d_logit, n, threshold, f->d_cnt, f->d_idx);
    k_gather<<<grid, 256, 0, st>>>(d_pairs, f->d_idx, f->d_cnt, f->d_kept);
    unsigned int nk = 0;
    FCU(cudaMemcpyAsync(&nk, f->d_cnt, sizeof nk, cudaMemcpyDeviceToHost, st));
    FCU(cudaStreamSynchronize(st));
    if (nk) {
        rc = pg_align_device(ctx, f->d_kept, nk, bl_roffset, bl_coffset, f->d_kres, stream);
        if (rc) return rc;
    }
    k_scatter<<<grid, 256, 0, st>>>(f->d_kres, f->d_idx, f->d_cnt, f->d_logit, n, threshold, d_out);
    FCU(cudaGetLastError());
    if (kept) *kept = nk;
    return PG_OK;
}

int pg_filter_nparams(void) { return NPARAM; }

}  // extern "C"
