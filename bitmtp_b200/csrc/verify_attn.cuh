// Block-verify attention over the shared KV buffer: one launch per layer for scores, softmax and numerators, whose split-KV
// partials are merged in the same launch (rows wanted) or by the one that quantises the rows (INT8 codes wanted).
//
// Replaces, for one layer of one replay, the attention of Attention.forward_sdlm_graph_kernel
// (src/bonsai_sft/gpu/model.py:989-1004: flex_attention closure or matmul/softmax/matmul and the
// permute back to [M, q_dim]) together with the additive mask tensor the host rebuilds before every
// replay (src/bonsai_sft/gpu/fast_runtime.py:345-372, 391-465) and, in the ROPE build, the q/k head
// norm, RoPE and KV append of _fused_qkv_qknorm_rope_kv_write (model.py:388-436).  Differences in
// kind, not in result:
//   * visibility is evaluated from (role, cache_len, n_pend) held in device memory (bm_visible in
//     bm_math.h), so nothing is rebuilt on the host and a captured graph serves every cache length;
//   * only history rows [0, cache_len) and the M rows of this replay are read, not the whole padded
//     buffer of sigma + M rows;
//   * the keys are cut into super-chunks of 128 (four sub-chunks of 32); one CTA serves one
//     (super-chunk, kv head, group of up to 16 query vectors), its 8 warps = 4 sub-chunks x 2 query
//     groups; the CTA merges its four sub-chunk partials in shared memory into one partial
//     per query vector, and the super-chunk partials are merged by whoever the build names (kMerge...).
//
// Arithmetic and order: see bmo_attention in oracle/bm_oracle.c; the two agree bit for bit.  All
// accumulation is fp32 on the CUDA cores in a fixed order; tensor-core accumulation order is not
// specified by the hardware documents and could not be mirrored on the CPU.
//
// Scratch (caller-allocated, bm_verify_attention_scratch_bytes; zero before the first call, the
// kernel leaves its counters zero):
//   1024 bytes                 224 ticket counters (rows wanted)
//   pm, pl fp32 [M, H, NJ]      super-chunk max / sum
//   po   fp32 [M, H, NJ, 128]   super-chunk numerators
//   rows bf16 [M, H*128]        attention rows between merge and codes (above 32 heads) when the caller passes no att_out
//   NJ = ceil(sigma/128) + 1; super-chunk NJ-1 holds the rows appended by this replay.
#pragma once

#include <algorithm>

#include "bm_common.cuh"
#include "fused_ops.cuh"

namespace bm {

constexpr int kAttnThreads = 256, kAttnWarps = kAttnThreads / 32;
constexpr int kAttnSub = BM_ATTN_SUPER / BM_ATTN_CHUNK;   // sub-chunks per super-chunk (4)
constexpr int kKeyStride = 136;        // bf16 elements per staged key row (128 + 8 pad = 272 bytes)
constexpr int kWeightStride = 8;        // fp32 softmax weights per key and warp (a warp serves up to 8 query vectors)
constexpr int kAttnHeaderBytes = 1024;
constexpr int kAttnTickets = 224;      // counters in the header
constexpr int kAttnMaxHeads = 1024;    // heads of one call (keeps the split's products in an int)
constexpr int kAttnMaxNV = 4;          // query vectors per half warp; a CTA serves up to 4 * kAttnMaxNV
constexpr int kAttnMaxNJ = 64;         // super-chunk partials one merging warp handles (2 per lane)
constexpr int kAttnMaxCluster = 16;    // super-chunks (CTAs) of one cluster in the cluster build

struct AttnParams {
    const uint16_t *q;        // [M, H, 128] rotated queries (plain build)
    const uint16_t *k_base;   // [Hkv, kv_rows, 128]
    const uint16_t *v_base;
    const StepState *state;
    int M, H, Hkv, kv_rows, sigma, NJ;
    unsigned int *tickets;    // [Hkv * z_max] a replay or slab, zero between launches
    unsigned int *amax;       // [M] row absmax bits, gathered by atomic max (zero on entry)
    float *pm, *pl, *po;
    uint16_t *att;            // [M, H*128] bf16 attention output
    int pdl;
    // ROPE build: the qkv projection output and what the rotation needs
    const uint16_t *xqkv;            // [M, (H + 2 Hkv) * 128] bf16
    const uint16_t *q_w, *k_w;       // head-norm weights, bf16 [128]
    const uint16_t *cos_t, *sin_t;   // bf16 [max_pos, 128]
    const int64_t *positions;        // [M]
    uint16_t *k_out, *v_out;         // the layer's planes (same memory as k_base / v_base)
    float eps;
    // Prompt mode (plain build only; slab_rows > 0): M prompt rows whose K / V already sit at rows
    // [slab_hist0, slab_hist0 + M) of the planes are served as AR-causal slabs of slab_rows rows: slab s
    // sees history [0, slab_hist0 + s * slab_rows) and its own rows.  blockIdx.x runs over the
    // (slab, super-chunk) pairs in slab order; `state` is not read; q, att, amax and the partials are
    // indexed by prompt row.
    int slab_rows, slab_hist0;
    int z_max;       // query groups the tickets are laid out for
    uint8_t pick[kAttnMaxNJ];        // replays: query vectors per half warp for n history super-chunks (attn_split)
};

__host__ __device__ inline size_t attn_scratch_bytes(int M, int H, int sigma) {
    const size_t NJ = (size_t)(sigma + BM_ATTN_SUPER - 1) / BM_ATTN_SUPER + 1;
    return kAttnHeaderBytes + (size_t)M * H * NJ * 4 * 2 + (size_t)M * H * NJ * 128 * 4 + (size_t)M * H * 128 * 2;
}

// A CTA serves 4 * nv query vectors, nv = 1 .. kAttnMaxNV: the warps of a sub-chunk split them in two groups, a warp's
// half warps in two again.  Shared memory is what level 0 waits for (attn_level0), and a CTA reads its keys once for all its
// vectors, so wide CTAs do less in all; but a launch is over when its fullest SM is.  So the widest split follows from the
// number of query vectors, and every CTA of a replay looks up, by the history length that it reads on the device, the split
// that leaves the least on the fullest SM.  Which CTA serves a vector changes nothing in the arithmetic.
__host__ __device__ inline int attn_nv(int QV) { return QV >= 4 * kAttnMaxNV ? kAttnMaxNV : (QV + 3) / 4; }
__host__ __device__ inline int attn_groups(int QV, int nv) { return (QV + 4 * nv - 1) / (4 * nv); }

// The splits of a replay over a segment of NJ - 1 history super-chunks.  The cost of n of them at a split is the time of the
// fullest SM, in units of about half a microsecond: a CTA alone takes 2 nv + 5 (7.4 us to codes with nv = 2, 9.2 with 3, 10.5
// with 4); two that share an SM overlap, 3 nv + 5 for the pair; an odd one after pairs takes 0.6 of a pair.  Where no split
// needs more CTAs than SMs, only such are taken and each CTA gets an SM to itself (codes only: `rows` calls, whose last launch
// merges, do better with two narrow CTAs an SM; held to one, 50 of 781 of them were 3 to 28 % slower than before there were wide
// CTAs, now 15, by 10 % at most).  The grid is that of the largest pick, not
// of the finest split: CTAs without work delayed the others by up to 2.6 us (2112 CTAs, 256 of them working).
// Fitted to the attention to codes for every nv, over 1566 calls (five head counts, 2 to 32 rows, 1 to 32 super-chunks, segments of
// 256 to 4096): 0.2 % over the fastest split on average, where the rule before (w (2 nv + 3) for w CTAs, grid of the finest split) was
// 6 % over it.  us then / now: 16 / 8 heads, width 9 behind 6 super-chunks of 1024 keys 9.1 / 9.1, behind 8 of 4096 13.2 / 10.9; width 16
// behind 8 of 1024 12.6 / 11.6, behind 8 of 4096 15.5 / 11.6; 32 / 8 heads, width 9 behind 3 of 1024 11.4 / 9.3, width 16 13.7 / 10.6.
struct AttnSplit {
    uint8_t pick[kAttnMaxNJ];   // nv for n history super-chunks
    bool single;                // the working CTAs never exceed the SMs
    int groups, pairs;          // most query groups, most (super-chunk, query group) pairs of any n
};
inline AttnSplit attn_split(int NJ, int QV, int Hkv, int sms, bool rows) {
    AttnSplit r = {};
    const int widest = attn_nv(QV);
    r.single = !rows && NJ * Hkv * attn_groups(QV, widest) <= sms;
    for (int n = 0; n < NJ; ++n) {
        int best = 0, cost = 0;
        for (int nv = 1; nv <= widest; ++nv) {
            const int ctas = (n + 1) * Hkv * attn_groups(QV, nv), w = (ctas + sms - 1) / sms;      // CTAs of the fullest SM
            if (r.single && ctas > sms) continue;
            const int c = w == 1 ? 10 * (2 * nv + 5) : (3 * nv + 5) * (w / 2 * 10 + w % 2 * 6);
            if (best == 0 || c < cost) { best = nv; cost = c; }
        }
        r.pick[n] = (uint8_t)best;
        r.groups = std::max(r.groups, attn_groups(QV, best));
        r.pairs = std::max(r.pairs, (n + 1) * attn_groups(QV, best));
    }
    // Up to 16 vectors a kv head, a CTA an SM: the finest split's grid, CTAs without work and all.  1.7B replays in a segment of
    // 1024 with the smaller grid / this, us: width 5 behind 300 and 500 keys 807 / 803 and 819 / 809, width 6 behind 300 827 / 815,
    // width 8 behind 120 830 / 824, behind 300 847 / 842.  Wider ones: level (width 9), or now one, now the other (width 16).
    if (r.single && attn_groups(QV, widest) == 1) r.pairs = NJ * attn_groups(QV, 1);
    return r;
}

// K (padded rows; after level 0 its space takes the sub-chunk numerators), V, queries, weights, sub-chunk max / sum.
// `slab`: kMergeHistory and kMergeHistoryFew, whose own rows are one sub-chunk (the K rows' space is then that of the numerators).
__host__ __device__ constexpr int attn_key_bytes(int nv, bool slab) {
    return slab ? kAttnSub * 4 * nv * 128 * 4 : BM_ATTN_SUPER * kKeyStride * 2;
}
__host__ __device__ constexpr int attn_value_bytes(bool slab) { return (slab ? BM_ATTN_CHUNK : BM_ATTN_SUPER) * 128 * 2; }
__host__ __device__ inline size_t attn_smem_bytes(int nv, bool slab = false) {
    const size_t QC = 4 * (size_t)nv;
    return (size_t)attn_key_bytes(nv, slab) + attn_value_bytes(slab) + QC * kKeyStride * 2 +
           (size_t)kAttnWarps * BM_ATTN_CHUNK * kWeightStride * 4 + (size_t)kAttnSub * QC * 2 * 4;
}
static_assert(BM_ATTN_CHUNK * kKeyStride * 2 <= attn_key_bytes(2, true), "a slab's K rows fit");
static_assert(kAttnSub * 4 * kAttnMaxNV * 128 * 4 <= BM_ATTN_SUPER * kKeyStride * 2, "sub-chunk numerators fit the K rows");

// History length of this replay.  The record is written by other launches (or by the caller through
// the C ABI), so it is clamped to [0, sigma] before anything is indexed with it: the scratch, the
// shared-memory arrays and the K/V planes are all sized from sigma.  Identity for every valid record.
__device__ __forceinline__ int attn_cache_len(const AttnParams &p) {
    return min(max(p.state->cache_len, 0), p.sigma);
}

// q/k head norm + RoPE of one 128-wide head vector by one warp, as qknorm_rope_kvappend_kernel does it:
// lane l owns elements 4l..4l+3 (`raw`: its four bf16 inputs, `wraw`: its norm weights, `craw` / `sraw`:
// its cos / sin table entries), the RoPE partner lives in lane l ^ 16.  Returns the sums before
// the final bf16 rounding.
__device__ __forceinline__ float4 rope_head_vector(uint2 raw, uint2 wraw, uint2 craw, uint2 sraw, float eps, int lane) {
    const float x[4] = {__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u),
                        __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u)};
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) acc = fmaf(x[i], x[i], acc);
    const float total = warp_sum_butterfly(acc);
    const float r = bm_rsqrtf((0.0f + total) / 128.0f + eps);
    const float wv[4] = {__uint_as_float(wraw.x << 16), __uint_as_float(wraw.x & 0xffff0000u),
                         __uint_as_float(wraw.y << 16), __uint_as_float(wraw.y & 0xffff0000u)};
    const float c[4] = {__uint_as_float(craw.x << 16), __uint_as_float(craw.x & 0xffff0000u),
                        __uint_as_float(craw.y << 16), __uint_as_float(craw.y & 0xffff0000u)};
    const float sn[4] = {__uint_as_float(sraw.x << 16), __uint_as_float(sraw.x & 0xffff0000u),
                         __uint_as_float(sraw.y << 16), __uint_as_float(sraw.y & 0xffff0000u)};
    float n[4], o[4];
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        float a = x[i] * r, b = x[i + 1] * r;
        bf16_round_pair(a, b);
        n[i] = wv[i] * a;
        n[i + 1] = wv[i + 1] * b;
        bf16_round_pair(n[i], n[i + 1]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float partner = __shfl_xor_sync(0xffffffffu, n[i], 16);
        const float rot = lane < 16 ? -partner : partner;
        o[i] = bm_bf16_rn(n[i] * c[i]) + bm_bf16_rn(rot * sn[i]);
    }
    return make_float4(o[0], o[1], o[2], o[3]);
}
// The same as a call, for the builds of more than four query vectors: up to six vectors a warp would be 30 KB of instructions
// that every launch fetches anew.
__device__ __noinline__ float4 rope_head_vector_call(uint2 raw, uint2 wraw, uint2 craw, uint2 sraw, float eps, int lane) {
    return rope_head_vector(raw, wraw, craw, sraw, eps, lane);
}

// Two fp32 values in a register pair, and the packed arithmetic on them: each half rounds as the scalar instruction does,
// at the same rate per value and half the issue slots.
typedef unsigned long long PaPair;
__device__ __forceinline__ PaPair pa_pack(float lo, float hi) {
    PaPair v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void pa_unpack(PaPair v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
// bm_expf for x <= 0, infinities or NaN, without its branches and the two conversions that issue at a quarter of the
// rate; the same values: adding 1.5 * 2^23 rounds |t| < 2^22 to the nearest even integer and leaves it in the low bits,
// and the exponent, -126 .. 0, goes in with one exact step.  For the attention, whose
// arguments are differences from a maximum.
__device__ __forceinline__ float pa_expf(float x) {
    const float biased = x * 1.44269504088896341f + 12582912.0f;
    const float n = biased - 12582912.0f;
    float r = fmaf(n, -0.693145751953125f, x);
    r = fmaf(n, -1.42860682030941723e-6f, r);
    float p = 1.3888889225e-3f;
    p = fmaf(p, r, 8.3333337680e-3f);
    p = fmaf(p, r, 4.1666667908e-2f);
    p = fmaf(p, r, 1.6666667163e-1f);
    p = fmaf(p, r, 0.5f);
    p = fmaf(p, r, 1.0f);
    p = fmaf(p, r, 1.0f);
    const float e = p * __uint_as_float((__float_as_uint(biased) - 0x4B400000u + 127u) << 23);
    return x >= -87.0f ? e : (x != x ? x : 0.0f);
}

__device__ __forceinline__ PaPair pa_add2(PaPair a, PaPair b) { PaPair d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ PaPair pa_mul2(PaPair a, PaPair b) { PaPair d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ PaPair pa_fma2(PaPair a, PaPair b, PaPair c) { PaPair d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ PaPair pa_both(float v) { return pa_pack(v, v); }

// Level 0: one warp, one sub-chunk of up to 32 keys, 2 * NVH query vectors; half warp h serves vectors 2t + h.
// What bounds it: the fma pipe and what feeds it.  A lane holds two keys (kl and kl + 16) against its half warp's vectors and
// queries are staged as the bf16 values that they are, so a load from shared memory, whose return path passes 128 bytes a
// cycle and SM also where all lanes read the same ones, feeds 16 fmas and more (one key per lane and fp32 queries: four).
// An SM takes 1.0 us and another 1.1 us per four vectors (128 keys); the fmas of four vectors are 0.5 us at their full rate.
// Queries staged twice over for packed fmas (twice the loads), 16 warps with half the vectors each, and the next loads
// requested a step ahead were level or slower.
// Scores and weight sums are the oracle's: a score is one fma chain in ascending d, the sum over the 32 keys the butterfly
// 16, 8, 4, 2, 1 whose first step is inside the lane.
//   Ks / Vs   the sub-chunk's rows in shared memory (Ks padded to kKeyStride);  Qs the warp's query rows (kKeyStride)
//   Pw        [32][kWeightStride] fp32 weights of this warp
//   hidden    history sub-chunks: the one key (0..31) that no row sees, or a number outside
//   oc, mc, lc  numerators [2 NVH][128], maxima and sums of this warp's vectors; oc overlays K rows that other warps may
//             still be reading, so it is written after the CTA barrier inside
// All warps of the CTA call this together (cn <= 0: nothing of the sub-chunk exists).
struct AttnView {
    int fresh, role, sigma, cache_len, n_pend, P, M, q_lo, key0;      // q_lo: first vector of the warp; key0: first key
};
template <int NVH>
__device__ __forceinline__ void attn_level0(const uint16_t *Ks, const uint16_t *Vs, const uint16_t *Qs, float *Pw,
                                            const AttnView &a, int cn, int hidden, int lane, float *mc, float *lc, float *oc) {
    const int kl = lane & 15, h = lane >> 4;
    PaPair o[NVH][4];                                                  // vectors (2i, 2i + 1), dims 4 lane + e
#pragma unroll
    for (int i = 0; i < NVH; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = 0ull;
    if (cn > 0) {
        float s0[NVH], s1[NVH];
#pragma unroll
        for (int t = 0; t < NVH; ++t) s0[t] = s1[t] = 0.0f;
        const uint16_t *k0 = Ks + (kl < cn ? kl : 0) * kKeyStride, *k1 = Ks + (kl + 16 < cn ? kl + 16 : 0) * kKeyStride;
        const uint16_t *qr = Qs + h * kKeyStride;
#pragma unroll 2
        for (int u = 0; u < 16; ++u) {
            float ka[8], kb[8];
            unpack8(*reinterpret_cast<const uint4 *>(k0 + 8 * u), ka);
            unpack8(*reinterpret_cast<const uint4 *>(k1 + 8 * u), kb);
#pragma unroll
            for (int t = 0; t < NVH; ++t) {
                float q[8];
                unpack8(*reinterpret_cast<const uint4 *>(qr + 2 * t * kKeyStride + 8 * u), q);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    s0[t] = fmaf(q[e], ka[e], s0[t]);
                    s1[t] = fmaf(q[e], kb[e], s1[t]);
                }
            }
        }
        bool v0[NVH], v1[NVH];
        float m[NVH], l[NVH];
#pragma unroll
        for (int t = 0; t < NVH; ++t) {
            v0[t] = kl < cn && kl != hidden;
            v1[t] = kl + 16 < cn && kl + 16 != hidden;
            if (a.fresh) {
                const int v = a.q_lo + 2 * t + h, row = v - v / a.M * a.M;
                v0[t] = kl < cn && bm_visible(a.role, row, a.key0 + kl, a.sigma, a.cache_len, a.n_pend, a.P);
                v1[t] = kl + 16 < cn && bm_visible(a.role, row, a.key0 + kl + 16, a.sigma, a.cache_len, a.n_pend, a.P);
            }
            s0[t] = v0[t] ? s0[t] * 0.08838834764831845f : -INFINITY;
            s1[t] = v1[t] ? s1[t] * 0.08838834764831845f : -INFINITY;
            m[t] = fmaxf(s0[t], s1[t]);
        }
#pragma unroll
        for (int off = 8; off > 0; off >>= 1)
#pragma unroll
            for (int t = 0; t < NVH; ++t) m[t] = fmaxf(m[t], __shfl_xor_sync(0xffffffffu, m[t], off));
#pragma unroll
        for (int t = 0; t < NVH; ++t) {
            const float e0 = pa_expf(s0[t] - m[t]), e1 = pa_expf(s1[t] - m[t]), p0 = v0[t] ? e0 : 0.0f, p1 = v1[t] ? e1 : 0.0f;
            l[t] = p0 + p1;
            Pw[kl * kWeightStride + 2 * t + h] = bm_bf16_rn(p0);
            Pw[(kl + 16) * kWeightStride + 2 * t + h] = bm_bf16_rn(p1);
        }
#pragma unroll
        for (int off = 8; off > 0; off >>= 1)
#pragma unroll
            for (int t = 0; t < NVH; ++t) l[t] = l[t] + __shfl_xor_sync(0xffffffffu, l[t], off);
        if (kl == 0) {
#pragma unroll
            for (int t = 0; t < NVH; ++t) {
                mc[2 * t + h] = m[t];
                lc[2 * t + h] = l[t];
            }
        }
        __syncwarp();
        // numerators: lane owns dims 4 lane .. 4 lane + 3 of all the warp's vectors, chains in ascending key order
        for (int cb = 0; cb < cn; cb += 4) {
            uint2 raw[4];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
                // keys past cn have weight 0 and are given value 0
                raw[cc] = cb + cc < cn ? *reinterpret_cast<const uint2 *>(Vs + (cb + cc) * 128 + 4 * lane) : make_uint2(0u, 0u);
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const float v[4] = {__uint_as_float(raw[cc].x << 16), __uint_as_float(raw[cc].x & 0xffff0000u),
                                    __uint_as_float(raw[cc].y << 16), __uint_as_float(raw[cc].y & 0xffff0000u)};
                const float *wp = Pw + (cb + cc) * kWeightStride;
                PaPair w[4];
                if (NVH > 1) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(wp);
                    w[0] = x.x; w[1] = x.y;
                } else {
                    w[0] = *reinterpret_cast<const PaPair *>(wp);
                }
                if (NVH > 3) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(wp + 4);
                    w[2] = x.x; w[3] = x.y;
                } else if (NVH > 2) {
                    w[2] = *reinterpret_cast<const PaPair *>(wp + 4);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const PaPair vv = pa_pack(v[e], v[e]);
#pragma unroll
                    for (int i = 0; i < NVH; ++i) o[i][e] = pa_fma2(w[i], vv, o[i][e]);
                }
            }
        }
    } else if (lane < 2 * NVH) {
        mc[lane] = -INFINITY;
        lc[lane] = 0.0f;
    }
    __syncthreads();                                                   // every warp is done with the K rows
#pragma unroll
    for (int i = 0; i < NVH; ++i) {
        float x[4], y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) pa_unpack(o[i][e], x[e], y[e]);
        *reinterpret_cast<float4 *>(oc + (2 * i) * 128 + 4 * lane) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4 *>(oc + (2 * i + 1) * 128 + 4 * lane) = make_float4(y[0], y[1], y[2], y[3]);
    }
}

// Level 0 where a CTA has one or two query vectors (width 1 of the 1.7B geometry): a warp serves one, a lane holds one key.
// attn_level0 would put both on the first four warps, a half warp each with two keys a lane, and have the others compute
// nothing: twice the chain.  Rows by clusters, 16 / 8 heads, width 1, us that way and this: 5.0 and 4.5 behind 20 keys, 5.7 and
// 5.0 behind 600, 6.3 and 5.6 behind 1000.  Same scores, same sums: the butterfly 16, 8, 4, 2, 1 now crosses lanes in its first
// step too.  a.q_lo: the vector; Qs its row; Pw 32 weights; oc one row.
__device__ __forceinline__ void attn_level0_one(const uint16_t *Ks, const uint16_t *Vs, const uint16_t *Qs, float *Pw,
                                                const AttnView &a, int cn, int hidden, int lane, float *mc, float *lc, float *oc) {
    float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};                             // dims 4 lane + e
    if (cn > 0) {
        float s = 0.0f;
        const uint16_t *kr = Ks + (lane < cn ? lane : 0) * kKeyStride;
#pragma unroll 4
        for (int u = 0; u < 16; ++u) {
            float k[8], q[8];
            unpack8(*reinterpret_cast<const uint4 *>(kr + 8 * u), k);
            unpack8(*reinterpret_cast<const uint4 *>(Qs + 8 * u), q);
#pragma unroll
            for (int e = 0; e < 8; ++e) s = fmaf(q[e], k[e], s);
        }
        const bool seen = lane < cn && (a.fresh ? bm_visible(a.role, a.q_lo - a.q_lo / a.M * a.M, a.key0 + lane, a.sigma,
                                                             a.cache_len, a.n_pend, a.P)
                                                : lane != hidden);
        s = seen ? s * 0.08838834764831845f : -INFINITY;
        const float m = warp_max(s), e = pa_expf(s - m), w = seen ? e : 0.0f, l = warp_sum_butterfly(w);
        Pw[lane] = bm_bf16_rn(w);
        if (lane == 0) { mc[0] = m; lc[0] = l; }
        __syncwarp();
        for (int cb = 0; cb < cn; cb += 4) {
            uint2 raw[4];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
                raw[cc] = cb + cc < cn ? *reinterpret_cast<const uint2 *>(Vs + (cb + cc) * 128 + 4 * lane) : make_uint2(0u, 0u);
            const float4 w4 = *reinterpret_cast<const float4 *>(Pw + cb);
            const float wk[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const float v[4] = {__uint_as_float(raw[cc].x << 16), __uint_as_float(raw[cc].x & 0xffff0000u),
                                    __uint_as_float(raw[cc].y << 16), __uint_as_float(raw[cc].y & 0xffff0000u)};
#pragma unroll
                for (int i = 0; i < 4; ++i) o[i] = fmaf(wk[cc], v[i], o[i]);
            }
        }
    } else if (lane == 0) {
        mc[0] = -INFINITY;
        lc[0] = 0.0f;
    }
    __syncthreads();                                                   // every warp is done with the K rows
    *reinterpret_cast<float4 *>(oc + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
}

// Level 2 of one query vector by one warp: super-chunk partials in ascending order (history chunks 0 .. n_hs - 1, then the
// replay's own rows, chunk NJ - 1), division, bf16 rounding.  pb: the vector's first partial.  OWN: the last partial
// (max own_m, sum own_l, numerators own_o) is in registers.
template <bool OWN>
__device__ __forceinline__ void attn_merge_vector(const float *pm, const float *pl, const float *po, size_t pb, int n_hs, int NJ,
                                                  int lane, float own_m, float own_l, float4 own_o, float (&v)[4]) {
    const int nv = n_hs + 1;
    constexpr int kBatch = 8;
    float4 part[kBatch];
    // the first batch of numerators is requested together with the maxima and sums: one round trip
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
        const int j = i < n_hs ? i : NJ - 1;
        part[i] = OWN && i == n_hs ? own_o
                  : i < nv ? __ldcg(reinterpret_cast<const float4 *>(po + (pb + j) * 128 + 4 * lane))
                           : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f;
    if (OWN && lane == n_hs) {
        m0 = own_m;
        l0 = own_l;
    } else if (lane < nv) {
        const int j = lane < n_hs ? lane : NJ - 1;
        m0 = __ldcg(pm + pb + j);
        l0 = __ldcg(pl + pb + j);
    }
    if (OWN && lane + 32 == n_hs) {
        m1 = own_m;
        l1 = own_l;
    } else if (lane + 32 < nv) {
        const int j = lane + 32 < n_hs ? lane + 32 : NJ - 1;
        m1 = __ldcg(pm + pb + j);
        l1 = __ldcg(pl + pb + j);
    }
    const float gmax = warp_max(fmaxf(m0, m1));
    const float w0 = m0 > -INFINITY ? pa_expf(m0 - gmax) : 0.0f;
    const float w1 = m1 > -INFINITY ? pa_expf(m1 - gmax) : 0.0f;
    float l = 0.0f, o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int b0 = 0; b0 < nv; b0 += kBatch) {
        if (b0 > 0) {
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int c = b0 + i;
                const int j = c < n_hs ? c : NJ - 1;
                part[i] = OWN && c == n_hs ? own_o
                          : c < nv ? __ldcg(reinterpret_cast<const float4 *>(po + (pb + j) * 128 + 4 * lane))
                                   : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const int c = b0 + i;
            if (c < nv) {                                          // warp-uniform
                const float w = __shfl_sync(0xffffffffu, c < 32 ? w0 : w1, c & 31);
                const float lj = __shfl_sync(0xffffffffu, c < 32 ? l0 : l1, c & 31);
                l = fmaf(lj, w, l);
                o[0] = fmaf(part[i].x, w, o[0]);
                o[1] = fmaf(part[i].y, w, o[1]);
                o[2] = fmaf(part[i].z, w, o[2]);
                o[3] = fmaf(part[i].w, w, o[3]);
            }
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = bm_bf16_rn(o[e] / l);
}
__device__ __forceinline__ uint2 attn_pack_row(const float (&v)[4]) {
    return make_uint2(bf16_pair(v[0], v[1]), bf16_pair(v[2], v[3]));
}
__device__ __forceinline__ float attn_row_amax(const float (&v)[4]) {
    return warp_max(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
}

// Who merges the super-chunk partials of a query vector (level 2).
//   kMergeTicket   the last CTA of a (kv head, query group) to finish, found by a ticket counter in the scratch
//   kMergeCluster  the NJ CTAs of a (kv head, query group) are one thread-block cluster (launch attribute (NJ, 1, 1), NJ <=
//                  kAttnMaxCluster).  The partials stay in the shared memory of the CTA that made them; the CTA of the
//                  replay's own rows (cluster rank NJ - 1, always working) reads them through distributed shared memory
//                  after one cluster barrier and merges them in the same order, so the fence, the ticket and the read-back
//                  from global memory drop out of the chain.  A second barrier keeps the other CTAs' shared memory alive
//                  until it has been read.  CTAs of super-chunks without rows take part in both barriers and do nothing else.
//   kMergeHistory  prompt mode only: prompt_hist_kernel has made the partials of the history super-chunks.  blockIdx.x is
//                  the slab; its CTAs make the partial of the slab's own rows, keep it in registers and merge at once.  A
//                  build of its own: as a run-time switch it made every other prompt-mode call 3.6 % slower (1 to 9 % over
//                  117 calls of 17 to 512 rows).  It stages 16 keys, not 128, so four CTAs share an SM (512 rows of 16 heads: 70.5
//                  us a call without history, now 62.3), which leaves a thread 64 registers and costs a call of few CTAs 2 us.
//   kMergeHistoryFew  the same, for few CTAs: 79 registers, three CTAs per SM
//   kMergeLater    the next launch (attn_merge_quant_kernel): this one ends with its partials.  A replay wants the rows as
//                  INT8 codes, for which a launch has to follow anyway; the end of a launch is then the only hand-over
//                  (fence, ticket, read-back and row-absmax atomics took 3.4 us of 12.4 at width 16).
// Attention to codes in a chain of such launches, 16 / 8 heads, before (ticket, up to 8 vectors a CTA, two CTAs per SM) and
// now, us: width 16 behind 120 / 300 / 600 / 900 keys 11.0 / 11.4 / 13.4 / 15.8, now 6.3 / 7.7 / 9.4 / 11.6; width 9 behind
// 120 / 600 10.2 / 10.9, now 6.2 / 7.6; 32 / 8 heads, width 16 behind 1100 keys 34.4, now 23.8.
enum : int { kMergeTicket = 0, kMergeCluster = 1, kMergeHistory = 2, kMergeLater = 3, kMergeHistoryFew = 4 };

// 256 threads.  NV: widest split (4 * NV query vectors per CTA); ROPE: queries and the replay's own K/V rows are made here
// from the qkv projection output.  Grid: replays (Hkv, NJ * finest query groups) - the (super-chunk, query group) pairs with
// work are the first in y, so that working CTAs are spread over the SMs and the rest leave; clusters and prompt mode
// (super-chunks or (slab, super-chunk) pairs, Hkv, query groups).
template <int NV, bool ROPE, int MERGE = kMergeTicket>
__global__ void __launch_bounds__(kAttnThreads, MERGE == kMergeHistory ? 4 : 2) attn_fused_kernel(const __grid_constant__ AttnParams p) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ unsigned int sh_ticket;
    constexpr int QC = 4 * NV, NQW = (QC + kAttnWarps - 1) / kAttnWarps;      // vectors per CTA; per warp outside level 0
    constexpr bool CLUSTER = MERGE == kMergeCluster, HIST_DONE = MERGE == kMergeHistory || MERGE == kMergeHistoryFew;
    pdl_launch_dependents();
    // BM_PDL_STABLE_STATE: the step record, the positions and the history rows were written by launches
    // that had completed before this call's chain of overlapped launches began, so they may be read
    // while the predecessor is still running.
    const bool early = (p.pdl & BM_PDL_STABLE_STATE) != 0;
    if (p.pdl && !early) pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // every load here is out before the first is used: record, positions (one a lane) and norm weights in one round trip
    long long pos_lane = 0;
    uint2 qw = make_uint2(0u, 0u), kw = qw;
    if (ROPE) {
        if (lane < p.M) pos_lane = p.positions[lane];
        qw = *reinterpret_cast<const uint2 *>(p.q_w + 4 * lane);
        kw = *reinterpret_cast<const uint2 *>(p.k_w + 4 * lane);
    }
    const bool slab = !ROPE && p.slab_rows > 0, flat = !CLUSTER && !slab;
    const int hk = flat ? blockIdx.x : blockIdx.y;
    int z = blockIdx.z, J = blockIdx.x, M_ = p.M, sigma_ = p.sigma, r0 = 0, cache_len, n_pend, role, P_, nv = NV;
    unsigned int *ticket = p.tickets;
    if (slab) {
        // prompt mode: find this CTA's slab; a slab with history h has ceil(h / 128) + 1 super-chunks
        int s = 0, rem = J, h = p.slab_hist0;
        if (HIST_DONE) {
            s = J;
            h += s * p.slab_rows;
            rem = (h + BM_ATTN_SUPER - 1) / BM_ATTN_SUPER;
        } else for (;;) {
            const int units = (h + BM_ATTN_SUPER - 1) / BM_ATTN_SUPER + 1;
            if (rem < units) break;
            rem -= units;
            ++s;
            h += p.slab_rows;
        }
        r0 = s * p.slab_rows;
        M_ = min(p.slab_rows, p.M - r0);
        cache_len = sigma_ = h;
        n_pend = 0; role = BM_ROLE_AR; P_ = 0;
        J = rem < (h + BM_ATTN_SUPER - 1) / BM_ATTN_SUPER ? rem : p.NJ - 1;
        ticket += (size_t)s * p.Hkv * p.z_max;
        if (M_ <= 0) return;
    } else {
        cache_len = attn_cache_len(p); n_pend = p.state->n_pend; role = p.state->role; P_ = p.state->P;
    }
    const int n_hs = (cache_len + BM_ATTN_SUPER - 1) / BM_ATTN_SUPER;     // history super-chunks with rows
    const int G = p.H / p.Hkv, QV = G * M_, heads = p.H + 2 * p.Hkv;
    if (!slab && NV > 1) nv = min((int)p.pick[n_hs], NV);
    const int qc = 4 * nv;
    if (flat) {
        // the replay's own rows first, then the history, all query groups of a super-chunk together
        const int zn = (QV + qc - 1) / qc, c = (int)blockIdx.y / zn;
        z = (int)blockIdx.y - c * zn;
        if (c > n_hs) return;
        J = c == 0 ? p.NJ - 1 : c - 1;
    }
    ticket += hk * p.z_max + z;
    const bool fresh = J == p.NJ - 1;
    const int q_lo = z * qc;
    if (q_lo >= QV) return;                // a surplus query group: all its CTAs (a whole cluster) leave here
    if (!fresh && J >= n_hs) {
        if (CLUSTER) {                     // a super-chunk without rows: both barrier phases, nothing else
            cluster_arrive(); cluster_wait();
            cluster_arrive(); cluster_wait();
        }
        return;
    }
    const int key0 = fresh ? sigma_ : J * BM_ATTN_SUPER;
    const int nkeys = fresh ? M_ : min(BM_ATTN_SUPER, cache_len - key0);

    uint16_t *Ks = reinterpret_cast<uint16_t *>(dyn);                              // [128][136]
    float *oc = reinterpret_cast<float *>(dyn);                                    // [4][QC][128], over the K rows
    uint16_t *Vs = Ks + attn_key_bytes(NV, HIST_DONE) / 2;                          // [128][128], a slab's [32][128]
    uint16_t *Qs = Vs + attn_value_bytes(HIST_DONE) / 2;                            // [QC][136]
    float *Ps = reinterpret_cast<float *>(Qs + QC * kKeyStride);                    // [8 warps][32 keys][8]
    float *mc = Ps + kAttnWarps * BM_ATTN_CHUNK * kWeightStride;                    // [4][QC]
    float *lc = mc + kAttnSub * QC;                                                 // [4][QC]

    // Nothing below depends on the previous kernel until the wait: history rows, table rows.  The history rows go straight
    // to shared memory (asynchronous 16-byte copies, no registers held; one bulk copy per padded K row took 3 us longer).
    auto copy_rows = [&]() {
        const uint4 *kg = reinterpret_cast<const uint4 *>(p.k_base + ((size_t)hk * p.kv_rows + key0) * 128);
        const uint4 *vg = reinterpret_cast<const uint4 *>(p.v_base + ((size_t)hk * p.kv_rows + key0) * 128);
        for (int i = tid; i < nkeys * 16; i += kAttnThreads) {
            cp_async16(Ks + (i >> 4) * kKeyStride + 8 * (i & 15), kg + i);
            cp_async16(Vs + 8 * i, vg + i);
        }
    };
    if (!fresh) copy_rows();
    // this warp's query vectors (warp, warp + 8) and, in the CTA of the replay's own rows, its
    // share of those rows (m = warp, warp + 8, ...: at most kFreshPerWarp)
    constexpr int kFreshPerWarp = BM_MAX_W / kAttnWarps;
    bool q_live[NQW];
    int qg_[NQW], qm[NQW];
    uint2 qcos[NQW], qsin[NQW], kcos[kFreshPerWarp], ksin[kFreshPerWarp];
#pragma unroll
    for (int k = 0; k < NQW; ++k) {
        const int qi = warp + k * kAttnWarps, qv = q_lo + qi;
        q_live[k] = qi < qc && qv < QV;
        qg_[k] = q_live[k] ? qv / M_ : 0;
        qm[k] = q_live[k] ? qv - qg_[k] * M_ : 0;
        if (ROPE) {
            const size_t pos = (size_t)__shfl_sync(0xffffffffu, pos_lane, qm[k]);
            qcos[k] = qsin[k] = make_uint2(0u, 0u);
            if (q_live[k]) {
                qcos[k] = *reinterpret_cast<const uint2 *>(p.cos_t + pos * 128 + 4 * lane);
                qsin[k] = *reinterpret_cast<const uint2 *>(p.sin_t + pos * 128 + 4 * lane);
            }
        }
    }
    if (ROPE && fresh) {
#pragma unroll
        for (int k = 0; k < kFreshPerWarp; ++k) {
            const int m = warp + k * kAttnWarps;
            const size_t pos = (size_t)__shfl_sync(0xffffffffu, pos_lane, m & 31);
            if (m < M_) {
                kcos[k] = *reinterpret_cast<const uint2 *>(p.cos_t + pos * 128 + 4 * lane);
                ksin[k] = *reinterpret_cast<const uint2 *>(p.sin_t + pos * 128 + 4 * lane);
            }
        }
    }
    if (early) pdl_wait();            // xqkv / q (and, in the plain build, the replay's own rows) come from the predecessor

    if (ROPE) {
        // every load that depends on the predecessor is issued before the first of them is used: one
        // memory round trip for the query vectors and the replay's own K / V rows together
        uint2 qraw[NQW], kraw[kFreshPerWarp], vraw[kFreshPerWarp];
#pragma unroll
        for (int k = 0; k < NQW; ++k) {
            qraw[k] = make_uint2(0u, 0u);
            if (q_live[k]) qraw[k] = *reinterpret_cast<const uint2 *>(p.xqkv + ((size_t)qm[k] * heads + hk * G + qg_[k]) * 128 + 4 * lane);
        }
        if (fresh) {
#pragma unroll
            for (int k = 0; k < kFreshPerWarp; ++k) {
                const int m = warp + k * kAttnWarps;
                if (m < M_) {
                    kraw[k] = *reinterpret_cast<const uint2 *>(p.xqkv + ((size_t)m * heads + p.H + hk) * 128 + 4 * lane);
                    vraw[k] = *reinterpret_cast<const uint2 *>(p.xqkv + ((size_t)m * heads + p.H + p.Hkv + hk) * 128 + 4 * lane);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < NQW; ++k) {
            const int qi = warp + k * kAttnWarps;
            if (qi >= qc) break;                                          // warp-uniform
            uint2 bits = make_uint2(0u, 0u);
            if (q_live[k]) {
                const float4 r = NV == 1 ? rope_head_vector(qraw[k], qw, qcos[k], qsin[k], p.eps, lane)
                                         : rope_head_vector_call(qraw[k], qw, qcos[k], qsin[k], p.eps, lane);
                bits = attn_pack_row({r.x, r.y, r.z, r.w});
            }
            *reinterpret_cast<uint2 *>(Qs + qi * kKeyStride + 4 * lane) = bits;
        }
        if (fresh) {
            // the replay's own rows: K through norm + RoPE, V as it is; the z == 0 CTA appends them to the planes
#pragma unroll
            for (int k = 0; k < kFreshPerWarp; ++k) {
                const int m = warp + k * kAttnWarps;
                if (m >= M_) break;                                       // warp-uniform
                const float4 r = NV == 1 ? rope_head_vector(kraw[k], kw, kcos[k], ksin[k], p.eps, lane)
                                         : rope_head_vector_call(kraw[k], kw, kcos[k], ksin[k], p.eps, lane);
                const uint2 kbits = attn_pack_row({r.x, r.y, r.z, r.w});
                *reinterpret_cast<uint2 *>(Ks + m * kKeyStride + 4 * lane) = kbits;
                *reinterpret_cast<uint2 *>(Vs + m * 128 + 4 * lane) = vraw[k];
                if (z == 0) {
                    const size_t row = ((size_t)hk * p.kv_rows + sigma_ + m) * 128 + 4 * lane;
                    *reinterpret_cast<uint2 *>(p.k_out + row) = kbits;
                    *reinterpret_cast<uint2 *>(p.v_out + row) = vraw[k];
                }
            }
        }
    } else {
        if (fresh) copy_rows();
#pragma unroll
        for (int k = 0; k < NQW; ++k) {
            const int qi = warp + k * kAttnWarps;
            if (qi >= qc) break;
            uint2 raw = make_uint2(0u, 0u);
            if (q_live[k])
                raw = *reinterpret_cast<const uint2 *>(p.q + ((size_t)(r0 + qm[k]) * p.H + hk * G + qg_[k]) * 128 + 4 * lane);
            *reinterpret_cast<uint2 *>(Qs + qi * kKeyStride + 4 * lane) = raw;
        }
    }
    cp_async_wait_all();
    __syncthreads();

    // level 0: warp = (sub-chunk c, query group g)
    {
        const int c = warp & (kAttnSub - 1), g = warp >> 2, cn = min(BM_ATTN_CHUNK, nkeys - c * BM_ATTN_CHUNK);
        // history keys are all visible but one, hidden from every row of a verify replay and of a draft without pending
        // rows: the last committed token, which such a replay appends again
        const bool hides = role == BM_ROLE_VERIFY || (role == BM_ROLE_DRAFT && min(max(n_pend, 0), P_) == 0);
        const int hidden = hides && !fresh ? cache_len - 1 - key0 - c * BM_ATTN_CHUNK : -1;
        const bool one = NV == 1 && QV - q_lo <= 2;                       // one vector per warp
        const AttnView a{fresh, role, sigma_, cache_len, n_pend, P_, M_, q_lo + (one ? 1 : 2 * nv) * g, key0 + c * BM_ATTN_CHUNK};
        const uint16_t *Kc = Ks + c * BM_ATTN_CHUNK * kKeyStride, *Vc = Vs + c * BM_ATTN_CHUNK * 128;
#define BM_ATTN_LEVEL0(N_)                                                                                                    \
    attn_level0<N_>(Kc, Vc, Qs + 2 * N_ * g * kKeyStride, Ps + warp * BM_ATTN_CHUNK * kWeightStride, a, cn, hidden, lane,       \
                    mc + c * QC + 2 * N_ * g, lc + c * QC + 2 * N_ * g, oc + ((size_t)c * QC + 2 * N_ * g) * 128)
        if (NV >= 4 && nv == 4) BM_ATTN_LEVEL0(4);
        else if (NV >= 3 && nv == 3) BM_ATTN_LEVEL0(3);
        else if (NV >= 2 && nv == 2) BM_ATTN_LEVEL0(2);
        else if (one)
            attn_level0_one(Kc, Vc, Qs + g * kKeyStride, Ps + warp * BM_ATTN_CHUNK * kWeightStride, a, cn, hidden, lane, mc + c * QC + g,
                            lc + c * QC + g, oc + ((size_t)c * QC + g) * 128);
        else BM_ATTN_LEVEL0(1);
#undef BM_ATTN_LEVEL0
    }
    __syncthreads();

    // level 1: the four sub-chunk partials of the warp's query vectors, merged in ascending sub-chunk order
    float MJ[NQW], L[NQW], O[NQW][4];
#pragma unroll
    for (int k = 0; k < NQW; ++k) {
        MJ[k] = -INFINITY;
        L[k] = O[k][0] = O[k][1] = O[k][2] = O[k][3] = 0.0f;
        if (!q_live[k]) continue;
        const int qi = warp + k * kAttnWarps;
        float mm[kAttnSub];
#pragma unroll
        for (int c = 0; c < kAttnSub; ++c) { mm[c] = mc[c * QC + qi]; MJ[k] = fmaxf(MJ[k], mm[c]); }
#pragma unroll
        for (int c = 0; c < kAttnSub; ++c) {
            const float w = mm[c] > -INFINITY ? pa_expf(mm[c] - MJ[k]) : 0.0f;
            L[k] = fmaf(lc[c * QC + qi], w, L[k]);
            const float4 o = *reinterpret_cast<const float4 *>(oc + ((size_t)c * QC + qi) * 128 + 4 * lane);
            O[k][0] = fmaf(o.x, w, O[k][0]);
            O[k][1] = fmaf(o.y, w, O[k][1]);
            O[k][2] = fmaf(o.z, w, O[k][2]);
            O[k][3] = fmaf(o.w, w, O[k][3]);
        }
        if (CLUSTER) {
            // the partial stays in this CTA: numerators over V rows, max and sum over the weights, both spent since the
            // CTA barrier after level 0
            *reinterpret_cast<float4 *>(reinterpret_cast<float *>(Vs) + qi * 128 + 4 * lane) = make_float4(O[k][0], O[k][1], O[k][2], O[k][3]);
            if (lane == 0) *reinterpret_cast<float2 *>(Ps + 2 * qi) = make_float2(MJ[k], L[k]);
        } else if (!HIST_DONE) {
            const size_t pb = ((size_t)(r0 + qm[k]) * p.H + hk * G + qg_[k]) * p.NJ + J;
            *reinterpret_cast<float4 *>(p.po + pb * 128 + 4 * lane) = make_float4(O[k][0], O[k][1], O[k][2], O[k][3]);
            if (lane == 0) { p.pm[pb] = MJ[k]; p.pl[pb] = L[k]; }
        }
    }
    if (MERGE == kMergeLater) return;
    if (CLUSTER) {
        cluster_arrive();
        cluster_wait();
        if (fresh) {
#pragma unroll
            for (int k = 0; k < NQW; ++k) {
                if (!q_live[k]) continue;
                // level 2 in the cluster: history super-chunks (cluster ranks 0 .. n_hs-1) in ascending order, then
                // this CTA's own partial; at most kAttnMaxCluster of them, requested in batches of eight
                const int qi = warp + k * kAttnWarps, np = n_hs + 1;
                const float *own_ml = Ps + 2 * qi, *own_o = reinterpret_cast<const float *>(Vs) + qi * 128 + 4 * lane;
                float2 ml = make_float2(-INFINITY, 0.0f);
                if (lane < n_hs) ml = cluster_ld2(cluster_map(own_ml, (uint32_t)lane));
                else if (lane == n_hs) ml = *reinterpret_cast<const float2 *>(own_ml);
                constexpr int kBatch = 8;
                float4 part[kBatch];
#pragma unroll
                for (int i = 0; i < kBatch; ++i)
                    part[i] = i < n_hs    ? cluster_ld4(cluster_map(own_o, (uint32_t)i))
                              : i == n_hs ? *reinterpret_cast<const float4 *>(own_o)
                                          : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                const float gmax = warp_max(ml.x);
                const float w0 = ml.x > -INFINITY ? pa_expf(ml.x - gmax) : 0.0f;
                float l = 0.0f, o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                for (int b0 = 0; b0 < np; b0 += kBatch) {
                    if (b0 > 0) {
#pragma unroll
                        for (int i = 0; i < kBatch; ++i) {
                            const int c = b0 + i;
                            part[i] = c < n_hs    ? cluster_ld4(cluster_map(own_o, (uint32_t)c))
                                      : c == n_hs ? *reinterpret_cast<const float4 *>(own_o)
                                                  : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < kBatch; ++i) {
                        const int c = b0 + i;
                        if (c < np) {                                      // warp-uniform
                            const float w = __shfl_sync(0xffffffffu, w0, c);
                            const float lj = __shfl_sync(0xffffffffu, ml.y, c);
                            l = fmaf(lj, w, l);
                            o[0] = fmaf(part[i].x, w, o[0]);
                            o[1] = fmaf(part[i].y, w, o[1]);
                            o[2] = fmaf(part[i].z, w, o[2]);
                            o[3] = fmaf(part[i].w, w, o[3]);
                        }
                    }
                }
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = bm_bf16_rn(o[e] / l);
                *reinterpret_cast<uint2 *>(p.att + (size_t)qm[k] * p.H * 128 + (hk * G + qg_[k]) * 128 + 4 * lane) = attn_pack_row(v);
                const float amax = attn_row_amax(v);
                if (lane == 0 && amax != 0.0f) atomicMax(&p.amax[qm[k]], __float_as_uint(amax));
            }
        }
        // every remote value has been consumed above: the other CTAs of the cluster may leave
        cluster_arrive();
        cluster_wait();
        return;
    }
    if (!HIST_DONE) {
        // ticket: the last CTA of this (kv head, query group) to get here merges the super-chunks
        __threadfence();
        __syncthreads();
        if (tid == 0) sh_ticket = atomicAdd(ticket, 1u);
        __syncthreads();
        if (sh_ticket != (unsigned int)n_hs) return;              // n_hs + 1 CTAs take part
        __threadfence();
        if (tid == 0) *ticket = 0u;                               // ready for the next launch
    }
#pragma unroll
    for (int k = 0; k < NQW; ++k) {
        if (!q_live[k]) continue;
        const size_t pb = ((size_t)(r0 + qm[k]) * p.H + hk * G + qg_[k]) * p.NJ;
        float v[4];
        attn_merge_vector<HIST_DONE>(p.pm, p.pl, p.po, pb, n_hs, p.NJ, lane, MJ[k], L[k],
                                     make_float4(O[k][0], O[k][1], O[k][2], O[k][3]), v);
        *reinterpret_cast<uint2 *>(p.att + (size_t)(r0 + qm[k]) * p.H * 128 + (hk * G + qg_[k]) * 128 + 4 * lane) = attn_pack_row(v);
        const float amax = attn_row_amax(v);
        if (lane == 0 && amax != 0.0f) atomicMax(&p.amax[r0 + qm[k]], __float_as_uint(amax));
    }
}

// =============================================================================
// Level 2 and the INT8 quantisation of the attention rows in one launch: one CTA per row, one warp per head; above 32
// heads (MANY) a warp takes every 32nd, and the rows go through memory between the merge and the codes.
// Follows attn_fused_kernel<.., kMergeLater>; replaces its ticket merge, the absmax atomics and the flat quantisation
// launch that had to read the rows again.  Same merge, same codes.
// =============================================================================
struct AttnMergeParams {
    const float *pm, *pl, *po;
    const StepState *state;
    int H, NJ, sigma, pdl;
    uint16_t *att;            // bf16 rows; optional up to 32 heads
    QuantSink q;
    float *s;
};

// Codes of the row's group `group` (row * H + head) by one warp; lane: dims 4 lane .. 4 lane + 3.
__device__ __forceinline__ void attn_emit_codes(const QuantSink &q, int group, const float (&v)[4], float s, int lane) {
    const size_t at = (size_t)group * 128;
    const uint32_t codes = quant_quad(v[0], v[1], v[2], v[3], s);
    if (q.nat) reinterpret_cast<uint32_t *>(q.nat + at)[lane] = codes;
    if (q.prep) {
        // GEMV-ready order: the 4 x 4 bytes of four consecutive lanes transposed in two exchanges
        const uint32_t x = __shfl_xor_sync(0xffffffffu, codes, 1), t = __byte_perm(codes, x, (lane & 1) ? 0x3715u : 0x6240u);
        const uint32_t y = __shfl_xor_sync(0xffffffffu, t, 2);
        reinterpret_cast<uint32_t *>(q.prep + at)[lane] = __byte_perm(t, y, (lane & 2) ? 0x3276u : 0x5410u);
        const int sum = __reduce_add_sync(0xffffffffu, __dp4a((int)codes, 0x01010101, 0));
        if (lane == 0) q.asum[group] = sum;
    }
}

template <bool MANY>
__global__ void __launch_bounds__(1024) attn_merge_quant_kernel(const AttnMergeParams p) {
    __shared__ unsigned int sh[32];
    pdl_launch_dependents();
    const bool early = (p.pdl & BM_PDL_STABLE_STATE) != 0;
    if (p.pdl && !early) pdl_wait();
    const int cache_len = min(max(p.state->cache_len, 0), p.sigma), n_hs = (cache_len + BM_ATTN_SUPER - 1) / BM_ATTN_SUPER;
    const int m = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (early) pdl_wait();
    // one head: merged rows (stored if asked for) and their absmax
    auto merge = [&](int head, float (&v)[4]) {
        const size_t row = (size_t)m * p.H + head;
        attn_merge_vector<false>(p.pm, p.pl, p.po, row * p.NJ, n_hs, p.NJ, lane, 0.0f, 0.0f, make_float4(0.0f, 0.0f, 0.0f, 0.0f), v);
        if (MANY || p.att) *reinterpret_cast<uint2 *>(p.att + row * 128 + 4 * lane) = attn_pack_row(v);
        return attn_row_amax(v);
    };
    float v[4], amax;
    if (MANY) {
        amax = 0.0f;
        for (int head = warp; head < p.H; head += 32) amax = fmaxf(amax, merge(head, v));
    } else {
        amax = merge(warp, v);
    }
    if (lane == 0) sh[warp] = __float_as_uint(amax);
    __syncthreads();
    const int nwarps = MANY ? 32 : p.H;
    const float s = bm_act_scale(__uint_as_float(__reduce_max_sync(0xffffffffu, lane < nwarps ? sh[lane] : 0u)));
    if (MANY) {
        for (int head = warp; head < p.H; head += 32) {
            const int row = m * p.H + head;
            const uint2 raw = *reinterpret_cast<const uint2 *>(p.att + (size_t)row * 128 + 4 * lane);   // (as this lane wrote it)
            const float u[4] = {__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                                __uint_as_float(raw.y & 0xffff0000u)};
            attn_emit_codes(p.q, row, u, s, lane);
        }
    } else {
        attn_emit_codes(p.q, m * p.H + warp, v, s, lane);
    }
    if (threadIdx.x == 0) p.s[m] = s;
}

}  // namespace bm
