// History part of the prompt attention: the super-chunk partials of MANY query rows at once.
//
// The prompt's causal attention runs in slabs of 16 rows: every row of slab s attends to the history
// [0, h_s), h_s = hist0 + 16 s, cut into super-chunks of 128 keys, and to the rows of its own slab (the
// reference's prompt forward: src/bonsai_sft/gpu/model.py:1306-1340).  attn_fused_kernel serves 8 query vectors
// per CTA, so it reads 64 KB of K / V per 262 K multiply-adds and repeats the staging, the waits and the
// level-1 merge for every eighth vector.  Here one CTA serves kPaQueries = 64 query vectors against one
// super-chunk as a register-blocked product on the CUDA cores (8 x 8 outputs per thread): scores S = Q K^T, the
// softmax of each 32-key sub-chunk, numerators O = P V and the merge of the four sub-chunks.  It writes the
// partials (max, sum, 128 numerators) that the slab's own CTA of attn_fused_kernel then merges in order.
//
// The work is fp32 arithmetic: 2 * 128 multiply-adds per (query vector, key).  Every one of them is the fma of
// attn_level0, in the same chain (scores ascending in d, numerators ascending in the key, sub-chunks
// ascending, the weight sum as the butterfly over the 32 keys), so the partials are the same bits; tensor
// cores would not give that order.  512 rows behind 2048 keys, 16 heads: 657 us by attn_fused_kernel alone; called from
// the host 414 us with scalar fmas and 356 with packed ones and an exponential without branches and conversions; 339 in
// a captured chain, 310 with every load of a tile out at once and the softmax on pairs too.  The fmas alone are 134 us at
// the fp32 rate.  Of a tile's 66000 cycles then the load took 8000, the scores 19000, the softmax 16000 and the numerators
// 21000: what is left is latency with two warps per scheduler, and nothing is loaded under the multiply.  Later: the merge
// weights of a vector made by one thread, not by each of its 16, and a slab kernel that stages 16 keys: 512 rows behind 2400
// keys 359 -> 327.  Three CTAs per SM (V over K^T, 168 registers) gave 330 there and lost 8 to 14 us a call where the tiles are
// few; 256 threads with 8 x 4 outputs each were level (their loads from shared memory then bind).
#pragma once

#include "verify_attn.cuh"

namespace bm {

constexpr int kPaThreads = 128;
constexpr int kPaQueries = 64;           // query vectors per CTA: 64 / G rows x G heads of a kv head
constexpr int kPaSlab = 16;              // rows per slab; a thread's 8 vectors and a warp's 16 lie in one slab
constexpr int kPaQStride = kPaQueries + 4;       // fp32 per d row of Q^T
constexpr int kPaKStride = BM_ATTN_SUPER + 8;    // bf16 per d row of K^T

struct PromptHistParams {
    const uint16_t *q;                   // [T, H, 128] rotated queries
    const uint16_t *k_base, *v_base;     // [Hkv, kv_rows, 128]
    float *pm, *pl, *po;                 // [T, H, NJ] and [T, H, NJ, 128]
    int T, H, Hkv, log_g, kv_rows, hist0, NJ, pdl;      // 2^log_g heads per kv head
};

// Q^T fp32 [128][kPaQStride] (after the scores its space holds P^T fp32 [128][64], see pa_weight), K^T bf16
// [128][kPaKStride], V bf16 [128][128], m and l fp32 [4][64].
constexpr int kPaQBytes = 128 * kPaQStride * 4, kPaKBytes = 128 * kPaKStride * 2, kPaVBytes = BM_ATTN_SUPER * 256;
constexpr int kPaSmem = kPaQBytes + kPaKBytes + kPaVBytes + 2 * kAttnSub * kPaQueries * 4;

// Whether the tile kernel takes a call; the launcher keeps attn_fused_kernel for every other slab height or
// head grouping.
__host__ __device__ inline bool prompt_hist_fits(int slab_rows, int H, int Hkv) {
    const int G = H / Hkv;
    return slab_rows == kPaSlab && (G == 1 || G == 2 || G == 4 || G == 8);
}

// History length of the slab that holds prompt row r.
__device__ __forceinline__ int pa_history(int hist0, int r) { return hist0 + r / kPaSlab * kPaSlab; }

// Keys of the super-chunk at key0 that the 16 vectors of a warp see; 0 where the warp has no row of the prompt.
__device__ __forceinline__ int pa_tile_keys(int hist0, int T, int row0, int log_g, int warp, int key0) {
    const int r = row0 + ((16 * warp) >> log_g);
    return r < T ? min(BM_ATTN_SUPER, pa_history(hist0, r) - key0) : 0;
}

// Word of weight (key, vector 8 vg) in P^T, whose 16-byte pieces are swizzled by the key's group of eight: the
// threads of a warp, eight keys apart, then store to different banks.  Vectors 8 vg + 4 .. + 7 are at ^ 4 words.
__device__ __forceinline__ int pa_weight(int key, int vg) { return key * kPaQueries + 4 * ((2 * vg) ^ (key >> 3)); }

// One step of the register-blocked products: acc[t][j] = fma(a[t], b[j], acc[t][j]), vectors t in pairs: the packed
// fma rounds each half as the scalar one does, runs at the same rate per value and takes half the issue slots.
__device__ __forceinline__ void pa_step(PaPair (&acc)[4][8], const float *a, const float *a4, const uint4 &braw) {
    float b[8];
    unpack8(braw, b);
    const ulonglong2 lo = *reinterpret_cast<const ulonglong2 *>(a), hi = *reinterpret_cast<const ulonglong2 *>(a4);
    const PaPair av[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const PaPair bb = pa_pack(b[j], b[j]);
#pragma unroll
        for (int t = 0; t < 4; ++t) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[t][j]) : "l"(av[t]), "l"(bb));
    }
}

// pa_expf of two values: the same roundings, two per instruction.  A NaN comes out of the products by itself.
__device__ __forceinline__ PaPair pa_expf2(PaPair x) {
    const PaPair biased = pa_add2(pa_mul2(x, pa_both(1.44269504088896341f)), pa_both(12582912.0f));
    const PaPair n = pa_add2(biased, pa_both(-12582912.0f));
    PaPair r = pa_fma2(n, pa_both(-0.693145751953125f), x);
    r = pa_fma2(n, pa_both(-1.42860682030941723e-6f), r);
    PaPair q = pa_fma2(pa_both(1.3888889225e-3f), r, pa_both(8.3333337680e-3f));
    q = pa_fma2(q, r, pa_both(4.1666667908e-2f));
    q = pa_fma2(q, r, pa_both(1.6666667163e-1f));
    q = pa_fma2(q, r, pa_both(0.5f));
    q = pa_fma2(q, r, pa_both(1.0f));
    q = pa_fma2(q, r, pa_both(1.0f));
    float b0, b1, x0, x1, e0, e1;
    pa_unpack(biased, b0, b1);
    pa_unpack(x, x0, x1);
    const PaPair pw = pa_pack(__uint_as_float((__float_as_uint(b0) - 0x4B400000u + 127u) << 23),
                              __uint_as_float((__float_as_uint(b1) - 0x4B400000u + 127u) << 23));
    pa_unpack(pa_mul2(q, pw), e0, e1);
    return pa_pack(x0 < -87.0f ? 0.0f : e0, x1 < -87.0f ? 0.0f : e1);
}

// Scores of 4 vector pairs x 8 keys -> bf16-rounded weights in place; maximum and weight sum of every vector's sub-chunk
// (the four threads of a sub-chunk hold 8 keys each).  FULL: every key is seen.
template <bool FULL>
__device__ __forceinline__ void pa_softmax(PaPair (&acc)[4][8], int lim, int kgp, int c, int v0, float *mc, float *lc) {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            acc[t][j] = pa_mul2(acc[t][j], pa_both(0.08838834764831845f));
            if (!FULL && 8 * kgp + j >= lim) acc[t][j] = pa_both(-INFINITY);
            float x0, x1;
            pa_unpack(acc[t][j], x0, x1);
            m0 = fmaxf(m0, x0);
            m1 = fmaxf(m1, x1);
        }
        m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 1));
        m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 1));
        m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 2));
        m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 2));
        const PaPair minus_m = pa_pack(-m0, -m1);
        PaPair s[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            PaPair pr = pa_expf2(pa_add2(acc[t][j], minus_m));
            if (!FULL && 8 * kgp + j >= lim) pr = 0ull;
            float p0, p1;
            pa_unpack(pr, p0, p1);
            // one conversion for both; a NaN is the canonical one, as bm_bf16_rn gives it
            uint32_t b;
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(b) : "f"(p1), "f"(p0));
            acc[t][j] = pa_pack(__uint_as_float(b << 16), __uint_as_float(b & 0xffff0000u));
            // butterfly over the 32 keys of the sub-chunk: offsets 16 and 8 lie across the four threads
            s[j] = pa_add2(pr, pa_pack(__shfl_xor_sync(0xffffffffu, p0, 2), __shfl_xor_sync(0xffffffffu, p1, 2)));
            pa_unpack(s[j], p0, p1);
            s[j] = pa_add2(s[j], pa_pack(__shfl_xor_sync(0xffffffffu, p0, 1), __shfl_xor_sync(0xffffffffu, p1, 1)));
        }
        const PaPair l = pa_add2(pa_add2(pa_add2(s[0], s[4]), pa_add2(s[2], s[6])), pa_add2(pa_add2(s[1], s[5]), pa_add2(s[3], s[7])));
        if ((kgp & 3) == 0) {
            float l0, l1;
            pa_unpack(l, l0, l1);
            *reinterpret_cast<float2 *>(mc + c * kPaQueries + v0 + 2 * t) = make_float2(m0, m1);
            *reinterpret_cast<float2 *>(lc + c * kPaQueries + v0 + 2 * t) = make_float2(l0, l1);
        }
    }
}

// grid (super-chunks of the longest history, Hkv, ceil(T * G / 64)), 128 threads = 8 vector groups x 16 key
// (then dim) groups.
__global__ void __launch_bounds__(kPaThreads, 2) prompt_hist_kernel(const PromptHistParams p) {
    extern __shared__ __align__(16) unsigned char pa_smem[];
    pdl_launch_dependents();
    if (p.pdl) pdl_wait();
    const int J = blockIdx.x, hk = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gmask = (1 << p.log_g) - 1, rows = kPaQueries >> p.log_g, row0 = blockIdx.z * rows;      // this tile's prompt rows
    const int row_end = min(row0 + rows, p.T);
    const int key0 = J * BM_ATTN_SUPER;
    const int keys_max = min(BM_ATTN_SUPER, pa_history(p.hist0, row_end - 1) - key0);
    if (keys_max <= 0) return;
    float *Qt = reinterpret_cast<float *>(pa_smem), *Pt = Qt;
    uint16_t *Kt = reinterpret_cast<uint16_t *>(pa_smem + kPaQBytes);
    uint16_t *Vs = reinterpret_cast<uint16_t *>(pa_smem + kPaQBytes + kPaKBytes);
    float *mc = reinterpret_cast<float *>(pa_smem + kPaQBytes + kPaKBytes + kPaVBytes), *lc = mc + kAttnSub * kPaQueries;

    // V as it is (16-byte asynchronous copies); K two rows per lane, transposed as bf16 pairs; Q one vector per
    // lane, transposed as fp32.  Consecutive lanes store consecutive words: no bank conflicts.
    const uint16_t *kg = p.k_base + ((size_t)hk * p.kv_rows + key0) * 128;
    const uint16_t *vg = p.v_base + ((size_t)hk * p.kv_rows + key0) * 128;
    for (int i = tid; i < keys_max * 16; i += kPaThreads) cp_async16(Vs + 8 * i, reinterpret_cast<const uint4 *>(vg) + i);
    {
        // Every load is out before the first store: the compiler may not move a load over a store to shared memory, and one
        // round trip per piece cost 8000 cycles of a tile's 66000.
        const int k0 = 2 * (lane + 32 * (warp & 1));                  // keys k0, k0 + 1
        const int v = lane + 32 * (warp & 1);                         // vector v of the tile: row v / G, head v % G
        const int r = row0 + (v >> p.log_g), head = (hk << p.log_g) + (v & gmask);
        uint4 ka[8], kb[8], qv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int d0 = 8 * ((warp >> 1) + 2 * j);
            ka[j] = kb[j] = qv[j] = make_uint4(0u, 0u, 0u, 0u);
            if (k0 < keys_max) ka[j] = *reinterpret_cast<const uint4 *>(kg + (size_t)k0 * 128 + d0);
            if (k0 + 1 < keys_max) kb[j] = *reinterpret_cast<const uint4 *>(kg + (size_t)(k0 + 1) * 128 + d0);
            if (r < p.T) qv[j] = *reinterpret_cast<const uint4 *>(p.q + ((size_t)r * p.H + head) * 128 + d0);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int d0 = 8 * ((warp >> 1) + 2 * j);
            const uint32_t aw[4] = {ka[j].x, ka[j].y, ka[j].z, ka[j].w}, bw[4] = {kb[j].x, kb[j].y, kb[j].z, kb[j].w};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                *reinterpret_cast<uint32_t *>(Kt + (d0 + 2 * w) * kPaKStride + k0) = __byte_perm(aw[w], bw[w], 0x5410);
                *reinterpret_cast<uint32_t *>(Kt + (d0 + 2 * w + 1) * kPaKStride + k0) = __byte_perm(aw[w], bw[w], 0x7632);
            }
            float f[8];
            unpack8(qv[j], f);
#pragma unroll
            for (int e = 0; e < 8; ++e) Qt[(d0 + e) * kPaQStride + v] = f[e];
        }
    }
    __syncthreads();

    const int vgp = tid >> 4, kgp = tid & 15;                         // vector group, key / dim group
    const int v0 = 8 * vgp;
    // Keys of this super-chunk that the warp's 16 vectors see: one slab, so one number, and the same in every lane also where
    // the prompt ends between the warp's two vector groups (the shuffles of the softmax take whole warps).
    const int lim = pa_tile_keys(p.hist0, p.T, row0, p.log_g, warp, key0);

    PaPair acc2[4][8];                                                // [vector pair][key]
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc2[t][j] = 0ull;
    if (lim > 0) {
        const float *qp = Qt + v0;
        const uint16_t *kp = Kt + 8 * kgp;
#pragma unroll 4
        for (int d = 0; d < 128; ++d)
            pa_step(acc2, qp + d * kPaQStride, qp + d * kPaQStride + 4, *reinterpret_cast<const uint4 *>(kp + d * kPaKStride));
    }
    __syncthreads();                                                  // Q^T is spent: its space takes P^T
    const int c = kgp >> 2;                                           // sub-chunk of this thread's keys
    if (lim >= BM_ATTN_SUPER) pa_softmax<true>(acc2, lim, kgp, c, v0, mc, lc);
    else pa_softmax<false>(acc2, lim, kgp, c, v0, mc, lc);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int w = pa_weight(8 * kgp + j, vgp);
        *reinterpret_cast<ulonglong2 *>(Pt + w) = make_ulonglong2(acc2[0][j], acc2[1][j]);
        *reinterpret_cast<ulonglong2 *>(Pt + (w ^ 4)) = make_ulonglong2(acc2[2][j], acc2[3][j]);
    }
    cp_async_wait_all();
    __syncthreads();
    // level 1 of a vector by one thread: maximum of its four sub-chunks, their weights (over the maxima) and the weight sum
    if (tid < kPaQueries) {
        float m[kAttnSub], MJ = -INFINITY, L = 0.0f;
#pragma unroll
        for (int s = 0; s < kAttnSub; ++s) { m[s] = mc[s * kPaQueries + tid]; MJ = fmaxf(MJ, m[s]); }
#pragma unroll
        for (int s = 0; s < kAttnSub; ++s) {
            const float w = m[s] > -INFINITY ? pa_expf(m[s] - MJ) : 0.0f;
            L = fmaf(lc[s * kPaQueries + tid], w, L);
            mc[s * kPaQueries + tid] = w;
        }
        const int r = row0 + (tid >> p.log_g), head = (hk << p.log_g) + (tid & gmask);
        if (r < p.T && pa_history(p.hist0, r) > key0) {
            const size_t pb = ((size_t)r * p.H + head) * p.NJ + J;
            p.pm[pb] = MJ;
            p.pl[pb] = L;
        }
    }
    __syncthreads();
    if (lim <= 0) return;

    // numerators: this thread's 8 vectors x dims 8 kgp .. 8 kgp + 7, one chain per sub-chunk, then the merge
    PaPair O[4][8];                                                   // [vector pair][dim]
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int e = 0; e < 8; ++e) O[t][e] = 0ull;
    for (int s = 0; s < kAttnSub; ++s) {
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc2[t][e] = 0ull;
        const int cn = min(BM_ATTN_CHUNK, lim - s * BM_ATTN_CHUNK);
        for (int k8 = 0; k8 < cn; k8 += 8) {
            const int key = s * BM_ATTN_CHUNK + k8, w = pa_weight(key, vgp);
            const uint16_t *vp = Vs + key * 128 + 8 * kgp;
            if (cn - k8 >= 8) {
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    pa_step(acc2, Pt + w + k * kPaQueries, Pt + (w ^ 4) + k * kPaQueries,
                            *reinterpret_cast<const uint4 *>(vp + k * 128));
            } else {                                                  // a history that ends inside the eight keys
                for (int k = 0; k < cn - k8; ++k)
                    pa_step(acc2, Pt + w + k * kPaQueries, Pt + (w ^ 4) + k * kPaQueries,
                            *reinterpret_cast<const uint4 *>(vp + k * 128));
            }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const PaPair w = *reinterpret_cast<const PaPair *>(mc + s * kPaQueries + v0 + 2 * t);
#pragma unroll
            for (int e = 0; e < 8; ++e) O[t][e] = pa_fma2(acc2[t][e], w, O[t][e]);
        }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        float lo[8], hi[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) pa_unpack(O[t][e], lo[e], hi[e]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int v = v0 + 2 * t + i, r = row0 + (v >> p.log_g), head = (hk << p.log_g) + (v & gmask);
            if (r >= p.T) continue;
            const float *o = i ? hi : lo;
            float *dst = p.po + (((size_t)r * p.H + head) * p.NJ + J) * 128 + 8 * kgp;
            *reinterpret_cast<float4 *>(dst) = make_float4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<float4 *>(dst + 4) = make_float4(o[4], o[5], o[6], o[7]);
        }
    }
}

}  // namespace bm
