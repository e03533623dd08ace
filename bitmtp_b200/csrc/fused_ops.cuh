// Small fused operators of the decode step: activation absmax/INT8 quantisation,
// (residual add +) RMSNorm (+ quantisation), SiLU*up + quantisation, q/k head
// norm + RoPE + KV append, embedding gather, argmax / confidence reductions.
//
// Each kernel states the reference expression it replaces.  All of them round
// where the reference's eager tensor code rounds (bf16 in memory, fp32
// arithmetic) and reduce in the order fixed by oracle/bm_oracle.c, so results
// equal the oracle's bit for bit.
#pragma once

#include "bm_common.cuh"

namespace bm {

// Device-resident description of the replay in flight.  Written by
// bm_set_step_state (a one-thread kernel, so it can sit in front of a captured
// graph) and read by the attention kernels, so that a captured graph can be
// replayed for any cache length and pending count.
struct StepState {
    int cache_len;   // history rows [0, cache_len) are valid
    int n_pend;      // pending rows at the head of a draft replay
    int role;        // BM_ROLE_*
    int P;           // M - D
};

// ---- block-wide helpers -------------------------------------------------------
// Sum of per-warp values in ascending warp order, same result in every thread.
__device__ __forceinline__ float block_sum_ordered(float warp_val, float *sh, int lane, int warp,
                                                   int nwarps) {
    if (lane == 0) sh[warp] = warp_val;
    __syncthreads();
    float t = 0.0f;
    for (int w = 0; w < nwarps; ++w) t += sh[w];
    __syncthreads();
    return t;
}

// The same for the row kernels.  `sh`: 32 floats, 16-byte aligned, that the block uses for nothing else (no barrier at the
// end).  Four values per load: one by one in a run-time loop they were a chain of shared-memory round trips.  With
// block_absmax and mean_of in the norm, 256 + 256 hybrid tokens 41.9 -> 41.45 ms (the width-1 GEMVs' own norm gained nothing).
__device__ __forceinline__ float block_sum_rows(float warp_val, float *sh, int lane, int warp, int nwarps) {
    if (lane == 0) sh[warp] = warp_val;
    __syncthreads();
    float t = 0.0f;
    int w = 0;
#pragma unroll 2
    for (; w + 4 <= nwarps; w += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(sh + w);
        t += v.x; t += v.y; t += v.z; t += v.w;
    }
    for (; w < nwarps; ++w) t += sh[w];
    return t;
}

// Maximum of values that are not negative (an absmax: never NaN, fmaxf drops it), the same result in every thread.  Such
// floats order as their bits, so both levels are one integer reduction each.  `sh` as above; nwarps <= 32.
__device__ __forceinline__ float block_absmax(float v, float *sh, int lane, int warp, int nwarps) {
    const unsigned int m = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
    if (lane == 0) sh[warp] = __uint_as_float(m);
    __syncthreads();
    return __uint_as_float(__reduce_max_sync(0xffffffffu, lane < nwarps ? __float_as_uint(sh[lane]) : 0u));
}

__device__ __forceinline__ float block_max(float v, float *sh, int lane, int warp, int nwarps) {
    v = warp_max(v);
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    float t = sh[0];
    for (int w = 1; w < nwarps; ++w) t = fmaxf(t, sh[w]);
    __syncthreads();
    return t;
}

__device__ __forceinline__ void unpack8(const uint4 &v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        w[i] = bf16_pair(f[2 * i], f[2 * i + 1]);
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Eight bf16 values as they are stored: a signalling NaN becomes a quiet one (bm_f32_to_bf16 of a value from memory).
__device__ __forceinline__ uint4 quiet8(uint4 v) {
    uint32_t *w = &v.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] |= __vcmpgtu2(w[i] & 0x7fff7fffu, 0x7f807f80u) & 0x00400040u;
    return v;
}

// h = bf16(h + r), the rounded sums also as they are stored.
__device__ __forceinline__ uint4 add8(float (&h)[8], const float (&r)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = h[i] + r[i];
    const uint4 v = pack8(h);
    unpack8(v, h);
    return v;
}

// n = bf16(w * bf16(h * r)); returns the largest |n| (a NaN is passed over).
__device__ __forceinline__ float norm8(const float (&h)[8], const float (&w)[8], float r, float (&n)[8]) {
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        float a = h[i] * r, b = h[i + 1] * r;
        bf16_round_pair(a, b);
        n[i] = w[i] * a;
        n[i + 1] = w[i + 1] * b;
        bf16_round_pair(n[i], n[i + 1]);
        amax = fmaxf(fmaxf(amax, fabsf(n[i])), fabsf(n[i + 1]));
    }
    return amax;
}

__device__ __forceinline__ uint2 quant8(const float (&f)[8], float s) {
    return make_uint2(quant_quad(f[0], f[1], f[2], f[3], s), quant_quad(f[4], f[5], f[6], f[7], s));
}

// Where the INT8 codes of a row go.  `nat` is the natural-order row the reference's
// operator API exposes; `prep` + `asum` are the GEMV-ready form: within every run of 16
// elements the bytes are transposed 4x4 (prep[4t+e] = nat[4e+t]), which is the order the
// GEMV kernels' fragments want, and asum[g] is the sum of the 128 codes of group g.  Any
// of the three may be null.
struct QuantSink {
    int8_t *nat;
    int8_t *prep;
    int32_t *asum;
};

// Stores the 8 codes of 8-element unit `unit` of a row.  Whole warps call this together
// (lanes whose unit lies past the row pass active = false): lane pairs (l, l^1) hold the
// two halves of a 16-element run and exchange them, 16 consecutive lanes hold one group.
__device__ __forceinline__ void emit_codes(const QuantSink &sink, size_t row_off, int K, int unit,
                                           uint2 codes, bool active, int lane) {
    if (sink.nat && active) reinterpret_cast<uint2 *>(sink.nat + row_off)[unit] = codes;
    if (sink.prep == nullptr) return;
    if (!active) codes = make_uint2(0u, 0u);
    const uint2 other = make_uint2(__shfl_xor_sync(0xffffffffu, codes.x, 1),
                                   __shfl_xor_sync(0xffffffffu, codes.y, 1));
    const bool odd = unit & 1;
    const uint2 lo = odd ? other : codes, hi = odd ? codes : other;
    const uint32_t sel = odd ? 0x7362u : 0x5140u;
    const uint32_t t = __byte_perm(lo.x, lo.y, sel), u = __byte_perm(hi.x, hi.y, sel);
    if (active)
        reinterpret_cast<uint2 *>(sink.prep + row_off)[unit] =
            make_uint2(__byte_perm(t, u, 0x5410), __byte_perm(t, u, 0x7632));
    int sum = __dp4a((int)codes.x, 0x01010101, 0);
    sum = __dp4a((int)codes.y, 0x01010101, sum);
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (active && (lane & 15) == 0) sink.asum[(row_off / K) * (K / BM_GROUP) + (unit >> 4)] = sum;
}

// =============================================================================
// quant_rows: per-row absmax INT8 quantisation of bf16 activations.
// Replaces T2LinearKernel.quant_input (src/bonsai_sft/gpu/model.py:632-636) and
// the inline copy in _lm_head (model.py:1247-1249).  One CTA per row.
// =============================================================================
constexpr int kRowThreads = 512;

__global__ void __launch_bounds__(kRowThreads) quant_rows_kernel(const uint16_t *x, int K, QuantSink sink, float *s_out, int pdl) {
    __shared__ float sh[kRowThreads / 32];
    pdl_launch_dependents();
    if (pdl) pdl_wait();
    const int m = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint4 *xr = reinterpret_cast<const uint4 *>(x + (size_t)m * K);
    const int units = K / 8;
    float amax = 0.0f;
    for (int u = threadIdx.x; u < units; u += kRowThreads) {
        float f[8];
        unpack8(xr[u], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(f[i]));
    }
    amax = block_absmax(amax, sh, lane, warp, kRowThreads / 32);
    const float s = bm_act_scale(amax);
    for (int u0 = 0; u0 < units; u0 += kRowThreads) {
        const int u = u0 + threadIdx.x;
        const bool active = u < units;
        float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (active) unpack8(xr[u], f);
        emit_codes(sink, (size_t)m * K, K, u, quant8(f, s), active, lane);
    }
    if (threadIdx.x == 0) s_out[m] = s;
}

// =============================================================================
// quant_rows with the row absmax already known: the gate|up projection with the SiLU epilogue
// (t2_gemv.cuh) leaves bf16 `inner` rows and, by atomic max, the bits of each row's absmax; this kernel
// turns them into INT8 codes for the down projection.  Replaces the quant_input half of
// `inner = F.silu(g) * u; quant_input(inner)` (model.py:1059-1061).  Units of 8 elements are dealt to
// the threads of a flat grid, so the work spreads over many SMs instead of one CTA per row.
// `amax_zero` (optional): M words cleared for the next producer (a different array from amax_in).
// =============================================================================
constexpr int kQuantAmaxThreads = 256;

__global__ void __launch_bounds__(kQuantAmaxThreads) quant_rows_amax_kernel(
    const uint16_t *x, const unsigned int *amax_in, unsigned int *amax_zero, int M, int K, QuantSink sink, float *s_out, int pdl) {
    pdl_launch_dependents();
    if (pdl) pdl_wait();
    const int units = K / 8, lane = threadIdx.x & 31;
    const int u = blockIdx.x * kQuantAmaxThreads + threadIdx.x;   // whole warps stay inside one row (units % 32 == 0)
    const bool active = u < M * units;
    const int m = active ? u / units : 0, i = active ? u - m * units : 0;
    float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    float s = 0.0f;
    if (active) {
        unpack8(reinterpret_cast<const uint4 *>(x + (size_t)m * K)[i], v);
        s = bm_act_scale(__uint_as_float(amax_in[m]));
        if (i == 0) s_out[m] = s;
    }
    emit_codes(sink, (size_t)m * K, K, i, quant8(v, s), active, lane);
    if (amax_zero != nullptr && blockIdx.x == 0)
        for (int r = threadIdx.x; r < M; r += kQuantAmaxThreads) amax_zero[r] = 0u;
}

// =============================================================================
// (gather | residual add) + RMSNorm + (INT8 quantisation | bf16 store).
// Replaces _fused_norm_quant (model.py:307-319), _fused_add_norm_quant
// (model.py:322-336), RMSNorm.forward on the logit rows (model.py:290-295,
// 1401-1402) and the embedding gather in front of layer 0 (model.py:1386).
//   x        bf16 rows; with `gather` row m is x[gather[m]] (embedding table)
//   res      optional bf16 [M, dim]: h = bf16(x + res)
//   h_out    optional bf16 [M, dim]: the (gathered / summed) row before the norm
//   q, s     optional INT8 row + multiplier of the normed row
//   n_out    optional bf16 normed row
// One CTA per row, dim/8 threads (dim a multiple of 256): thread t owns
// elements 8t..8t+7, which is exactly the lane-partial of the oracle's
// sum-of-squares order; warps are its 256-element chunks.
// =============================================================================
// Row of a gathered table, kept inside the table whatever the id is (a corrupt id then reads a valid
// row instead of memory far outside the allocation).
__device__ __forceinline__ size_t gather_row(int64_t id, int rows) {
    return (size_t)(id < 0 ? 0 : (id >= rows ? rows - 1 : id));
}

// sum / n, by a product where that is the same value (n a power of two).
__device__ __forceinline__ float mean_of(float sum, int n) {
    return (n & (n - 1)) == 0 ? sum * __uint_as_float((uint32_t)(96 + __clz(n)) << 23) : sum / (float)n;
}

struct NormParams {
    const uint16_t *x;
    const int64_t *gather;
    int gather_rows;   // rows of x when `gather` is given: indices are clamped to [0, gather_rows)
    const uint16_t *res;
    const uint16_t *w;
    uint16_t *h_out;
    QuantSink q;
    float *s;
    uint16_t *n_out;
    float eps;
    int dim;
    int row0;        // first row of x / res to read (logit rows start at logits_start)
    int pdl;
};

__global__ void __launch_bounds__(1024) rmsnorm_kernel(const NormParams p) {
    __shared__ __align__(16) float sh[64];
    pdl_launch_dependents();
    const int m = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nwarps = blockDim.x >> 5;
    // the norm weights do not depend on the previous kernel: requested before the wait, used after the sum
    const uint4 wraw = reinterpret_cast<const uint4 *>(p.w)[t];
    if (p.pdl) pdl_wait();
    const size_t src_row = p.gather ? gather_row(p.gather[m], p.gather_rows) : (size_t)(p.row0 + m);
    float h[8];
    uint4 hraw = reinterpret_cast<const uint4 *>(p.x + src_row * p.dim)[t];
    unpack8(hraw, h);
    if (p.res) {
        float r[8];
        unpack8(reinterpret_cast<const uint4 *>(p.res + (size_t)(p.row0 + m) * p.dim)[t], r);
        hraw = add8(h, r);
    } else {
        hraw = quiet8(hraw);
    }
    if (p.h_out) reinterpret_cast<uint4 *>(p.h_out + (size_t)m * p.dim)[t] = hraw;
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc = fmaf(h[i], h[i], acc);
    const float total = block_sum_rows(warp_sum_butterfly(acc), sh, lane, warp, nwarps);
    const float r = bm_rsqrtf(mean_of(total, p.dim) + p.eps);
    float wv[8], n[8];
    unpack8(wraw, wv);
    const float amax_row = norm8(h, wv, r, n);
    if (p.n_out) reinterpret_cast<uint4 *>(p.n_out + (size_t)m * p.dim)[t] = pack8(n);
    if (p.s) {
        const float amax = block_absmax(amax_row, sh + 32, lane, warp, nwarps);
        const float s = bm_act_scale(amax);
        emit_codes(p.q, (size_t)m * p.dim, p.dim, t, quant8(n, s), true, lane);
        if (t == 0) p.s[m] = s;
    }
}

// =============================================================================
// SiLU(gate) * up + INT8 quantisation of the down-projection input.
// Replaces `inner = F.silu(g) * u; quant_input(inner)` (model.py:1059-1061).
// gu bf16 [M, 2F] holds gate | up.  One CTA per row; the bf16 products wait in
// shared memory between the absmax pass and the quantisation pass.
// =============================================================================
__global__ void __launch_bounds__(kRowThreads) silu_mul_quant_kernel(
    const uint16_t *gu, int F, QuantSink sink, float *s_out, uint16_t *inner_out, int pdl) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ float sh[kRowThreads / 32];
    pdl_launch_dependents();
    if (pdl) pdl_wait();
    uint4 *inner = reinterpret_cast<uint4 *>(dyn);
    const int m = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint4 *g = reinterpret_cast<const uint4 *>(gu + (size_t)m * 2 * F);
    const uint4 *u = reinterpret_cast<const uint4 *>(gu + (size_t)m * 2 * F + F);
    const int units = F / 8;
    float amax = 0.0f;
    for (int i = threadIdx.x; i < units; i += kRowThreads) {
        float gf[8], uf[8], v[8];
        unpack8(g[i], gf);
        unpack8(u[i], uf);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[e] = bm_bf16_rn(bm_silu_bf16(gf[e]) * uf[e]);
            amax = fmaxf(amax, fabsf(v[e]));
        }
        const uint4 packed = pack8(v);
        inner[i] = packed;
        if (inner_out) reinterpret_cast<uint4 *>(inner_out + (size_t)m * F)[i] = packed;
    }
    amax = block_absmax(amax, sh, lane, warp, kRowThreads / 32);
    const float s = bm_act_scale(amax);
    for (int i0 = 0; i0 < units; i0 += kRowThreads) {
        const int i = i0 + threadIdx.x;
        const bool active = i < units;
        float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (active) unpack8(inner[i], v);
        emit_codes(sink, (size_t)m * F, F, i, quant8(v, s), active, lane);
    }
    if (threadIdx.x == 0) s_out[m] = s;
}

// =============================================================================
// Split qkv, per-head RMSNorm of q and k, RoPE, append K and V rows.
// Replaces _fused_qkv_qknorm_rope_kv_write (model.py:388-436).
//   xqkv bf16 [M, (H + 2*Hkv)*128]; cos/sin bf16 [max_pos, 128]; positions int64
//   k_base/v_base: one layer of the shared KV buffer, bf16 [Hkv, kv_rows, 128];
//   rows [sigma, sigma+M) are written.  q_out bf16 [M, H, 128].
// One warp per head vector: lane l owns elements 4l..4l+3 (the oracle's lane
// partial for a 128-wide row); the RoPE partner i +- 64 lives in lane l ^ 16.
// =============================================================================
struct RopeParams {
    const uint16_t *xqkv;
    const uint16_t *q_w, *k_w;
    const uint16_t *cos_t, *sin_t;
    const int64_t *positions;
    uint16_t *k_base, *v_base, *q_out;
    float eps;
    int M, H, Hkv, kv_rows, sigma, pdl;
};

__global__ void __launch_bounds__(128) qknorm_rope_kvappend_kernel(const RopeParams p) {
    pdl_launch_dependents();
    if (p.pdl) pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int heads = p.H + 2 * p.Hkv;
    const int m = blockIdx.y;
    const int hd = blockIdx.x * 4 + warp;
    if (hd >= heads) return;
    const uint16_t *src = p.xqkv + ((size_t)m * heads + hd) * 128 + 4 * lane;
    const uint2 raw = *reinterpret_cast<const uint2 *>(src);
    if (hd >= p.H + p.Hkv) {                          // V head: plain copy
        const int hk = hd - p.H - p.Hkv;
        *reinterpret_cast<uint2 *>(p.v_base + ((size_t)hk * p.kv_rows + p.sigma + m) * 128 + 4 * lane) = raw;
        return;
    }
    float x[4] = {__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u),
                  __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u)};
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) acc = fmaf(x[i], x[i], acc);
    const float total = warp_sum_butterfly(acc);      // one chunk: 0 + chunk sum
    const float r = bm_rsqrtf((0.0f + total) / 128.0f + p.eps);
    const uint16_t *wsrc = (hd < p.H ? p.q_w : p.k_w) + 4 * lane;
    const uint2 wraw = *reinterpret_cast<const uint2 *>(wsrc);
    const float w[4] = {__uint_as_float(wraw.x << 16), __uint_as_float(wraw.x & 0xffff0000u),
                        __uint_as_float(wraw.y << 16), __uint_as_float(wraw.y & 0xffff0000u)};
    const size_t pos = (size_t)p.positions[m];
    const uint2 craw = *reinterpret_cast<const uint2 *>(p.cos_t + pos * 128 + 4 * lane);
    const uint2 sraw = *reinterpret_cast<const uint2 *>(p.sin_t + pos * 128 + 4 * lane);
    const float c[4] = {__uint_as_float(craw.x << 16), __uint_as_float(craw.x & 0xffff0000u),
                        __uint_as_float(craw.y << 16), __uint_as_float(craw.y & 0xffff0000u)};
    const float sn[4] = {__uint_as_float(sraw.x << 16), __uint_as_float(sraw.x & 0xffff0000u),
                         __uint_as_float(sraw.y << 16), __uint_as_float(sraw.y & 0xffff0000u)};
    float n[4], o[4];
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        float a = x[i] * r, b = x[i + 1] * r;
        bf16_round_pair(a, b);
        n[i] = w[i] * a;
        n[i + 1] = w[i + 1] * b;
        bf16_round_pair(n[i], n[i + 1]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float partner = __shfl_xor_sync(0xffffffffu, n[i], 16);
        const float rot = lane < 16 ? -partner : partner;
        o[i] = bm_bf16_rn(n[i] * c[i]) + bm_bf16_rn(rot * sn[i]);
    }
    const uint2 packed = make_uint2(
        bf16_pair(o[0], o[1]), bf16_pair(o[2], o[3]));
    uint16_t *dst = hd < p.H
                        ? p.q_out + ((size_t)m * p.H + hd) * 128
                        : p.k_base + ((size_t)(hd - p.H) * p.kv_rows + p.sigma + m) * 128;
    *reinterpret_cast<uint2 *>(dst + 4 * lane) = packed;
}

// =============================================================================
// Step state and KV row promotion
// =============================================================================
__global__ void set_step_state_kernel(StepState *st, int cache_len, int n_pend, int role, int P) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        st->cache_len = cache_len;
        st->n_pend = n_pend;
        st->role = role;
        st->P = P;
    }
}

// Token ids, positions and the step record of one replay in ONE launch (the reference fills them with
// half a dozen tensor ops per step, fast_generate.py:1015-1037 draft, 1040-1055 verify, 247-256 AR).
//   kind 0  draft of width M = P + D:  tok = pending[0..n_pend) | 0.. | pending[n_pend-1] | MASK..,
//           pos = cache_len + i for the pending rows, 0 for the padding rows,
//           cache_len + n_pend - 1 + k for the D block rows
//   kind 1  verify of width M = D + 1: tok = pending[n_pend-1] | draft[0..D), pos = cache_len - 1 + i
//   kind 2  AR (M = 1): tok = src_a[0], pos = cache_len
//   kind 3  prompt slab of width M with n_pend real rows: tok = src_a[0..n_pend) | 0.., pos = cache_len + i | 0..
// `src_a` = pending tokens (prompt rows for kind 3), `src_b` = draft tokens (kind 1).  The record is what bm_set_step_state writes.
__global__ void stage_replay_inputs_kernel(int kind, const int64_t *__restrict__ src_a,
                                           const int64_t *__restrict__ src_b, int n_pend, int cache_len, int M, int D,
                                           int64_t mask_id, int role, int P, int state_n_pend,
                                           int64_t *__restrict__ tok, int64_t *__restrict__ pos, StepState *st) {
    const int i = threadIdx.x;
    if (i == 0) {
        st->cache_len = cache_len;
        st->n_pend = state_n_pend;
        st->role = role;
        st->P = P;
    }
    if (i >= M) return;
    if (kind == 0) {
        int64_t t, q;
        if (i > P) { t = mask_id; q = cache_len + n_pend - 1 + (i - P); }
        else if (i == P) { t = src_a[n_pend - 1]; q = cache_len + n_pend - 1; }
        else if (i < n_pend) { t = src_a[i]; q = cache_len + i; }
        else { t = 0; q = 0; }
        tok[i] = t;
        pos[i] = q;
    } else if (kind == 1) {
        tok[i] = i == 0 ? src_a[n_pend - 1] : src_b[i - 1];
        pos[i] = cache_len - 1 + i;
    } else if (kind == 2) {
        tok[i] = src_a[0];
        pos[i] = cache_len;
    } else {
        tok[i] = i < n_pend ? src_a[i] : 0;
        pos[i] = i < n_pend ? cache_len + i : 0;
    }
}

// The end of one decode step and the start of the next in one launch: the committed ids go to the output
// buffer and become the pending rows (all of them after a confidence commit, the last one = the verifier's
// token after a verified step: fast_generate.py:1121-1140), then the draft inputs are staged from them as
// stage_replay_inputs_kernel kind 0 does.  One warp; n_commit <= 32.  stage == 0: commit only.
__global__ void commit_stage_draft_kernel(const int64_t *__restrict__ src, int n_commit, int verified,
                                          int64_t *__restrict__ gen_dst, int64_t *__restrict__ pending, int stage,
                                          int cache_len, int M, int D, int64_t mask_id, int role, int P,
                                          int64_t *__restrict__ tok, int64_t *__restrict__ pos, StepState *st) {
    const int i = threadIdx.x;
    if (i < n_commit) {
        const int64_t t = src[i];
        gen_dst[i] = t;
        if (!verified) pending[i] = t;
        else if (i == n_commit - 1) pending[0] = t;
    }
    if (!stage) return;
    __syncwarp();
    const int n_pend = verified ? 1 : n_commit;
    if (i == 0) {
        st->cache_len = cache_len;
        st->n_pend = n_pend > P ? P : n_pend;
        st->role = role;
        st->P = P;
    }
    if (i >= M) return;
    int64_t t, q;
    if (i > P) { t = mask_id; q = cache_len + n_pend - 1 + (i - P); }
    else if (i == P) { t = pending[n_pend - 1]; q = cache_len + n_pend - 1; }
    else if (i < n_pend) { t = pending[i]; q = cache_len + i; }
    else { t = 0; q = 0; }
    tok[i] = t;
    pos[i] = q;
}

// Copies rows [src_row, src_row + n) to [dst_row, dst_row + n) in every
// (k|v, layer, kv head) plane of the shared buffer [planes, kv_rows, 128] bf16.
// Replaces GraphAtlas.commit_kv / commit_kv_from_verify
// (src/bonsai_sft/gpu/fast_runtime.py:467-508); the two ranges never overlap
// because the source rows sit at or beyond sigma and the destination below it.
__global__ void kv_copy_rows_kernel(uint16_t *kv, int planes, int kv_rows, int src_row, int dst_row,
                                    int n) {
    const int plane = blockIdx.x;
    if (plane >= planes) return;
    uint4 *base = reinterpret_cast<uint4 *>(kv + (size_t)plane * kv_rows * 128);
    for (int i = threadIdx.x; i < n * 16; i += blockDim.x)
        base[(size_t)dst_row * 16 + i] = base[(size_t)src_row * 16 + i];
}

// =============================================================================
// Freeze + pack: bf16 weights [N, K] -> the {-s, 0, +s} grid of each 128-group and its packed form.
// Replaces, on the device, freeze_quantize_to_ternary_g128 (src/bonsai_sft/ternary_modules.py:86-93)
// followed by _pack_t2_g128 (src/bonsai_sft/gpu/convert_bonsai_mtp_to_gpu.py:127-144), which the
// reference's converter runs tensor by tensor on the CPU:
//   s = max(absmax of the group, 1e-8) (fp32); q = clamp(round_half_even(w / s), -1, 1);
//   frozen = bf16(q * s); scale = bf16(absmax of frozen) (= bf16(s) unless the group is all zero);
//   code = q + 2, element j of a row in bits 2 (j % 4) of byte j / 4.
// The groups are numbered through the matrix (K % 128 == 0: group u of the matrix is 128 consecutive weights,
// 32 packed bytes and one scale), half a warp per group, lane l of the half owning elements 8l .. 8l+7.
// Bound by HBM (2.27 bytes per weight), so a warp requests the 512 bytes of each of kPackGroupPairs pairs of
// groups before it uses the first, and nothing is divided:
//   * round_half_even(w / s) with |w| <= s is +-1 exactly when |w| > s / 2 (the bf16 neighbours of s / 2 give a
//     quotient at least 2^-9 away from one half, 2^-11 where s is the 1e-8 floor, which is no bf16 value: its
//     rounding cannot reach one half), i.e. when 2|w| > s;
//   * the scale is a function of the group's absmax alone (the absmax element itself rounds to +-1), so the
//     second reduction, over the frozen values, and the packer's second division (exact +-1 or 0) drop out.
// 12288 x 2048, one call after another: 88.1 us with two IEEE divisions per weight and one 512-byte request per warp, 16.4
// without, 13.6 where a launch overlaps the end of the one before (57 MB: 8.7 us at the measured copy rate; two or eight
// pairs a warp about 1 us more).  Letting the next launch start with this one's first block was no faster (13.7), and products
// behind it then requested codes that were not there yet.
// NaN weights pack as 0 and are ignored by the absmax; a group with an infinity has scale 0 and all codes 0, as
// `inf / inf` and `0 * inf` of the expressions above give.
// =============================================================================
constexpr int kPackGroupPairs = 4;       // pairs of groups per warp
constexpr int kPackThreads = 256;

template <bool FROZEN>
__global__ void __launch_bounds__(kPackThreads) pack_t2_g128_kernel(const uint16_t *w, long long groups, uint8_t *packed,
                                                                    uint16_t *scale, uint16_t *frozen) {
    // No launch_dependents: every product requests its weights before its own wait, and these are what is written here.  The
    // launch itself overlaps the previous one; nothing is read or written before this wait.
    pdl_wait();
    const int lane = threadIdx.x & 31, sub = lane & 15;
    const long long u0 = ((long long)blockIdx.x * (kPackThreads / 32) + (threadIdx.x >> 5)) * (2 * kPackGroupPairs) + (lane >> 4);
    uint4 raw[kPackGroupPairs];
#pragma unroll
    for (int i = 0; i < kPackGroupPairs; ++i)
        raw[i] = u0 + 2 * i < groups ? __ldcs(reinterpret_cast<const uint4 *>(w) + (u0 + 2 * i) * 16 + sub)
                                     : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int i = 0; i < kPackGroupPairs; ++i) {
        const long long u = u0 + 2 * i;
        float x[8];
        unpack8(raw[i], x);
        float amax = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(x[e]));
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        if (u >= groups) continue;
        const float s = fmaxf(amax, 1e-8f);
        uint32_t two = 0;
        float fr[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const bool one = 2.0f * fabsf(x[e]) > s;
            two |= (one ? (x[e] < 0.0f ? 1u : 3u) : 2u) << (2 * e);
            if (FROZEN) fr[e] = x[e] != x[e] ? __uint_as_float(0x7fffffffu) : bm_bf16_rn(copysignf(one ? 1.0f : 0.0f, x[e]) * s);
        }
        reinterpret_cast<uint16_t *>(packed)[u * 16 + sub] = (uint16_t)two;
        if (sub == 0) scale[u] = (2.0f * amax > s && amax < INFINITY) ? bm_f32_to_bf16(s) : (uint16_t)0;
        if (FROZEN) reinterpret_cast<uint4 *>(frozen)[u * 16 + sub] = pack8(fr);
    }
}

// =============================================================================
// Logit reductions
// =============================================================================
// Row argmax with the lowest index winning ties.  logits fp32 [rows, ld].
// Replaces `.argmax(dim=-1)` on logits_out (fast_generate.py:786,809,1079) and
// the max of _fused_draft_chain (fast_generate.py:125).  One CTA per row.
__global__ void __launch_bounds__(1024) argmax_rows_kernel(const float *__restrict__ logits,
                                                           int vocab, int ld,
                                                           int64_t *__restrict__ idx,
                                                           float *__restrict__ max_out) {
    __shared__ float sv[32];
    __shared__ int si[32];
    const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float *x = logits + (size_t)r * ld;
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int v = threadIdx.x; v < vocab; v += blockDim.x) {
        const float f = x[v];
        if (bm_argmax_better(f, v, best, bi)) { best = f; bi = v; }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (bm_argmax_better(ob, oi, best, bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { sv[warp] = best; si[warp] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
            if (bm_argmax_better(sv[w], si[w], best, bi)) { best = sv[w]; bi = si[w]; }
        idx[r] = bi;
        if (max_out) max_out[r] = best;
    }
}

// Sum of exp(x - max) per row in the oracle's chunk order (256-element chunks:
// 32 lanes x 8 consecutive terms, butterfly, chunks added in ascending order),
// then conf = exp(max - (max + log(sum))).  One CTA of 8 warps per row: warp w
// takes chunks w, w+8, ... and keeps their sums in shared memory; thread 0 adds
// them in order.  Part of _fused_draft_chain (fast_generate.py:126-127).
constexpr int kConfMaxChunks = 1024;   // vocab <= 262144

__global__ void __launch_bounds__(256) row_confidence_kernel(const float *__restrict__ logits,
                                                             int vocab, int ld,
                                                             const float *__restrict__ row_max,
                                                             float *__restrict__ conf) {
    __shared__ float chunk_sum[kConfMaxChunks];
    const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float *x = logits + (size_t)r * ld;
    const float mx = row_max[r];
    const int nchunks = (vocab + 255) / 256;
    for (int c = warp; c < nchunks; c += 8) {
        float acc = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int v = c * 256 + lane * 8 + e;
            if (v < vocab) acc += bm_expf(x[v] - mx);
        }
        acc = warp_sum_butterfly(acc);
        if (lane == 0) chunk_sum[c] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float total = 0.0f;
        for (int c = 0; c < nchunks; ++c) total += chunk_sum[c];
        const float lse = mx + bm_logf(total);
        conf[r] = bm_expf(mx - lse);
    }
}

// iter_accept = 1 + longest prefix of rows r >= 1 with conf[r] > tau
// (fast_generate.py:128-129); accept = longest prefix with draft == verify
// (fast_generate.py:146).  Single-thread kernels over <= 32 values.
__global__ void chain_length_kernel(const float *conf, int D, float tau, int *out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int n = 1;
    for (int r = 1; r < D; ++r) {
        if (conf[r] > tau) ++n; else break;
    }
    *out = n;
}

// ---- the same reductions spread over many CTAs ------------------------------------------------
// One CTA per logit row leaves 140 of 148 SMs idle on rows of 151936 values (measured: 129 us for the
// confidence chain of 8 rows, 37 us for an argmax).  Here a row is cut into S ranges of whole 256-element
// chunks, one CTA each (S = logit_splits(rows): more ranges when there are few rows); the last CTA of a row to finish (a
// ticket counter in the caller's scratch) combines the row, and for the confidence chain the last row
// to finish computes the chain length.  Results are identical to the one-CTA kernels: the argmax
// comparison does not depend on order, the chunk sums are the same chunk sums and are added in ascending
// chunk order by one thread.  Scratch (LogitScratch, zero before first use; the kernels leave the
// counters zero again).
constexpr int kLogitMaxRows = 32;
constexpr int kLogitMaxParts = 512;      // rows * S

__host__ __device__ inline int logit_splits(int rows) {
    int s = kLogitMaxParts / rows;       // 16 at 32 rows
    return s > 128 ? 128 : (s > 32 && rows > 2 ? 32 : s);
}

struct LogitScratch {
    unsigned int arg_tickets[kLogitMaxRows];
    unsigned int conf_tickets[kLogitMaxRows];
    unsigned int rows_done;
    unsigned int pad[63];
    float part_max[kLogitMaxParts];
    int part_idx[kLogitMaxParts];
    float chunk_sum[kLogitMaxRows * kConfMaxChunks];
};

__device__ __forceinline__ void logit_split_range(int vocab, int split, int S, int &v_lo, int &v_hi) {
    const int nchunks = (vocab + 255) / 256;
    const int per = (nchunks + S - 1) / S;
    v_lo = min(vocab, split * per * 256);
    v_hi = min(vocab, (split + 1) * per * 256);
}

// grid (S, rows), 256 threads
__global__ void __launch_bounds__(256) argmax_split_kernel(const float *__restrict__ logits, int vocab, int ld,
                                                          int64_t *__restrict__ idx, float *__restrict__ max_out,
                                                          LogitScratch *sc) {
    __shared__ float sv[8];
    __shared__ int si[8];
    __shared__ unsigned int ticket;
    const int split = blockIdx.x, S = gridDim.x, r = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float *x = logits + (size_t)r * ld;
    int v_lo, v_hi;
    logit_split_range(vocab, split, S, v_lo, v_hi);
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int v = v_lo + threadIdx.x; v < v_hi; v += 256) {
        const float f = x[v];
        if (bm_argmax_better(f, v, best, bi)) { best = f; bi = v; }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (bm_argmax_better(ob, oi, best, bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { sv[warp] = best; si[warp] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w)
            if (bm_argmax_better(sv[w], si[w], best, bi)) { best = sv[w]; bi = si[w]; }
        sc->part_max[r * S + split] = best;
        sc->part_idx[r * S + split] = bi;
        __threadfence();
        ticket = atomicAdd(&sc->arg_tickets[r], 1u);
    }
    __syncthreads();
    if (ticket != (unsigned int)(S - 1) || threadIdx.x != 0) return;
    // last CTA of the row: every partial is visible
    __threadfence();
    best = -INFINITY;
    bi = 0x7fffffff;
    for (int s = 0; s < S; ++s) {
        const float f = __ldcg(&sc->part_max[r * S + s]);
        const int i = __ldcg(&sc->part_idx[r * S + s]);
        if (bm_argmax_better(f, i, best, bi)) { best = f; bi = i; }
    }
    idx[r] = bi;
    if (max_out) max_out[r] = best;
    sc->arg_tickets[r] = 0u;
}

// grid (S, D), 256 threads.  row_max[r] must be final (argmax_split_kernel of the same rows has
// completed: stream order).  The last row to finish writes the chain length.
__global__ void __launch_bounds__(256) confidence_split_kernel(const float *__restrict__ logits, int vocab, int ld,
                                                              const float *__restrict__ row_max,
                                                              float *__restrict__ conf, int D, float tau,
                                                              int *__restrict__ n_out, LogitScratch *sc) {
    __shared__ unsigned int ticket;
    const int split = blockIdx.x, S = gridDim.x, r = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float *x = logits + (size_t)r * ld;
    const float mx = row_max[r];
    const int nchunks = (vocab + 255) / 256;
    const int per = (nchunks + S - 1) / S;
    const int c_lo = min(nchunks, split * per), c_hi = min(nchunks, (split + 1) * per);
    float *sums = sc->chunk_sum + (size_t)r * kConfMaxChunks;
    const bool vec = (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
    for (int c = c_lo + warp; c < c_hi; c += 8) {
        const int v0 = c * 256 + lane * 8;
        float acc = 0.0f;
        if (vec && v0 + 8 <= vocab) {
            const float4 a = *reinterpret_cast<const float4 *>(x + v0), b = *reinterpret_cast<const float4 *>(x + v0 + 4);
            acc += bm_expf(a.x - mx); acc += bm_expf(a.y - mx); acc += bm_expf(a.z - mx); acc += bm_expf(a.w - mx);
            acc += bm_expf(b.x - mx); acc += bm_expf(b.y - mx); acc += bm_expf(b.z - mx); acc += bm_expf(b.w - mx);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (v0 + e < vocab) acc += bm_expf(x[v0 + e] - mx);
        }
        acc = warp_sum_butterfly(acc);
        if (lane == 0) sums[c] = acc;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        ticket = atomicAdd(&sc->conf_tickets[r], 1u);
    }
    __syncthreads();
    if (ticket != (unsigned int)(S - 1)) return;
    // last CTA of the row: add the chunk sums in ascending order.  All threads fetch them into shared memory
    // first (one round trip instead of one per addend); thread 0 then adds them in the same order as before.
    __threadfence();
    __shared__ float staged[kConfMaxChunks];
    for (int c = threadIdx.x; c < nchunks; c += blockDim.x) staged[c] = __ldcg(&sums[c]);
    __syncthreads();
    if (threadIdx.x != 0) return;
    float total = 0.0f;
    for (int c = 0; c < nchunks; ++c) total += staged[c];
    const float lse = mx + bm_logf(total);
    conf[r] = bm_expf(mx - lse);
    sc->conf_tickets[r] = 0u;
    __threadfence();
    if (atomicAdd(&sc->rows_done, 1u) != (unsigned int)(D - 1)) return;
    // last row: the chain length over all confidences
    __threadfence();
    int n = 1;
    for (int q = 1; q < D; ++q) {
        if (__ldcg(&conf[q]) > tau) ++n; else break;
    }
    *n_out = n;
    sc->rows_done = 0u;
}

// ---- the confidence chain of a draft block in ONE launch -----------------------------------------
// argmax_split_kernel + confidence_split_kernel as one kernel: the kDraftClusterCtas CTAs of a logit row are a
// thread-block cluster (grid (kDraftClusterCtas, D), cluster (kDraftClusterCtas, 1, 1)).  Each CTA reads its
// range of whole 256-element chunks ONCE, into shared memory, and finds its maximum; the partial maxima go to
// every CTA of the cluster through distributed shared memory, so after one cluster barrier each CTA knows the
// row's maximum and argmax (same comparison, ranges in ascending order) and sums exp(x - max) over its chunks
// from shared memory in the oracle's order (lane = 8 consecutive terms, butterfly); the chunk sums go to the
// first CTA of the cluster, which after a second barrier adds them in ascending order and finishes the row as
// confidence_split_kernel does (the last row to finish writes the chain length).  Same results, one launch
// instead of two, the logits read once instead of twice, no fence / ticket / read-back inside a row.
constexpr int kDraftClusterCtas = 16;

__global__ void __launch_bounds__(256) draft_chain_cluster_kernel(const float *__restrict__ logits, int vocab, int ld,
                                                                 int64_t *__restrict__ idx, float *__restrict__ max_out,
                                                                 float *__restrict__ conf, int D, float tau,
                                                                 int *__restrict__ n_out, LogitScratch *sc) {
    extern __shared__ __align__(16) float slice[];            // this CTA's chunks of the row
    __shared__ float sv[8];
    __shared__ int si[8];
    __shared__ float part_max[kDraftClusterCtas];
    __shared__ int part_idx[kDraftClusterCtas];
    __shared__ float sums[kConfMaxChunks];                    // chunk sums of the whole row (used in CTA 0)
    __shared__ float row_best;
    __shared__ int row_idx;
    const int rank = blockIdx.x, r = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    cluster_arrive();                      // waited for below, before the first store into another CTA: all have started
    const float *x = logits + (size_t)r * ld;
    const int nchunks = (vocab + 255) / 256;
    const int per = (nchunks + kDraftClusterCtas - 1) / kDraftClusterCtas;
    const int c_lo = min(nchunks, rank * per), c_hi = min(nchunks, (rank + 1) * per);
    const int v_lo = min(vocab, c_lo * 256), v_hi = min(vocab, c_hi * 256);
    // the whole range is requested at once (16-byte asynchronous copies where the row is aligned for them, so
    // that a thread has all its loads in flight together), then scanned from shared memory
    const int len = v_hi - v_lo;
    const bool vec = (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
    const int len4 = vec ? len / 4 : 0;
    for (int i = threadIdx.x; i < len4; i += 256) cp_async16(slice + 4 * i, x + v_lo + 4 * i);
    for (int i = 4 * len4 + threadIdx.x; i < len; i += 256) slice[i] = x[v_lo + i];
    cp_async_wait_all();
    __syncthreads();
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < len; i += 256) {
        const float f = slice[i];
        if (bm_argmax_better(f, v_lo + i, best, bi)) { best = f; bi = v_lo + i; }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (bm_argmax_better(ob, oi, best, bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { sv[warp] = best; si[warp] = bi; }
    __syncthreads();
    cluster_wait();
    if (warp == 0) {
        // lane t hands this CTA's partial to CTA t of the cluster
        best = sv[0]; bi = si[0];
        for (int w = 1; w < 8; ++w)
            if (bm_argmax_better(sv[w], si[w], best, bi)) { best = sv[w]; bi = si[w]; }
        if (lane < kDraftClusterCtas) {
            cluster_st_f32(cluster_map(&part_max[rank], (uint32_t)lane), best);
            cluster_st_s32(cluster_map(&part_idx[rank], (uint32_t)lane), bi);
        }
    }
    cluster_arrive();
    cluster_wait();
    if (threadIdx.x == 0) {
        best = -INFINITY;
        bi = 0x7fffffff;
        for (int s = 0; s < kDraftClusterCtas; ++s)
            if (bm_argmax_better(part_max[s], part_idx[s], best, bi)) { best = part_max[s]; bi = part_idx[s]; }
        row_best = best;
        row_idx = bi;
    }
    __syncthreads();
    const float mx = row_best;
    for (int c = c_lo + warp; c < c_hi; c += 8) {
        const int v0 = c * 256 + lane * 8;
        float acc = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (v0 + e < vocab) acc += bm_expf(slice[v0 + e - v_lo] - mx);
        acc = warp_sum_butterfly(acc);
        if (lane == 0) cluster_st_f32(cluster_map(&sums[c], 0u), acc);
    }
    cluster_arrive();
    cluster_wait();
    if (rank != 0 || threadIdx.x != 0) return;
    float total = 0.0f;
    for (int c = 0; c < nchunks; ++c) total += sums[c];
    const float lse = mx + bm_logf(total);
    conf[r] = bm_expf(mx - lse);
    idx[r] = row_idx;
    max_out[r] = mx;
    __threadfence();
    if (atomicAdd(&sc->rows_done, 1u) != (unsigned int)(D - 1)) return;
    // last row: the chain length over all confidences
    __threadfence();
    int n = 1;
    for (int q = 1; q < D; ++q) {
        if (__ldcg(&conf[q]) > tau) ++n; else break;
    }
    *n_out = n;
    sc->rows_done = 0u;
}

__global__ void verify_accept_kernel(const int64_t *draft, const int64_t *verify, int D, int *out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int n = 0;
    while (n < D && draft[n] == verify[n]) ++n;
    *out = n;
}

}  // namespace bm
