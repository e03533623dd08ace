// Packed T2-g128 product for MANY rows at once (a prompt): C[T, N] = ((A x ternary(B)) per-group
// scaled) / s, every row bit-identical to what the decode GEMV (t2_gemv.cuh) gives that row alone.
//
// Replaces, for the prompt forward, the dense fallback of T2LinearKernel.forward
// (src/bonsai_sft/gpu/model.py:650-656: unpack the layer to bf16, fake-quantise, cuBLAS) behind
// forward_sdlm_prefill (model.py:1306-1340).  Here the prompt goes through the packed integer path
// and nothing dense is ever materialised.
//
// The contraction runs on the 5th-generation tensor cores: tcgen05.mma kind::i8 with 128 weight rows
// as M (A operand: the u8 codes, expanded 2 -> 8 bits in registers and kept in TENSOR MEMORY, so they
// cost no shared-memory bandwidth), NT prompt rows as N (B operand: the s8 activations, a 128-byte-
// swizzled tile that TMA brings) and four K = 32 steps per 128-group.  An accumulator is one group's
// integer sum of code * a: the format has one scale per 128 weights and the canonical fp32 order (header
// of t2_gemv.cuh) one fma per group, so the fp32 side costs per output and group a subtraction, an fma and
// a tree addition, done two outputs at a time (f32x2).  Accumulators are set to kGroupSumBias before the
// MMAs: the int32 that comes out is then the bit pattern of the float 1.5*2^23 + sum, and subtracting the
// column's 1.5*2^23 + 2*sum(a) gives (float)G exactly, without the quarter-rate conversion.
//
// Measured (us; before: mma.sync tiles of 128 x 32 with the codes unpacked by every warp): 12288 x 2048, 1024 rows
// 149.5 -> 88.5, 2048 x 6144, 1024 rows 82.3 -> 46.0, 19456 x 2560, 1024 rows 311 -> 187, 4096 x 2048, 17 rows 12.6 -> 10.4.
// Bound by instruction issue (73 % of the slots; 2660 warp instructions per 128 x 64 x 128 block), then by the per-step
// hand-over of one tile; the MMAs of a group take 240 cycles whatever NT is, 1000 pass.  16 columns a worker (not 32: 103 us)
// put four worker warps on a scheduler; two groups a step halve the waits (8 x 51200: 180 -> 121 us); the scales and column
// constants come through a ring, because as tables of the tile they stopped every warp for 4700 cycles at its start.
//
// fp32 order: group g -> slot g % 16, slot = fma(G, scale, slot) in ascending g, the 16 slots summed as
// a butterfly tree, times 1/s.  Groups are visited slot by slot; a finished slot goes into a binary
// counter: sums of one and two slots wait in registers, of four and eight in shared memory.
//
// Roles in a CTA, by warp:
//   workers    NT/16 x 4 (warp w: TMEM lanes 32 (w % 4).., i.e. weight rows, and 16 columns): every group's
//              accumulator -> fp32 slots and tree, then the output;
//   expanders  4 (one per 32 weight rows): a group's codes 2 -> 8 bits into TMEM; the group's scales and
//              column constants into shared memory, fetched two groups ahead;
//   one lane issues the MMAs, one lane of another warp the TMA copies.
// Rings: stages (TMA), kTcABufs code buffers and as many accumulators (TMEM), kTcTabs scale / constant
// tables.  Persistent: a CTA walks tiles blockIdx.x, + gridDim.x, ..., and the rings run on across tiles.
#pragma once

#include "bm_common.cuh"
#include "t2_gemv_rowwarp.cuh"

#include <type_traits>

namespace bm {

constexpr int kTcRows = 128;            // weight rows per tile
constexpr int kTcCols = 16;             // columns per worker warp
constexpr int kTcStep = 2;              // groups per step of the rings: one wait, commit and hand-over for both
constexpr int kTcBufs = 2;              // steps of expanded codes (32 TMEM columns a group) and of accumulators
constexpr int kTcStages = 4;            // TMA stages (steps)
constexpr int kTcDone = 4;              // barriers of ended MMAs (>= kTcStages, > kTcBufs: no waiter is lapped)
constexpr int kTcTabs = 8;              // steps of tables: a worker that has read step u is done with the tables of u - 1
enum : int { kErrGemmWaitTimeout = 5 };

struct TcParams {
    CUtensorMap a_map;      // activations [T, K] int8, box NT x 128 bytes, 128-byte swizzle
    CUtensorMap b_map;      // codes [N, K/4], box 128 x 32 bytes, 32-byte swizzle
    const int32_t *asum;    // [T, K/128]
    const float *s;         // [T]
    const uint16_t *ws;     // [N, K/128] bf16
    uint16_t *C;            // [T, ldc] bf16
    int T, N, K, ldc, pdl, tiles, t_tiles;
};

__host__ __device__ constexpr int tc_workers(int NT) { return NT / kTcCols * 4; }
__host__ __device__ constexpr int tc_threads(int NT) { return (tc_workers(NT) + 6) * 32; }
__host__ __device__ constexpr int tc_tmem_cols(int NT) { return kTcBufs * kTcStep * (NT + 32) <= 256 ? 256 : 512; }
__host__ __device__ constexpr int tc_stage_bytes(int NT) { return kTcStep * (NT * 128 + kTcRows * 32); }
__host__ __device__ constexpr int tc_table_floats(int NT) { return kTcRows + NT; }          // per group: scales of the rows, constants of the columns
// stages, sums of four and of eight slots, tables, 1/s of the workers' columns; slack to align the stages
__host__ __device__ constexpr int tc_smem_bytes(int NT) {
    return kTcStages * tc_stage_bytes(NT) + 2 * kTcRows * NT * 4 + kTcTabs * kTcStep * tc_table_floats(NT) * 4 + NT * 4 * 4 + 1024;
}

// ---- tcgen05 wrappers ---------------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 16 columns of this warp's 32 lanes.  The wait belongs to the load, so that nothing uses the registers before it (as a
// statement of its own with the registers as operands it made the compiler copy all of them).
__device__ __forceinline__ void tc_ld16(uint32_t (&x)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];\n\ttcgen05.wait::ld.sync.aligned;"
        : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7]), "=r"(x[8]),
          "=r"(x[9]), "=r"(x[10]), "=r"(x[11]), "=r"(x[12]), "=r"(x[13]), "=r"(x[14]), "=r"(x[15])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t addr, const uint32_t (&x)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15};"
        ::"r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(x[8]), "r"(x[9]),
        "r"(x[10]), "r"(x[11]), "r"(x[12]), "r"(x[13]), "r"(x[14]), "r"(x[15]), "r"(addr)
        : "memory");
}

// The same value into 16 columns.  `v`: four registers that hold it (given one, the compiler copies it for every store).
__device__ __forceinline__ void tc_fill16(uint32_t addr, const uint32_t (&v)[4]) {
#pragma unroll
    for (int c = 0; c < 16; c += 4)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
                     ::"r"(addr + c), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}

// D[128 x N] += A (TMEM, u8) x B (shared memory, s8), K = 32.
__device__ __forceinline__ void tc_mma_i8(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, 1, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc) : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_tma_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint4 tc_lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t tc_add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t tc_pack(uint32_t lo, uint32_t hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
    return d;
}
__device__ __forceinline__ float2 tc_unpack(uint64_t v) {
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
    return make_float2(__uint_as_float(lo), __uint_as_float(hi));
}

// Shared-memory descriptor of a K-major tile with the 128-byte swizzle: rows of 128 bytes, 1024 bytes per 8 rows.
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3ffff) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

// The slot-major sequence of groups: slot s (0..15) has groups s, s + 16, ...
__device__ __forceinline__ void tc_next_group(int &g, int ng) {
    g += BM_SLOTS;
    if (g < ng) return;
    g = (g & (BM_SLOTS - 1)) + 1;
    if (g >= ng || g == BM_SLOTS) g = 0;                       // the last slot that has a group is done
}

// Wait for a phase with an iteration limit.  When it runs out, or another wait of the CTA has run out, the caller goes on
// with whatever is there (every later wait then returns at once), and the CTA reports the error when it ends.
__device__ __forceinline__ void tc_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
    uint32_t it = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (*abort_flag) return;
        if (++it > (1u << 22)) *abort_flag = 1;
    }
}

// ONE: K == 2048, one group per slot: a step is a pair of slots.
template <int NT, bool ONE>
__global__ void __launch_bounds__(tc_threads(NT), NT == 32 ? 2 : 1) t2_gemm_tc_kernel(const __grid_constant__ TcParams p) {
    extern __shared__ unsigned char tc_raw[];
    __shared__ uint64_t full[kTcStages], ready[kTcBufs], done[kTcDone];
    __shared__ uint32_t tmem_base_sh;
    __shared__ int abort_flag;
    constexpr int NW = tc_workers(NT), kStage = tc_stage_bytes(NT), kTab = tc_table_floats(NT);
    constexpr int kCodes = kTcStep * NT * 128;                   // a stage: both groups' prompt rows, then both groups' codes
    constexpr uint32_t kACol = kTcBufs * kTcStep * NT;
    constexpr uint32_t kIdesc = (2u << 4) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kTcRows >> 4) << 24);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int ng = p.K / BM_GROUP;                       // the last step of a tile may hold one group
    unsigned char *sm = tc_raw + ((1024 - (smem_u32(tc_raw) & 1023)) & 1023);
    float4 *sums = reinterpret_cast<float4 *>(sm + kTcStages * kStage);
    float *tabs = reinterpret_cast<float *>(sm + kTcStages * kStage + 2 * kTcRows * NT * 4);
    float *inv = tabs + kTcTabs * kTcStep * kTab;

    if (warp == NW + 4) {
        if (lane == 0) {
            for (int i = 0; i < kTcStages; ++i) mbar_init(&full[i], 1);
            for (int i = 0; i < kTcBufs; ++i) mbar_init(&ready[i], 4 + NW);
            for (int i = 0; i < kTcDone; ++i) mbar_init(&done[i], 1);
            abort_flag = 0;
            mbar_fence_init();
        }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                     "r"((uint32_t)tc_tmem_cols(NT)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_sh, lanes = (uint32_t)((warp & 3) * 32) << 16;
    pdl_launch_dependents();
    if (p.pdl) pdl_wait();

    if (warp == NW + 5) {
        // ---- copies ---------------------------------------------------------------------------------------
        if (lane == 0) {
            int u = 0;
            for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
                const int n0 = (tile / p.t_tiles) * kTcRows, t0 = (tile % p.t_tiles) * NT;
                int g = 0;
                for (int i = 0; i < ng; i += kTcStep, ++u) {
                    const int st = u & (kTcStages - 1), n = ng - i < kTcStep ? 1 : kTcStep;
                    // the stage is free once the MMAs of the step that used it have ended (its codes were read before them)
                    if (u >= kTcStages) tc_wait(&done[st], (uint32_t)((u - kTcStages) / kTcDone) & 1, &abort_flag);
                    unsigned char *buf = sm + st * kStage;
                    mbar_expect_tx(&full[st], (uint32_t)(n * (kStage / kTcStep)));
                    for (int k = 0; k < n; ++k) {
                        tc_tma_2d(buf + k * NT * 128, &p.a_map, g * BM_GROUP, t0, &full[st]);
                        tc_tma_2d(buf + kCodes + k * kTcRows * 32, &p.b_map, g * (BM_GROUP / 4), n0, &full[st]);
                        tc_next_group(g, ng);
                    }
                }
            }
            // after an error some stages may not have been waited for: give their copies a bounded chance to land
            if (abort_flag)
                for (int r = u > kTcStages ? u - kTcStages : 0; r < u; ++r)
                    for (int it = 0; it < (1 << 12); ++it)
                        if (mbar_try_wait(&full[r & (kTcStages - 1)], (uint32_t)(r / kTcStages) & 1)) break;
        }
        __syncwarp();
    } else if (warp == NW + 4) {
        // ---- MMAs -----------------------------------------------------------------------------------------
        if (lane == 0) {
            const uint64_t desc0 = tc_desc(smem_u32(sm));
            int u = 0;
            for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
                for (int i = 0; i < ng; i += kTcStep, ++u) {
                    const int b = u & (kTcBufs - 1);
                    // the step's codes are in TMEM (so its stage has arrived) and its accumulators have been read
                    tc_wait(&ready[b], (uint32_t)(u / kTcBufs) & 1, &abort_flag);
                    tc_fence_after();
                    const uint64_t desc = desc0 + (uint32_t)((u & (kTcStages - 1)) * (kStage >> 4));
#pragma unroll
                    for (int h = 0; h < kTcStep; ++h) {
                        if (i + h >= ng) break;
                        const int a = b * kTcStep + h;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            tc_mma_i8(tmem + a * NT, tmem + kACol + a * 32 + 8 * k, desc + h * (NT * 128 >> 4) + 2 * k, kIdesc);
                    }
                    tc_commit(&done[u & (kTcDone - 1)]);
                }
            }
            if (u > 0) tc_wait(&done[(u - 1) & (kTcDone - 1)], (uint32_t)((u - 1) / kTcDone) & 1, &abort_flag);
        }
        __syncwarp();
    } else if (warp >= NW) {
        // ---- expanders ------------------------------------------------------------------------------------
        // Word w of a row (16 codes) gives four registers, bit plane t holding codes 4e + t, which is the order of
        // GEMV-ready activations.
        const int q = warp & 3, row = q * 32 + lane;
        const uint32_t code0 = smem_u32(sm) + kCodes + row * 32 + 16 * ((row >> 2) & 1);
        const bool has_col = lane < NT / 4;
        // scales and constants of the next step, fetched a step ahead
        const uint16_t *ws_row = nullptr;
        const int32_t *as_row = nullptr;
        int cg = 0, ci = 0, ct = blockIdx.x;
        auto fetch = [&](uint32_t (&sc)[kTcStep], int (&as)[kTcStep]) {
            if (ct >= p.tiles) return;
            if (ci == 0) {
                ws_row = p.ws + (size_t)min((ct / p.t_tiles) * kTcRows + row, p.N - 1) * ng;
                const int t = (ct % p.t_tiles) * NT + q * (NT / 4) + lane;
                as_row = has_col && t < p.T ? p.asum + (size_t)t * ng : nullptr;
            }
#pragma unroll
            for (int h = 0; h < kTcStep; ++h) {
                if (ci + h < ng) {
                    sc[h] = __ldg(ws_row + cg);
                    as[h] = as_row != nullptr ? __ldg(as_row + cg) : 0;
                    tc_next_group(cg, ng);
                }
            }
            ci += kTcStep;
            if (ci >= ng) { ci = 0; ct += gridDim.x; }
        };
        uint32_t sc[kTcStep] = {}, sn[kTcStep] = {};
        int as[kTcStep] = {}, an[kTcStep] = {}, u = 0;
        fetch(sc, as);
        for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
            for (int i = 0; i < ng; i += kTcStep, ++u) {
                const int st = u & (kTcStages - 1), b = u & (kTcBufs - 1);
                fetch(sn, an);
                tc_wait(&full[st], (uint32_t)(u / kTcStages) & 1, &abort_flag);
                // the code buffers are free, and the tables of step u - kTcTabs have been read
                if (u >= kTcBufs) tc_wait(&done[(u - kTcBufs) & (kTcDone - 1)], (uint32_t)((u - kTcBufs) / kTcDone) & 1, &abort_flag);
                __syncwarp();
                tc_fence_after();
                const uint32_t a0 = code0 + st * kStage;
                float *tab = tabs + (u & (kTcTabs - 1)) * (kTcStep * kTab);
                uint4 x[kTcStep][2];
#pragma unroll
                for (int h = 0; h < kTcStep; ++h)
#pragma unroll
                    for (int k = 0; k < 2; ++k) x[h][k] = tc_lds128((a0 + h * kTcRows * 32) ^ (16u * k));
#pragma unroll
                for (int h = 0; h < kTcStep; ++h) {
                    tab[h * kTab + row] = __uint_as_float(sc[h] << 16);
                    if (has_col) tab[h * kTab + kTcRows + q * (NT / 4) + lane] = -(float)(12582912 + 2 * as[h]);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const uint32_t wv[4] = {x[h][k].x, x[h][k].y, x[h][k].z, x[h][k].w};
                        uint32_t a[16];
#pragma unroll
                        for (int w = 0; w < 4; ++w)
#pragma unroll
                            for (int t = 0; t < 4; ++t) a[4 * w + t] = (wv[w] >> (2 * t)) & 0x03030303u;
                        tc_st16(tmem + lanes + kACol + (b * kTcStep + h) * 32 + 16 * k, a);
                    }
                    sc[h] = sn[h];
                    as[h] = an[h];
                }
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ready[b]);
            }
        }
    } else {
        // ---- workers --------------------------------------------------------------------------------------
        const int cb = warp >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t acc0 = tmem + lanes + cb * kTcCols;
        ulonglong2 *l4 = reinterpret_cast<ulonglong2 *>(sums) + tid, *l8 = l4 + 4 * NW * 32;     // this thread's, every NW * 32
        uint32_t bias[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) asm volatile("mov.u32 %0, %1;" : "=r"(bias[c]) : "n"(kGroupSumBias));
#pragma unroll
        for (int a = 0; a < kTcBufs * kTcStep; ++a) tc_fill16(acc0 + a * NT, bias);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0)
            for (int b = 0; b < kTcBufs; ++b) mbar_arrive(&ready[b]);
        int u = 0, half = 0, left = ng;              // step, group of the step, groups of the tile still to come

        auto enter = [&]() {
            tc_wait(&done[u & (kTcDone - 1)], (uint32_t)(u / kTcDone) & 1, &abort_flag);
            // (complete since before the MMAs; the expanders' tables are read after it)
            tc_wait(&ready[u & (kTcBufs - 1)], (uint32_t)(u / kTcBufs) & 1, &abort_flag);
            __syncwarp();
            tc_fence_after();
        };
        // the step's accumulators, set to the bias again, may take step u + kTcBufs
        auto leave = [&]() {
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[u & (kTcBufs - 1)]);
            ++u;
        };
        // Group h of the step: acc = fma((float)G, scale, acc) for this thread's row and 16 columns.  FIRST: the product (the
        // first fma of a slot adds to zero; a product of minus zero is undone where the sixteen slots have been added).
        auto group = [&](uint64_t (&acc)[8], int h, auto first) {
            const uint32_t addr = acc0 + ((u & (kTcBufs - 1)) * kTcStep + h) * NT;
            const float *tab = tabs + ((u & (kTcTabs - 1)) * kTcStep + h) * kTab;
            const float sc = tab[row];
            const uint64_t sc2 = tc_pack(__float_as_uint(sc), __float_as_uint(sc));
            const ulonglong2 *cp = reinterpret_cast<const ulonglong2 *>(tab + kTcRows + cb * kTcCols);
            uint32_t x[16];
            tc_ld16(x, addr);
            tc_fill16(addr, bias);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const ulonglong2 k2 = cp[c];
                const uint64_t lo = tc_add2(tc_pack(x[4 * c], x[4 * c + 1]), k2.x);
                const uint64_t hi = tc_add2(tc_pack(x[4 * c + 2], x[4 * c + 3]), k2.y);
                if (decltype(first)::value) {
                    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(acc[2 * c]) : "l"(lo), "l"(sc2));
                    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(acc[2 * c + 1]) : "l"(hi), "l"(sc2));
                } else {
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[2 * c]) : "l"(lo), "l"(sc2));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[2 * c + 1]) : "l"(hi), "l"(sc2));
                }
            }
        };
        auto step = [&](uint64_t (&acc)[8], auto first) {
            if (half == 0) enter();
            group(acc, half, first);
            --left;
            if (half == kTcStep - 1 || left == 0) {
                leave();
                half = 0;
            } else {
                ++half;
            }
        };
        auto slot = [&](uint64_t (&acc)[8], int g) {
            if (g < ng) step(acc, std::true_type());
            else {
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[c] = 0ull;
            }
#pragma unroll 1
            for (g += BM_SLOTS; g < ng; g += BM_SLOTS) step(acc, std::false_type());
        };

        for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
            const int n = (tile / p.t_tiles) * kTcRows + row, t0 = (tile % p.t_tiles) * NT + cb * kTcCols;
            const float s_col = lane < kTcCols && t0 + lane < p.T ? __ldg(p.s + t0 + lane) : 1.0f;
            uint64_t acc[8], one[8], two[8];
            left = ng;
#pragma unroll 1
            for (int pair = 0; pair < 8; ++pair) {             // slots 2 pair, 2 pair + 1
                if (ONE) {
                    enter();
                    group(one, 0, std::true_type());
                    group(acc, 1, std::true_type());
                    leave();
                } else {
                    slot(one, 2 * pair);
                    slot(acc, 2 * pair + 1);
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[c] = tc_add2(one[c], acc[c]);
                if ((pair & 1) == 0) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) two[c] = acc[c];
                    continue;
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[c] = tc_add2(two[c], acc[c]);
                // four slots summed: the higher levels of the tree
                if ((pair & 2) == 0) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) l4[c * NW * 32] = make_ulonglong2(acc[2 * c], acc[2 * c + 1]);
                    continue;
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const ulonglong2 v = l4[c * NW * 32];
                    acc[2 * c] = tc_add2(v.x, acc[2 * c]);
                    acc[2 * c + 1] = tc_add2(v.y, acc[2 * c + 1]);
                }
                if (pair == 3) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) l8[c * NW * 32] = make_ulonglong2(acc[2 * c], acc[2 * c + 1]);
                }
            }
            // (a warp's 1/s: its own 16 words)
            if (lane < kTcCols) inv[warp * kTcCols + lane] = 1.0f / s_col;
            __syncwarp();
            const float4 *iv = reinterpret_cast<const float4 *>(inv + warp * kTcCols);
            uint16_t *dst = p.C + (size_t)t0 * p.ldc + n;
            const int live = n < p.N ? p.T - t0 : 0;                              // prompt rows to store
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const ulonglong2 v = l8[c * NW * 32];
                const float4 i4 = iv[c];
                const float2 lo = tc_unpack(tc_add2(tc_add2(v.x, acc[2 * c]), 0ull)), hi = tc_unpack(tc_add2(tc_add2(v.y, acc[2 * c + 1]), 0ull));
                const float y[4] = {lo.x * i4.x, lo.y * i4.y, hi.x * i4.z, hi.y * i4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (4 * c + e < live) *dst = bm_f32_to_bf16(y[e]);
                    dst += p.ldc;
                }
            }
            __syncwarp();
        }
    }
    // every MMA has ended (the issuing lane waited for the last one) and every worker has read what it needs
    tc_fence_before();
    __syncthreads();
    if (warp == NW + 4) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)tc_tmem_cols(NT)) : "memory");
    }
    if (tid == 0 && abort_flag) report_error(kErrGemmWaitTimeout);
}

}  // namespace bm
