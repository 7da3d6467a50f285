// Fused RPTC decode + matvec for one or two activation rows in the TILED layout: the kernel, in the forms that gemv.cu (activations from memory,
// glue of a decode step) and gemv_alone.cu (a layer's input side) launch.
//
// Work decomposition.  Rows are taken 32 at a time (a "row block": lane l owns row 32*rb + l) and a
// row's stream is cut into 128-bit units.  The (row block, unit) grid is flattened row-block-major
// and cut into equal contiguous ranges over a persistent grid of one 512-thread CTA per SM, so that
// every SM gets the same number of units whatever m and n are.  In the native TILED
// layout that flattened order is the memory order: a warp's range is one linear stream of 512-byte
// units.  The 16-bit shift-register windows are rebuilt in registers with funnel shifts and hashed /
// looked up in a shared-memory table.  A warp walks along its rows, so the 16 bits of history a unit
// needs are simply the last word of the unit before it (one extra 32-bit load at the start of a run).
// Partial row sums are added to the fp32 accumulator in global memory with atomics.  W may come in
// banks of rows with a table each: the CTAs are then dealt out to the banks.
//
#pragma once
#include "common.cuh"
#include "fwht.cuh"
#include "matmul.cuh"

#include <type_traits>

namespace rptc {

#ifndef RPTC_GEMV_THREADS
#define RPTC_GEMV_THREADS 512
#endif
#ifndef RPTC_GEMV_STAGES
#define RPTC_GEMV_STAGES 3
#endif
constexpr int kGemvThreads = RPTC_GEMV_THREADS;
constexpr int kGemvWarps = kGemvThreads / 32;
constexpr int kStages = RPTC_GEMV_STAGES;        // ring depth per warp
constexpr int kStageUnits = 2;                   // units per stage: one of each row block of a granule
constexpr uint32_t kUnitBytes = 512;             // 32 rows x 128 bits
constexpr uint32_t kStageBytes = kStageUnits * kUnitBytes;
constexpr uint32_t kBarBytes = 1024;             // the barrier of the table's bulk copy, the glue's sums; the ring starts behind it
constexpr uint32_t kGlueSums = 512, kWarpFirst = 256;
constexpr uint32_t kRingBytes = kGemvWarps * kStages * kStageBytes;
static_assert(kBarBytes + kRingBytes + 1024 <= kHashLutWindow, "ring must fit below the HASH table window");

struct GemvParams {
    const uint4 *codes;
    UnitStrides st;
    const __half *lut;
    const uint32_t *carry_in;
    const __half *x;
    int64_t ld_x;
    float *acc;
    int64_t ld_acc;
    int64_t m, n;
    int32_t n_units, seg_units;
    int32_t L, S, quirk, x_order;
    unsigned int *status;
    // activations computed in the launch (gemv_rows_kernel, MODE 1): the caller's descriptor
    rptc_gemv_input in;
    // gemv_rows_kernel, MODE 2: the gated-MLP middle that produces this layer's activations, and a range to zero
    SwigluParams sw;
    float *clear;
    int64_t clear_count;
    // gemv_rows_kernel, MODE 0: fp16 elements from one bank's table to the next
    int64_t lut_stride;
    // MODE 1: where the glue exchanges values
    int32_t ex_on_ring;
};

// MODE 3 and 4 of gemv_rows_kernel: see GemvInput; sums put down per CTA.
struct GemvAlone {
    const uint4 *codes;
    const __half *lut;
    const uint32_t *carry_in;
    float *acc;                  // the sums, and their rows' distance
    int64_t ld_acc;
    int64_t m, n;
    int32_t n_units, seg_units;
    int32_t L, S;
    unsigned int *status;
    GemvInput in;
    GemvSums sums;
    int64_t lut_stride;
    int32_t ex_on_ring;
};
template <int MODE>
using RowsParams = std::conditional_t<(MODE >= 3), GemvAlone, GemvParams>;

// Source pair of stream pair s under the fused reference kernel's x staging (inference.cu:216-221,249).
__device__ __forceinline__ int64_t k2_legacy_pair(int64_t s, int64_t n) {
    const int64_t it = s >> 10;
    const int lane = (int)(s >> 5) & 31, o = (int)(s >> 2) & 7, j = (int)s & 3;
    const int k = (0x36251407 >> (4 * o)) & 7;       // window register met at stream position o: 7,0,4,1,5,2,6,3
    const int64_t p = ((it * 8 + k) * 4 + j) * 32 + lane;
    const int64_t q8 = n >> 3;
    return 4 * (p % q8) + p / q8;
}

// ---- the input side of a layer, made by every CTA for itself (MODE 3 and 4 below) ---------------------------------------------------
// xs[row] = fp16(x * scales_in); with `sums` the warps' shares of (sum of x, <biases_in, x>) go to red[16 row + warp].
template <int BATCH, typename Hook>
__device__ __forceinline__ void scaled_input(const GemvInput &in, int n, unsigned char *xs, uint32_t stride, float2 *red, bool sums, Hook &&after_loads) {
#pragma unroll 1
    for (int b = 0; b < BATCH; ++b) {
        float s = 0.f, d = 0.f;
        for (int i = 8 * threadIdx.x; i < n; i += 8 * kGemvThreads) {      // n is a multiple of 64
            float f[8];
            const char *src = static_cast<const char *>(in.x) + ((int64_t)b * n + i) * (in.dtype == 2 ? 4 : 2);
            const uint4 r0 = ld_ordered_u128(src);
            uint4 r1 = r0;
            if (in.dtype == 2) r1 = ld_ordered_u128(src + 16);
            const float4 c0 = __ldg(reinterpret_cast<const float4 *>(in.scales_in + i)), c1 = __ldg(reinterpret_cast<const float4 *>(in.scales_in + i) + 1);
            float4 d0 = make_float4(0.f, 0.f, 0.f, 0.f), d1 = d0;
            if (sums) d0 = __ldg(reinterpret_cast<const float4 *>(in.biases_in + i)), d1 = __ldg(reinterpret_cast<const float4 *>(in.biases_in + i) + 1);
            after_loads();
            const uint32_t w[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t pair = w[j >> 1];
                if (in.dtype == 2) f[j] = __uint_as_float(w[j]);
                else if (in.dtype == 1) f[j] = __uint_as_float(j & 1 ? pair & 0xFFFF0000u : pair << 16);
                else f[j] = __half2float(j & 1 ? __high2half(u32_as_half2(pair)) : __low2half(u32_as_half2(pair)));
            }
            uint4 o;
            o.x = half2_as_u32(__floats2half2_rn(f[0] * c0.x, f[1] * c0.y));
            o.y = half2_as_u32(__floats2half2_rn(f[2] * c0.z, f[3] * c0.w));
            o.z = half2_as_u32(__floats2half2_rn(f[4] * c1.x, f[5] * c1.y));
            o.w = half2_as_u32(__floats2half2_rn(f[6] * c1.z, f[7] * c1.w));
            *reinterpret_cast<uint4 *>(xs + b * stride + 2 * i) = o;
            s += ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
            d += ((f[0] * d0.x + f[1] * d0.y) + (f[2] * d0.z + f[3] * d0.w)) + ((f[4] * d1.x + f[5] * d1.y) + (f[6] * d1.z + f[7] * d1.w));
        }
        if (sums) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o), d += __shfl_xor_sync(0xFFFFFFFFu, d, o);
            if ((threadIdx.x & 31) == 0) red[16 * b + (threadIdx.x >> 5)] = make_float2(s, d);
        }
    }
}

// xs = fp16(H(signs * x) * norm) over blocks of in.block (a power of two; n a multiple of it and of 256, at most 4096), one row.  Unit u of
// 256 threads takes columns 2048 u and up, eight a thread; a block of 4096 is the first unit's, sixteen a thread.  ex: kUnitFloats per unit.
template <typename Hook>
__device__ __forceinline__ void transformed_input(const GemvInput &in, int n, __half *xs, float *ex, Hook &&after_loads) {
    const int unit = threadIdx.x / kUnitThreads, t = threadIdx.x & (kUnitThreads - 1);
    float *unit_ex = ex + unit * kUnitFloats;
    const __half *x = static_cast<const __half *>(in.x);
    if (in.block == 4096) {
        if (unit > 0) return;
        uint4 rx[2], rs[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            rx[q] = ld_ordered_u128(x + 16 * t + 8 * q);
            rs[q] = ld_ordered_u128(in.signs + 16 * t + 8 * q);
        }
        after_loads();
        float v[16], sg[16];
        unpack16(rx, v);
        unpack16(rs, sg);
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] *= sg[q];
        unit_transform_to_far(v, unit_ex, t, 1 + unit);
#pragma unroll
        for (int q = 0; q < 16; ++q) xs[t + 256 * q] = __float2half_rn(v[q] * in.norm);
        return;
    }
    const int col = unit * 2048 + 8 * t;
    const bool inside = col < n;                                // of whole warps
    uint4 rx = make_uint4(0u, 0u, 0u, 0u), rs = rx;
    if (inside) rx = ld_ordered_u128(x + col), rs = ld_ordered_u128(in.signs + col);
    after_loads();
    float v[8], sg[8];
    unpack8(rx, v);
    unpack8(rs, sg);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] *= sg[i];
#pragma unroll
    for (int h = 1; h < 8; h <<= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if ((i & h) == 0) {
                const float a = v[i], b = v[i + h];
                v[i] = a + b;
                v[i + h] = a - b;
            }
    for (int lm = 1; lm < 32 && 8 * lm < in.block; lm <<= 1) {
        const bool upper = (t & lm) != 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float o = __shfl_xor_sync(0xFFFFFFFFu, v[i], lm);
            v[i] = upper ? o - v[i] : v[i] + o;
        }
    }
    if (in.block > 256) {                                       // groups of 256 columns through shared memory: a thread takes column r of each
        float4 *own = reinterpret_cast<float4 *>(unit_ex) + 2 * t;
        own[0] = make_float4(v[0], v[1], v[2], v[3]);
        own[1] = make_float4(v[4], v[5], v[6], v[7]);
        unit_barrier(1 + unit);
        float z[8];
#pragma unroll
        for (int g = 0; g < 8; ++g) z[g] = unit_ex[256 * g + t];
#pragma unroll
        for (int h = 1; h < 8; h <<= 1)
            if (256 * h < in.block) {
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    if ((g & h) == 0) {
                        const float a = z[g], b = z[g + h];
                        z[g] = a + b;
                        z[g + h] = a - b;
                    }
            }
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            const int c = unit * 2048 + 256 * g + t;
            if (c < n) xs[c] = __float2half_rn(z[g] * in.norm);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] *= in.norm;
    if (inside) store8_f16(xs + col, v);
}

// ---- batch 1-2: lane = row, products on the tensor cores -----------------------------------------------------------
// A granule is one 128-bit unit of two adjacent 32-row blocks; lane l owns rows 64*p + l and 64*p + 32 + l of block
// pair p, and a warp walks along its rows.
//
// Products.  One mma.sync m16n8k16 (fp16 in, fp32 accumulate) takes FOUR decoded pairs of a lane at once: pairs 2i and
// 2i+1 of the lane's row in block a (a0, a2) and of its row in block b (a1, a3).  Rows g and g+8 of the A tile are then
// a mix of the four lanes (g, 0..3), i.e. of four different rows of W -- which is harmless, because B separates them
// again: lane t's k slots meet the activations only in output column n = t (first activation row) and n = 4 + t
// (second), every other entry of B is zero.  D[g][4b + t] is the partial dot product of row 4g + t of block a with
// activation row b, D[g+8][4b + t] the same for block b.  The lane that supplies column n = g of B reads the
// activations when g % 4 == t (and g / 4 < BATCH) and holds zeros otherwise, so only four (eight) lanes of a warp take
// part in the shared-memory loads of x.  Against packed fp16 multiply-adds this issues a quarter of the multiply
// instructions per unit and row block, and there is no fp16 partial sum: the accumulation is fp32 throughout.
//
// Codes.  Each lane copies its own 16 bytes of a unit from global memory into a per-warp shared-memory ring with
// cp.async (the 32 rows of a unit are 512 contiguous bytes in the TILED layout: one fully coalesced request per warp),
// three granules ahead, and reads back only its own bytes: the per-thread group wait is the whole synchronisation --
// no barrier, no lane that issues copies on behalf of the others, no register or scoreboard held by a load in flight.
//
// MODE 0: activations copied from memory.  MODE 1: computed by every CTA from the previous layer's accumulator and the
// residual stream (rptc_gemv_glued).  MODE 2: the down projection of a gated MLP -- granules ordered by 256-column
// blocks first, each CTA makes the blocks of x it needs from the gate-up accumulator (rptc_gemv_swiglu).
// MODE 3 and 4 (gemv_alone): the first kernel of a layer's call.  Every CTA makes the activations from the layer's input for itself
// (3: scaled, 4: signs and Hadamard transform), and nothing has to be zeroed in front: the warps' sums of a CTA meet in shared memory, the
// CTAs' sums of a row are put down side by side, and the layer's output side adds them up (GemvSums) -- in a fixed order, so that equal
// calls give equal bits.  One launch and one trip through memory less than with a kernel for the input side.
template <int CODE, int K, int BATCH, int MODE>
__global__ void __launch_bounds__(kGemvThreads, 1) gemv_rows_kernel(const RowsParams<MODE> p) {
    constexpr int WPU = 128 / K;
    constexpr int PAIRS = WPU / 2;
    constexpr int NW2 = 2 * GroupShape<K>::kWords;
    constexpr uint32_t UPB = 256 / WPU;                       // units per 256-column block (MODE 2)
    constexpr bool ALONE = MODE >= 3, BANKED = MODE == 0 || MODE == 3;
    constexpr uint32_t kRunBytes = ALONE ? kGemvWarps * 64 * BATCH * 4 : 0;      // sums of the warps' first runs
    static_assert(BATCH == 1 || BATCH == 2, "eight output columns: four rows x two activation rows");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const uint32_t s0 = smem_addr(smem_raw);
    const uint32_t ring = s0 + kBarBytes + (uint32_t)warp * kStages * kStageBytes;
    uint32_t lut_tab, xs;
    if (CODE == RPTC_CODE_HASH) {
        lut_tab = kHashLutWindow;
        xs = kHashLutWindow + kHashLutBytes;
    } else {
        lut_tab = s0 + kBarBytes + kRingBytes + kRunBytes;
        xs = lut_tab + lut_bytes<CODE>(p.L, p.S);
    }
    if (CODE == RPTC_CODE_HASH && s0 + kBarBytes + kRingBytes + kRunBytes > kHashLutWindow) {
        if (threadIdx.x == 0) atomicExch(p.status, kStatusSmemPlan);
        return;
    }
    // the bank this CTA works on (one grid row per bank), and its number among the bank's CTAs
    const uint32_t bank = BANKED ? blockIdx.y : 0u, n_ctas = gridDim.x, cta = blockIdx.x;
    const __half *table = p.lut;
    if constexpr (BANKED) table += (int64_t)bank * p.lut_stride;
    const uint4 *codes = p.codes + (BANKED ? (int64_t)bank * p.m * p.n_units : 0);
    float *acc = p.acc + (BANKED ? (int64_t)bank * p.m : 0);
    // ---- prologue: nothing here depends on the kernels before this one ----
    // The table code's codebook (128 KiB at L = 16) is a plain image: one bulk copy, awaited in front of the main loop.
    LutPending lut_pending;
    auto fetch_table = [&]() {
        if (CODE == RPTC_CODE_LUT) {
            if (threadIdx.x == 0) {
                mbar_init(s0, 1);
                mbar_fence_init();
                mbar_expect_tx(s0, 2u << p.L);
                bulk_g2s(lut_tab, table, 2u << p.L, s0);
            }
            lut_pending.deferred = false;
        } else {
            lut_pending = lut_fill_begin<CODE>(lut_tab, table, p.L, p.S);
        }
    };
    if (!ALONE) fetch_table();
    const Lut<CODE> lut = lut_view<CODE>(lut_tab, p.L, p.S);
    if (!ALONE) pdl_allow_next_grid();

    const uint32_t n_rb = (uint32_t)(p.m >> 5), n_rbp = (n_rb + 1) >> 1;
    const uint32_t x_batch_stride = (uint32_t)p.seg_units * WPU * 2u;
    const int64_t rb_stride = (int64_t)p.n_units << 5;        // 128-bit units between row blocks of the TILED layout
    // this lane's column of B: activation row g / 4 for the lanes with g % 4 == t, zeros for the others
    const bool feeds_x = (g & 3) == t4 && (g >> 2) < BATCH;
    // where this lane's sums end up: D[g][2t], D[g][2t+1] are rows 4g + (2t & 3) + {0, 1}, activation row t / 2
    const int out_row = 4 * g + ((2 * t4) & 3), out_batch = t4 >> 1;
    bool waited_prior = ALONE;
    uint32_t *warp_first = reinterpret_cast<uint32_t *>(smem_raw + kWarpFirst);      // ALONE: the warps' first granules, the CTA's end

    for (int32_t useg0 = 0; useg0 < p.n_units; useg0 += p.seg_units) {
        const int32_t nu = MODE >= 2 ? p.n_units : min(p.seg_units, p.n_units - useg0);
        // Two-level even split of the T granules: contiguous ranges per CTA (sizes differ by at most one), then per warp
        // inside the CTA (again by at most one).  The warps that carry one granule more are thereby spread over all SMs
        // -- and over the four schedulers of each -- instead of filling the first CTAs of the grid.
        uint32_t cta_g0, cta_n, g0, count;
        if constexpr (ALONE) {
            // the same, counted in blocks of 32 rows: where their number is odd the last granules have one instead of two
            const uint32_t v0 = p.sums.begin(cta), v1 = p.sums.begin(cta + 1), dv = v1 - v0;
            cta_g0 = p.sums.granule_at(v0);
            cta_n = p.sums.granule_at(v1) - cta_g0;
            g0 = p.sums.granule_at(v0 + (uint32_t)((uint64_t)dv * warp / kGemvWarps));
            count = p.sums.granule_at(v0 + (uint32_t)((uint64_t)dv * (warp + 1) / kGemvWarps)) - g0;
            if (lane == 0) warp_first[warp] = g0;
            if (threadIdx.x == 0) warp_first[kGemvWarps] = cta_g0 + cta_n;
        } else {
            const uint32_t T = n_rbp * (uint32_t)nu;
            const uint32_t cta_per = T / n_ctas, cta_extra = T - cta_per * n_ctas;
            cta_g0 = cta * cta_per + min(cta, cta_extra);
            cta_n = cta_per + (cta < cta_extra ? 1u : 0u);
            const uint32_t w_per = cta_n / kGemvWarps, w_extra = cta_n - w_per * kGemvWarps;
            g0 = cta_g0 + (uint32_t)warp * w_per + min((uint32_t)warp, w_extra);
            count = w_per + ((uint32_t)warp < w_extra ? 1u : 0u);
        }

        // ---- granule order.  MODE 0/1: pairs of row blocks outermost, units along the row.  MODE 2: 256-column
        // blocks outermost, then pairs of row blocks, then the units of the block.
        struct Cursor {
            uint32_t rbp;       // pair of row blocks
            int32_t u;          // unit within the row (MODE 2) or within the segment (MODE 0/1)
            const uint4 *ptr;   // this lane's 16 bytes of block a
        };
        const uint32_t cell = n_rbp * UPB;
        auto cursor_at = [&](uint32_t gi) {
            Cursor c;
            if (MODE == 2) {
                const uint32_t cb = gi / cell, rem = gi - cb * cell;
                c.rbp = rem / UPB;
                c.u = (int32_t)(cb * UPB + (rem - c.rbp * UPB));
            } else {
                c.rbp = gi / (uint32_t)nu;
                c.u = (int32_t)(gi - c.rbp * (uint32_t)nu);
            }
            c.ptr = codes + (int64_t)(2 * c.rbp) * rb_stride + ((int64_t)(useg0 + c.u) << 5) + lane;
            return c;
        };
        auto advance = [&](Cursor &c) {      // to the next granule in this kernel's order
            ++c.u;
            c.ptr += 32;
            if (MODE == 2) {
                if (((uint32_t)c.u & (UPB - 1)) == 0) {      // end of the 256-column block: same block, next pair of row blocks
                    c.u -= (int32_t)UPB;
                    if (++c.rbp == n_rbp) {
                        c.rbp = 0;
                        c.u += (int32_t)UPB;
                    }
                    c.ptr = codes + (int64_t)(2 * c.rbp) * rb_stride + ((int64_t)c.u << 5) + lane;
                }
            } else if (c.u == nu) {
                c.u = 0;
                ++c.rbp;
                c.ptr = codes + (int64_t)(2 * c.rbp) * rb_stride + ((int64_t)useg0 << 5) + lane;
            }
        };
        Cursor fc = cursor_at(count ? g0 : 0u);      // fetch cursor
        Cursor cc = fc;                              // decode cursor
        // ---- the first PF granules and the 16 stream bits in front of the first one: all of it weights, so all of it
        // can be under way before anything that depends on the grid in front
        // Each lane copies its own 16 bytes of both row blocks into the warp's ring with asynchronous copies (tracked per
        // thread in groups, one group per granule: no register, scoreboard or barrier is tied up while they travel) and
        // reads back only what it copied itself, so the group wait is all the synchronisation there is.
        uint32_t fetched = 0;
        auto fetch = [&](uint32_t slot) {
            if (fetched < count) {
                const uint32_t dst = ring + slot * kStageBytes + 16u * lane;
                cp_async16(dst, fc.ptr);
                cp_async16(dst + kUnitBytes, 2 * fc.rbp + 1 < n_rb ? fc.ptr + rb_stride : fc.ptr);      // no second block: block a again, sums dropped
                advance(fc);
                ++fetched;
            }
            cp_async_commit();      // an empty group when nothing is left keeps the count of groups in flight constant
        };
        // Before the dependency wait only the first granule is requested: a lane's copies queue up in the load/store unit,
        // and a full ring of them ahead of the activation loads would delay those -- the critical ones -- by a trip to DRAM.
        // The rest of the ring follows as soon as the activation loads are on their way (`late_prologue`).
        if (MODE == 0) fetch(0);
        bool late_pending = true;
        auto late_prologue = [&]() {
            if (!late_pending) return;
            late_pending = false;
#pragma unroll
            for (int i = MODE == 0 ? 1 : 0; i < kStages; ++i) fetch(i);
            lut_fill_end<CODE>(lut_tab, lut_pending, p.S);      // the codebook loads were issued long ago
        };
        // The 16 stream bits in front of a run's first unit (the last word of the unit before it in the same rows, or the
        // shard's carry_in at a row start) are fetched one run ahead: those of the first two runs here, before the wait.
        auto load_history = [&](const Cursor &c, uint32_t &pa, uint32_t &pb) {
            const int64_t row_a = ((int64_t)c.rbp << 6) + lane;
            const bool has_b = 2 * c.rbp + 1 < n_rb;
            if (useg0 + c.u == 0) {
                pa = p.carry_in ? __ldg(p.carry_in + row_a) : 0u;
                pb = (p.carry_in && has_b) ? __ldg(p.carry_in + row_a + 32) : 0u;
            } else {
                const uint32_t *last = reinterpret_cast<const uint32_t *>(c.ptr - 32) + 3;
                pa = __ldg(last);
                pb = has_b ? __ldg(last + 4 * rb_stride) : 0u;
            }
        };
        auto run_length = [&](const Cursor &c) -> uint32_t {      // granules from c to the end of its run
            return MODE == 2 ? UPB - ((uint32_t)c.u & (UPB - 1)) : (uint32_t)(nu - c.u);
        };
        auto run_after = [&](const Cursor &c) {                    // first granule of the run after the one c lies in
            Cursor n = c;
            if (MODE == 2) {
                n.u = (int32_t)((uint32_t)c.u & ~(UPB - 1));
                if (++n.rbp == n_rbp) {
                    n.rbp = 0;
                    n.u += (int32_t)UPB;
                }
            } else {
                n.u = 0;
                ++n.rbp;
            }
            n.ptr = codes + (int64_t)(2 * n.rbp) * rb_stride + ((int64_t)(useg0 + n.u) << 5) + lane;
            return n;
        };
        // A call's first kernel reads nothing, and lets no other kernel start, before all work in front of the call is done.
        if (ALONE) {
            pdl_wait_prior_grids();
            pdl_allow_next_grid();
            fetch_table();
        }
        uint32_t prev_a = 0u, prev_b = 0u, next_prev_a = 0u, next_prev_b = 0u;
        uint32_t left_after_run = 0;          // granules of this warp behind the current run
        if (count) {
            load_history(cc, prev_a, prev_b);
            const uint32_t len = min(run_length(cc), count);
            left_after_run = count - len;
            if (left_after_run) load_history(run_after(cc), next_prev_a, next_prev_b);
        }

        // ---- activations -> shared memory ----
        if (!waited_prior) {
            pdl_wait_prior_grids();
            waited_prior = true;
        }
        if (useg0 > 0) __syncthreads();
        if constexpr (MODE == 2) {
            // column blocks of this CTA's warps together (its granules are consecutive)
            const uint32_t cb_first = cta_g0 / cell, cb_last = cta_n ? (cta_g0 + cta_n - 1) / cell : cb_first;
            if (p.clear) {
                float4 *z = reinterpret_cast<float4 *>(p.clear);
                for (int64_t i = (int64_t)blockIdx.x * kGemvThreads + threadIdx.x; 4 * i < p.clear_count; i += (int64_t)gridDim.x * kGemvThreads)
                    z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            __half *x_sm = reinterpret_cast<__half *>(smem_raw + (xs - s0));
            // (a CTA without granules would start behind the last block: the layer of a narrow model has fewer granules than there are SMs)
            for (uint32_t b = cb_first + warp; cta_n && b <= cb_last; b += kGemvWarps)
#pragma unroll 1
                for (int r = 0; r < BATCH; ++r)
                    swiglu_chunk(p.sw, r, (int64_t)b * 256 + 8 * lane, nullptr, false,
                                 x_sm + (size_t)r * (x_batch_stride >> 1) + (size_t)(b - cb_first) * 256 + 8 * lane, late_prologue);
            // x of unit u sits at xs + (u - cb_first * UPB) * 2 WPU: fold the offset into the base
            xs -= cb_first * UPB * (uint32_t)(WPU * 2);
        } else if constexpr (MODE == 1) {
            // one segment by construction (the host refuses wider rows)
            if (p.in.clear) {
                float4 *z = reinterpret_cast<float4 *>(p.in.clear);
                for (int64_t i = (int64_t)blockIdx.x * kGemvThreads + threadIdx.x; 4 * i < p.in.clear_count;
                     i += (int64_t)gridDim.x * kGemvThreads)
                    z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            // Exchange buffers of the glue, one per unit of 256 threads: behind x, or, beside a table that leaves no room there, in
            // the ring, which is then filled behind the glue.
            const bool on_ring = p.ex_on_ring;
            float *ex = reinterpret_cast<float *>(smem_raw + (on_ring ? kBarBytes : (xs - s0) + BATCH * x_batch_stride));
            FinishNormParams q;
            q.acc = const_cast<float *>(p.in.acc);
            q.ld_acc = p.in.ld_acc;
            q.signs_out = static_cast<const __half *>(p.in.signs_out);
            q.scale_out = p.in.scale_out;
            q.h = const_cast<__half *>(static_cast<const __half *>(p.in.h_in));
            q.h_out = static_cast<__half *>(p.in.h_out);
            q.ld_h = p.in.ld_h;
            q.w_norm = static_cast<const __half *>(p.in.w_norm);
            q.eps = p.in.eps;
            q.signs_in = static_cast<const __half *>(p.in.signs_in);
            q.transform_in = 1;
            q.out = reinterpret_cast<__half *>(smem_raw + (xs - s0));
            q.ld_out = x_batch_stride >> 1;
            q.n = (int32_t)p.n;
            q.block = 4096;
            const int unit = warp >> 3;
            float *unit_ex = ex + unit * kUnitFloats;
            float *red = reinterpret_cast<float *>(smem_raw + kGlueSums);      // 16 floats per row
            auto hook = [&]() {
                if (!on_ring) late_prologue();
            };
            if (p.n == 4096) {                       // a unit per row
                if (unit < BATCH)
                    finish_norm_unit(q, unit, 0, unit_ex, red + 16 * unit, 1 + unit, 3, false, blockIdx.x == 0, hook);
            } else {                                 // both units on one row after the other
#pragma unroll 1
                for (int b = 0; b < BATCH; ++b) {
                    finish_norm_unit(q, b, unit, unit_ex, red + 16 * b, 1 + unit, 3, false, blockIdx.x == 0, hook);
                    if (b + 1 < BATCH) __syncthreads();      // the buffers are read to the end before the next row
                }
            }
            if (on_ring) __syncthreads();
        } else if constexpr (MODE == 3) {
            scaled_input<BATCH>(p.in, (int)p.n, smem_raw + (xs - s0), x_batch_stride, reinterpret_cast<float2 *>(smem_raw + kGlueSums),
                                blockIdx.x + blockIdx.y == 0, late_prologue);
        } else if constexpr (MODE == 4) {
            const bool on_ring = p.ex_on_ring;
            auto hook = [&]() {
                if (!on_ring) late_prologue();
            };
            transformed_input(p.in, (int)p.n, reinterpret_cast<__half *>(smem_raw + (xs - s0)),
                              reinterpret_cast<float *>(smem_raw + (on_ring ? kBarBytes : (xs - s0) + BATCH * x_batch_stride)), hook);
            if (on_ring) __syncthreads();
        } else {
            const int64_t col0 = (int64_t)useg0 * WPU;
            const int pairs = nu * PAIRS;
            if (p.x_order == RPTC_XORDER_NATURAL && ((p.ld_x | col0) & 7) == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0) {
                const int vecs = pairs >> 2;
#pragma unroll
                for (int b = 0; b < BATCH; ++b) {
                    const uint4 *src = reinterpret_cast<const uint4 *>(p.x + (int64_t)b * p.ld_x + col0);
                    const uint32_t dst = xs + (uint32_t)b * x_batch_stride;
                    for (int i0 = threadIdx.x; i0 < vecs; i0 += 4 * kGemvThreads) {
                        uint4 v[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (i0 + k * kGemvThreads < vecs) v[k] = ld_ordered_u128(src + i0 + k * kGemvThreads);
                        late_prologue();                                                       // under the loads above
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (i0 + k * kGemvThreads < vecs)
                                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + 16u * (i0 + k * kGemvThreads)),
                                             "r"(v[k].x), "r"(v[k].y), "r"(v[k].z), "r"(v[k].w)
                                             : "memory");
                    }
                }
            } else {
                for (int i = threadIdx.x; i < BATCH * pairs; i += kGemvThreads) {
                    const int b = i / pairs, s = i - b * pairs;
                    int64_t src = (col0 >> 1) + s;
                    if (p.x_order == RPTC_XORDER_K2_LEGACY) src = k2_legacy_pair(src, p.n);
                    const uint32_t v = ld_ordered_u32(reinterpret_cast<const uint32_t *>(p.x + (int64_t)b * p.ld_x) + src);
                    asm volatile("st.shared.u32 [%0], %1;" ::"r"(xs + (uint32_t)b * x_batch_stride + 4u * s), "r"(v) : "memory");
                }
            }
        }
        late_prologue();      // threads that loaded nothing, other paths
        __syncthreads();
        if constexpr (MODE == 3) {
            if (blockIdx.x + blockIdx.y == 0 && threadIdx.x < BATCH) {
                const float2 *red = reinterpret_cast<const float2 *>(smem_raw + kGlueSums) + 16 * threadIdx.x;
                float2 tot = make_float2(0.f, 0.f);
                for (int w = 0; w < kGemvWarps; ++w) tot.x += red[w].x, tot.y += red[w].y;
                p.in.sums[threadIdx.x] = tot;
            }
        }
        if (CODE == RPTC_CODE_LUT && useg0 == 0 && !mbar_wait(s0, 0, p.status)) {
            cp_async_wait<0>();
            break;
        }

        // ---- main loop: one granule per step ----
        const uint32_t x_base = xs + (uint32_t)(g >> 2) * x_batch_stride;
        float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};      // two accumulator tiles: two shorter MMA chains
        // ALONE: a warp's range meets two runs at most; the sums of the first go behind the ring, those of the last over it
        auto put_run = [&](uint32_t at) {
            if (out_batch < BATCH) {
                const uint32_t dst = at + 4u * (uint32_t)(64 * out_batch + out_row);
                asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(dst), "f"(c0[0] + c1[0]), "f"(c0[1] + c1[1]) : "memory");
                asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(dst + 128u), "f"(c0[2] + c1[2]), "f"(c0[3] + c1[3]) : "memory");
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) c0[i] = c1[i] = 0.f;
        };
        const uint32_t first_runs = s0 + kBarBytes + kRingBytes;
        auto flush = [&](uint32_t rbp) {
            if (out_batch < BATCH) {
                const int64_t row_a = ((int64_t)rbp << 6) + out_row;
                const bool has_b = 2 * rbp + 1 < n_rb;
                float *dst = acc + (int64_t)out_batch * p.ld_acc + row_a;
                atomicAdd(dst, c0[0] + c1[0]);
                atomicAdd(dst + 1, c0[1] + c1[1]);
                if (has_b) {
                    atomicAdd(dst + 32, c0[2] + c1[2]);
                    atomicAdd(dst + 33, c0[3] + c1[3]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) c0[i] = c1[i] = 0.f;
        };
        // One granule: windows, 16 (K = 2) lookups per row block, 8 MMAs; then the bookkeeping of run ends.
        uint32_t slot = 0;
        auto granule = [&](uint32_t k, auto both) {
            constexpr bool kBoth = decltype(both)::value;
            cp_async_wait<kStages - 1>();      // all but the kStages - 1 youngest groups have landed: this granule is here
            const uint32_t stage = ring + slot * kStageBytes + 16u * lane;
            const uint4 va = lds128(stage), vb = kBoth ? lds128(stage + kUnitBytes) : va;
            uint32_t Ra[NW2], Rb[NW2];
            {
                const uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
                make_windows<K>(wa, prev_a, Ra);
                make_windows<K>(wb, prev_b, Rb);
            }
            prev_a = va.w;
            prev_b = vb.w;
            fetch(slot);                       // the words are in registers: the slot takes the granule kStages ahead
            if (++slot == kStages) slot = 0;
            const uint32_t xu = x_base + (uint32_t)cc.u * (uint32_t)(WPU * 2);
            uint4 xv = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int pi = 0; pi < PAIRS; pi += 4) {
                // only the four (eight) lanes whose column of B is in use read activations; the others hold zeros
                lds128_if(xv, xu + 4u * pi, feeds_x);
                uint32_t wa[4], wb[4] = {};
                decode_quad_bits<CODE, K>(Ra, lut, pi, wa);
                if constexpr (kBoth) decode_quad_bits<CODE, K>(Rb, lut, pi, wb);
                mma_16816(c0, wa[0], wb[0], wa[1], wb[1], xv.x, xv.y);
                mma_16816(c1, wa[2], wb[2], wa[3], wb[3], xv.z, xv.w);
            }
            // the next granule: same rows one unit on, or (end of the row / of the column block) other rows
            const uint32_t rbp_done = cc.rbp;
            const int32_t u_done = cc.u;
            advance(cc);
            if (cc.rbp != rbp_done || cc.u != u_done + 1) {
                if constexpr (!ALONE) flush(rbp_done);
                else if (k + 1 < count) put_run(first_runs + (uint32_t)warp * (64 * BATCH * 4));
                prev_a = next_prev_a;
                prev_b = next_prev_b;
                if (k + 1 < count) {
                    const uint32_t len = min(run_length(cc), left_after_run);
                    left_after_run -= len;
                    if (left_after_run) load_history(run_after(cc), next_prev_a, next_prev_b);
                }
            } else if (!ALONE && k + 1 == count) {
                flush(rbp_done);
            }
        };
#pragma unroll 1
        for (uint32_t k = 0; k < count; ++k) {
            // banks of rows may end with a block that stands alone: half the lookups
            if (ALONE && 2 * cc.rbp + 1 == n_rb) granule(k, std::false_type());
            else granule(k, std::true_type());
        }
        cp_async_wait<0>();                    // nothing of this segment's ring is in flight any more
        if constexpr (ALONE) {
            __syncwarp();
            put_run(ring);
            __syncthreads();
            // the CTA's sums: row by row, the warps in turn
            if (cta_n > 0) {
                const uint32_t p0 = cta_g0 / (uint32_t)nu, p1 = (cta_g0 + cta_n - 1) / (uint32_t)nu;
                for (uint32_t i = threadIdx.x; i < (p1 - p0 + 1) * (64 * BATCH); i += kGemvThreads) {
                    const uint32_t rbp = p0 + i / (64 * BATCH), b = i / 64 % BATCH, row = i % 64;
                    const uint32_t lo = rbp * (uint32_t)nu, hi = lo + (uint32_t)nu;
                    float sum = 0.f;
#pragma unroll 4
                    for (int w = 0; w < kGemvWarps; ++w) {
                        const uint32_t first = warp_first[w], end = warp_first[w + 1];
                        if (first == end || end <= lo || first >= hi) continue;
                        const uint32_t at = end <= hi ? s0 + kBarBytes + (uint32_t)w * kStages * kStageBytes : first_runs + (uint32_t)w * (64 * BATCH * 4);
                        sum += __uint_as_float(lds32(at + 4u * (64 * b + row)));
                    }
                    if (row < 32 || 2 * rbp + 1 < n_rb)
                        __stcg(acc + (int64_t)(cta - p.sums.cta_of(p.sums.weight(lo))) * p.sums.plane + b * p.ld_acc + 64 * rbp + row, sum);
                }
            }
        }
        if (MODE != 0) break;      // computed activations live in one segment
    }
    if (!waited_prior) pdl_wait_prior_grids();
}

template <int CODE, int K, int BATCH, int MODE>
static int launch_gemv_rows(const RowsParams<MODE> &p, size_t smem, cudaStream_t stream, dim3 grid = dim3(num_sms())) {
    static SmemOptIn opted;
    auto kern = gemv_rows_kernel<CODE, K, BATCH, MODE>;
    if (int e = allow_max_smem(kern, opted)) return e;
    return launch(kern, grid, dim3(kGemvThreads), smem, stream, p);
}

// The code and width of a format as template arguments.
template <typename F>
static int with_code(const rptc_format &f, F &&call) {
    switch (f.code) {
        case RPTC_CODE_LUT:
            if (f.K == 2) return call(std::integral_constant<int, RPTC_CODE_LUT>(), std::integral_constant<int, 2>());
            if (f.K == 4) return call(std::integral_constant<int, RPTC_CODE_LUT>(), std::integral_constant<int, 4>());
            break;
        case RPTC_CODE_HASH:
            if (f.K == 2) return call(std::integral_constant<int, RPTC_CODE_HASH>(), std::integral_constant<int, 2>());
            break;
        case RPTC_CODE_LITE:
            if (f.K == 2) return call(std::integral_constant<int, RPTC_CODE_LITE>(), std::integral_constant<int, 2>());
            if (f.K == 4) return call(std::integral_constant<int, RPTC_CODE_LITE>(), std::integral_constant<int, 4>());
            break;
    }
    return RPTC_ERR_UNSUPPORTED;
}

constexpr size_t kMaxSmem = 227 * 1024 - 1024;     // leave room for the 1 KiB the system may reserve
// Shared memory in front of the activations (must mirror the kernels').  HASH: addresses are absolute in the window.
static size_t fixed_smem(const rptc_format &f, size_t ring) {
    if (f.code == RPTC_CODE_HASH) return kHashLutWindow + kHashLutBytes;
    return kBarBytes + ring + (f.code == RPTC_CODE_LUT ? (size_t(2) << f.L) : (size_t(128) << f.S)) + 128;
}

}  // namespace rptc
