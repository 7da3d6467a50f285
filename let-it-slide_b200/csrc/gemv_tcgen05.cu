// Fused RPTC decode + matrix product for a few activation rows on the sm_100a tensor cores:
//   acc[t][row] += sum_c x[t][c] * W[row][c]        x: [tokens][n] fp16, up to 96 tokens, W decoded on the fly
//
// The decoded weights never touch shared memory: they are the A operand of tcgen05.mma and go from the registers they are
// decoded into straight to tensor memory (tcgen05.st; M = 128 weight rows in the 128 lanes), and the activations are the B
// operand (N = tokens rounded up to 16, K-major in shared memory, brought in by TMA).  What is left for shared memory are
// the table lookups, so that the cost of a step is that of its decode whatever the number of tokens -- the fused GEMM,
// which decodes into shared memory, pays 32 KiB of stores and 48 KiB of operand reads per 256 rows x 64 columns, and the
// mma.sync kernels repeat the decode for every eight activation rows.
//
// A tile is RB x 128 weight rows (RB = 1, 2, 4); a step is 64 columns of it.  The tiles' steps, laid end to end, are cut
// into equal ranges, one per CTA of a persistent grid; a CTA's range meets a tile in one segment.  Sixteen producer warps
// form four groups of four (a warp reaches the 32 tensor-memory lanes of its number modulo four): a group owns one of the
// RB row blocks and one of 4 / RB equal parts of a segment's steps, so that it walks along its rows and keeps the 16 bits
// of history.  A thread owns a row: its code bits arrive through a private ring of asynchronous copies, four steps ahead.
// Warp 16 loads the activations, taking the parts' steps in turn: position j of part 0, 1, ...  A part has a ring of stages of its
// own: a stage's full barrier tells only whether its phase is odd or even, so whoever waits on it has to have seen every phase
// before (one ring for all parts let a warp that skips the others' positions take a stage that still held an older one).  Each
// group has an MMA warp and an accumulator of its own: issuing a step (two waits, four MMAs, two commits) takes one thread about
// 600 clocks, as long as a group takes to decode it, so that one issuer for all four groups held the kernel to a
// quarter of the speed.  A segment's sums are added to the caller's fp32 accumulator with atomics.
// More activation rows (SHARED): a tile is RB x 128 weight rows (RB = 1, 2) x up to 256 (RB = 2: 192) tokens, and the groups that take parts
// of the same rows' steps share one accumulator, filled by one MMA warp.  A step of 256 x 192 takes the tensor core 768
// clocks and its decode about 430 issue slots per scheduler, so that decoding again for the next 192 tokens is free.
// ORDERED: segments' sums are put down side by side instead, and a second kernel adds them up in their order.
// Every wait on an mbarrier is bounded; a wait that runs out raises the device status word and the CTA drains and returns.
#include <algorithm>

#include "common.cuh"
#include "matmul.cuh"
#include "tc_ptx.cuh"

namespace rptc {

static_assert(4 * kFewOwnTokens <= 512 - 128 && 4 * 2 * 48 <= 512 - 128, "an accumulator per group beside the decoded weights in tensor memory");
constexpr int kFewWarps = 16, kFewTmaWarp = 16, kFewMmaWarp = 17, kFewThreads = 32 * (kFewMmaWarp + 4);
// Steps of a thread's code bits in flight.  Two beside a table, whose look-ups take a group more than two microseconds a step: at L = 16 the table
// leaves little room, and 16 KiB more hold two stages of 256 tokens.  With one stage fewer tokens fit into a tile, and every weight is looked up
// once per tile: layers of 4096 x 4096 in 32 banks, 256 tokens (two tiles of 128, now one) 32.1 -> 29.4 us, 384 tokens 47.2 -> 36.7; 4096 x 11008 in
// eight, 256 tokens 68.9 -> 50.1; up to 144 tokens the same time.  Smaller tables have the room for four as well, which is within 1 % either way (four /
// two: 4096 x 4096 in 32, L = 8, 256 tokens 26.5 / 26.2, 400 32.1 / 32.3; 11008 x 4096 in 8, L = 12, 320 74.5 / 75.1), so one form serves all.
constexpr int few_ahead(int code, bool shared) { return shared && code == RPTC_CODE_LUT ? 2 : 4; }
constexpr uint32_t kFewBars = 0x400, kFewHistory = 0x800, kFewCodes = 0x2800, kFewTop = 0x38800;
constexpr int kFewMaxXStages = 8;
constexpr int kFewACols = 32 * 4;                    // tensor-memory columns of the decoded weights: 64 fp16 per group and lane
constexpr int kFewTmemCols = 512;

// 64 registers per thread and no more shared memory than the plan needs: the CTAs of the small kernels in front of and behind
// this one in a decode step (norms, SwiGLU, attention) then fit on an SM beside one of its own, so that they are in place when the
// last sum is in, one to an SM, and this kernel fetches codes and table under them.  Without it they were packed onto the first SMs
// that came free, and those SMs started the next product 2 us late.
constexpr int kFewRegisterThreads = 1024;

struct FewParams {
    const uint4 *codes;
    const __half *lut;
    const uint32_t *carry_in;
    float *acc;                                      // ORDERED: the partial sums
    int64_t ld_acc;
    int64_t m, lut_stride;                           // rows of a bank, fp16 elements from one bank's table to the next
    int32_t n_steps, n_units;                        // 64-column steps, 128-bit units per row
    int32_t tokens, n_cols;                          // activation rows, rounded up to 16
    int32_t tiles, ctas;                             // per bank
    int32_t token_tiles;                             // tiles of the same weight rows, n_cols tokens each
    int32_t L, S;
    uint32_t lut_addr, x_addr;
    int32_t n_xstages;                               // per ring: one for each part, SHARED one
    bool shared;                                     // more than kFewOwnTokens activation rows (host side: SHARED)
    int32_t n_sums, max_steps;                       // accumulators per group (1 or 2), longest segment
    unsigned int *status;
};
// The tensor map behind the parameters starts on a 64-byte boundary: with one byte more it would move up, and a launch with more
// than 256 bytes of parameters starts later (22016 x 4096, 8 rows: the layer takes 24.5 instead of 24.0 us).
static_assert(sizeof(FewParams) <= 128, "parameters of gemv_few_kernel");

// A segment: the steps [s0, s1) of one tile, and the part of them that one group takes.
template <bool SHARED>
struct FewSegment {
    int32_t tile, s0, s1;                            // tile: of weight rows
    int32_t t0;                                      // first token
    uint32_t end;                                    // where the next segment starts in the CTA's range
    __device__ __forceinline__ FewSegment(uint32_t pos, uint32_t range_end, const FewParams &p) {
        tile = (int32_t)(pos / (uint32_t)p.n_steps);
        s0 = (int32_t)(pos - (uint32_t)tile * (uint32_t)p.n_steps);
        s1 = min(p.n_steps, s0 + min((int32_t)(range_end - pos), p.max_steps));
        end = pos + (uint32_t)(s1 - s0);
        t0 = 0;
        if (SHARED && p.token_tiles > 1) {
            const int32_t rows = tile / p.token_tiles;
            t0 = (tile - rows * p.token_tiles) * p.n_cols;
            tile = rows;
        }
    }
    template <int PARTS>
    __device__ __forceinline__ int32_t part_begin(int part) const { return s0 + (s1 - s0) * part / PARTS; }
};

template <int CODE, int K, int RB, bool SHARED, bool ORDERED>
__global__ void __launch_bounds__(kFewRegisterThreads, 1) gemv_few_kernel(const FewParams p, const __grid_constant__ CUtensorMap x_map) {
    constexpr int UPS = K / 2;                       // 128-bit units per step
    constexpr int PARTS = 4 / RB, RINGS = SHARED ? 1 : PARTS;
    constexpr int NW = 4 * UPS, kAhead = few_ahead(CODE, SHARED);
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (smem_addr(smem_raw) > kFewBars) {            // the dynamic area starts later than the plan says
        if (tid == 0) atomicExch(p.status, kStatusSmemPlan);
        return;
    }
    const uint32_t full_x = kFewBars, empty_x = full_x + 8 * kFewMaxXStages, full_a = empty_x + 8 * kFewMaxXStages, empty_a = full_a + 32,
                   sums = empty_a + 32, drained = sums + 8, table_bar = drained + 8, tmem_slot = table_bar + 8;
    const int bank = blockIdx.x / p.ctas;
    const uint32_t cta = blockIdx.x - bank * p.ctas;
    // this CTA's range of the bank's steps
    const uint32_t total = (uint32_t)(SHARED ? p.tiles * p.token_tiles : p.tiles) * (uint32_t)p.n_steps;
    const uint32_t per = total / p.ctas, extra = total - per * p.ctas;
    const uint32_t c0 = cta * per + min(cta, extra), c1 = c0 + per + (cta < extra ? 1u : 0u);

    // entries of the table that this thread spreads over the banks: asked for first, stored when its copies are under way
    LutPending entries;
    if (CODE != RPTC_CODE_LUT) entries = lut_fill_begin<CODE>(p.lut_addr, p.lut + (int64_t)bank * p.lut_stride, p.L, p.S);
    if (warp == kFewTmaWarp && lane == 0) tma_prefetch_map(&x_map);
    if (tid == 0) {
        for (int i = 0; i < kFewMaxXStages; ++i) mbar_init(full_x + 8 * i, 1), mbar_init(empty_x + 8 * i, RB);
        for (int g = 0; g < 4; ++g) mbar_init(full_a + 8 * g, 4), mbar_init(empty_a + 8 * g, 1);
        mbar_init(sums, SHARED ? RB : 4);
        mbar_init(drained, kFewWarps);
        mbar_init(table_bar, 1);
        mbar_fence_init();
        if (CODE == RPTC_CODE_LUT) {                 // a plain image of the codebook: one bulk copy
            mbar_expect_tx(table_bar, 2u << p.L);
            bulk_g2s(p.lut_addr, p.lut + (int64_t)bank * p.lut_stride, 2u << p.L, table_bar);
        }
    }
    if (warp == kFewMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "n"(kFewTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    bool ok = true;

    // ---- a producer's code bits: private ring of copies ----
    const int group = warp >> 2, block = group % RB, part = group / RB;
    const int32_t lane_row = block * 128 + (warp & 3) * 32 + lane;       // row inside the tile
    const uint32_t ring = kFewCodes + (uint32_t)warp * (kAhead * UPS * 512) + 16u * lane, hist = kFewHistory + 4u * tid;
    const uint4 *bank_codes = p.codes + (int64_t)bank * p.m * p.n_units;
    // rows past the bank's end decode its last block of 32 rows; their sums are not used
    auto row_in_bank = [&](int32_t tile) { return min((int64_t)tile * (RB * 128) + lane_row, p.m - 32 + lane); };
    uint32_t f_next = c0, slot = 0;                                       // fetch cursor: next segment; ring slot (of the fetch and of the decode)
    int32_t f_left = 0;                                                   // steps left of the part at hand
    const uint4 *f_src = nullptr;
    auto copy_step = [&]() {
#pragma unroll
        for (int q = 0; q < UPS; ++q) cp_async16(ring + (slot * UPS + q) * 512u, f_src + q * 32);
        f_src += UPS * 32;
        --f_left;
    };
    auto fetch_any = [&]() {                                              // one step into `slot`, if any is left
        bool fresh = false;
        int32_t s = 0;
        int64_t row = 0;
        while (f_left == 0 && f_next < c1) {                              // the next segment in which this part has steps
            const FewSegment<SHARED> g(f_next, c1, p);
            f_next = g.end;
            s = g.part_begin<PARTS>(part);
            f_left = g.part_begin<PARTS>(part + 1) - s;
            fresh = true;
            row = row_in_bank(g.tile);
            f_src = bank_codes + ((row >> 5) * (int64_t)p.n_units + (int64_t)s * UPS) * 32 + (row & 31);
        }
        if (f_left == 0) return;
        if (fresh) {
            const uint32_t dst = hist + 2048u * slot;
            if (s == 0) {
                const uint32_t v = p.carry_in ? __ldg(p.carry_in + row) : 0u;
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst), "r"(v) : "memory");
            } else {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(reinterpret_cast<const uint32_t *>(f_src - 32) + 3) : "memory");
            }
        }
        copy_step();
    };
    auto fetch = [&]() {
        if (f_left > 0) copy_step();
        else fetch_any();
        cp_async_commit();                                                // an empty group when nothing is left keeps the count constant
        slot = (slot + 1) % kAhead;
    };
    if (warp < kFewWarps) {
#pragma unroll 1
        for (int i = 0; i < kAhead; ++i) fetch();
    }
    // ---- table filled
    if (CODE != RPTC_CODE_LUT) lut_fill_end<CODE>(p.lut_addr, entries, p.S);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_allow_next_grid();
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
    tmem = __shfl_sync(0xFFFFFFFFu, tmem, 0);                             // the same in all lanes, and known to be
    const uint32_t a_cols = tmem + (kFewTmemCols - kFewACols);

    if (warp < kFewWarps) {
        // ================= decode =================
        const Lut<CODE> lut = lut_view<CODE>(p.lut_addr, p.L, p.S);
        if (CODE == RPTC_CODE_LUT) ok = mbar_wait(table_bar, 0, p.status);
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        uint32_t a_phase = 1u, seg_phase = 0u;
        for (uint32_t pos = c0; pos < c1 && ok;) {
            const FewSegment<SHARED> g(pos, c1, p);
            pos = g.end;
            const int64_t row = (int64_t)g.tile * (RB * 128) + lane_row;
            const int32_t len = g.part_begin<PARTS>(part + 1) - g.part_begin<PARTS>(part);
            uint32_t prevw = 0;
#pragma unroll 1
            for (int32_t i = 0; i < len && ok; ++i) {
                cp_async_wait<kAhead - 1>();      // this step's words have landed
                uint32_t R[2 * NW], out[16];
                if (i == 0) prevw = lds32(hist + 2048u * slot);
#pragma unroll
                for (int q = 0; q < UPS; ++q) {
                    const uint4 v = lds128(ring + (slot * UPS + q) * 512u);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        R[8 * q + 2 * k] = __funnelshift_l(w[k], prevw, 16);
                        R[8 * q + 2 * k + 1] = w[k];
                        prevw = w[k];
                    }
                }
                fetch();                             // the words are in registers: the slot takes the step kAhead further on
#pragma unroll
                for (int pi = 0; pi < 32; pi += 4) {
                    uint32_t four[4];
                    decode_quad_bits<CODE, K>(R, lut, pi, four);
                    out[pi & 15] = four[0], out[(pi & 15) + 1] = four[1], out[(pi & 15) + 2] = four[2], out[(pi & 15) + 3] = four[3];
                    if (pi == 12) {                  // the MMAs have read the group's last step
                        ok = mbar_wait(empty_a + 8 * group, a_phase, p.status);
                        a_phase ^= 1u;
                        tc_fence_after();
                    }
                    if ((pi & 15) == 12) tmem_store16_begin(a_cols + 32u * (uint32_t)group + (uint32_t)(pi & 16) + lanes, out);
                }
                tmem_store_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(full_a + 8 * group);
            }
            // ---- the segment's sums: this thread's row, eight tokens at a time, the parts in turn ----
            if (ok) ok = mbar_wait(sums, seg_phase, p.status);
            seg_phase ^= 1u;
            tc_fence_after();
            if (ok && row < p.m) {                   // of a whole warp: m is a multiple of 32
                float *dst = p.acc + (int64_t)bank * p.m + row;
                bool again = false;                  // ORDERED: the CTA's second segment of this tile, added to its first
                if (ORDERED) {
                    const uint32_t from = g.end - (uint32_t)(g.s1 - g.s0), tile_from = from - (uint32_t)g.s0;
                    const uint32_t first = tile_from < extra * (per + 1) ? tile_from / (per + 1) : extra + (tile_from - extra * (per + 1)) / per;
                    dst += (int64_t)(cta - first) * p.tokens * p.ld_acc;
                    again = from > max(tile_from, c0);
                }
                auto put = [&](float *to, float v) {
                    if (!ORDERED) atomicAdd(to, v);
                    else if (again) __stcg(to, __ldcg(to) + v);
                    else __stcg(to, v);
                };
                const int tokens = SHARED ? min(p.tokens - g.t0, p.n_cols) : p.tokens;
#pragma unroll 1
                for (int t0 = 8 * part; t0 < tokens; t0 += 8 * PARTS) {
                    float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
                    for (int a = 0; a < (SHARED ? 1 : PARTS); ++a) {
                        if (!SHARED && g.part_begin<PARTS>(a) == g.part_begin<PARTS>(a + 1)) continue;      // no step of this segment
                        uint32_t v[8], w[8] = {};
                        const uint32_t src = tmem + lanes + (uint32_t)((a * RB + block) * p.n_sums * p.n_cols + t0);
                        tmem_load8_begin(src, v);
                        if (p.n_sums == 2) tmem_load8_begin(src + (uint32_t)p.n_cols, w);
                        tmem_load_wait(v, w);
#pragma unroll
                        for (int e = 0; e < 8; ++e) sum[e] += __uint_as_float(v[e]) + __uint_as_float(w[e]);
                    }
                    float *to = dst + (int64_t)(g.t0 + t0) * p.ld_acc;
                    if (t0 + 8 <= tokens) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) put(to + (int64_t)e * p.ld_acc, sum[e]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 7; ++e)
                            if (t0 + e < tokens) put(to + (int64_t)e * p.ld_acc, sum[e]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(drained);
        }
        cp_async_wait<0>();
    } else if (warp == kFewTmaWarp) {
        // ================= activations =================
        pdl_wait_prior_grids();
        RingPos px[RINGS];
#pragma unroll
        for (int q = 0; q < RINGS; ++q) px[q] = {0, 1u};
        const uint32_t bytes = 128u * (uint32_t)p.n_cols;
        for (uint32_t pos = c0; pos < c1;) {
            const FewSegment<SHARED> g(pos, c1, p);
            pos = g.end;
            const int32_t rounds = (g.s1 - g.s0 + PARTS - 1) / PARTS;
            for (int32_t j = 0; j < rounds; ++j)
#pragma unroll
                for (int q = 0; q < PARTS; ++q) {
                    const int32_t s = g.part_begin<PARTS>(q) + j;
                    if (s >= g.part_begin<PARTS>(q + 1)) continue;
                    const int ring = SHARED ? 0 : q, stage = ring * p.n_xstages + px[ring].s;
                    const bool issues = elect_one();
                    ok = ok && mbar_wait(empty_x + 8 * stage, px[ring].phase, p.status);
                    if (issues && ok) {
                        mbar_expect_tx(full_x + 8 * stage, bytes);
                        tma_load_2d(p.x_addr + (uint32_t)stage * bytes, &x_map, s * 64, g.t0, full_x + 8 * stage);
                    }
                    px[ring].advance(p.n_xstages);
                }
        }
    } else if (!SHARED || warp < kFewMmaWarp + RB) {
        // ================= MMA issue for one accumulator (a group's, or SHARED a row block's): the whole warp waits, one lane issues =================
        const int grp = __shfl_sync(0xFFFFFFFFu, warp, 0) - kFewMmaWarp, mine = grp / RB, ring = SHARED ? 0 : mine * p.n_xstages;
        RingPos px = {0, 0u};
        uint32_t a_phase = 0u, seg = 0;              // a_phase: bit q for the group that takes part q
        const uint32_t bytes = 128u * (uint32_t)p.n_cols, idesc = instr_desc(p.n_cols);
        const uint32_t d_tmem = tmem + (uint32_t)(grp * p.n_sums * p.n_cols), a_first = a_cols + 32u * (uint32_t)grp;
        // the four MMAs of a step go round the accumulators
        const uint32_t d1 = p.n_sums == 2 ? (uint32_t)p.n_cols : 0u;
        for (uint32_t pos = c0; pos < c1; ++seg) {
            const FewSegment<SHARED> g(pos, c1, p);
            pos = g.end;
            if (seg > 0) ok = ok && mbar_wait(drained, (seg - 1) & 1u, p.status);      // the last segment's sums have been taken
            tc_fence_after();
            const int32_t rounds = (g.s1 - g.s0 + PARTS - 1) / PARTS;
            uint32_t accumulate = 0u;
            for (int32_t j = 0; j < rounds; ++j)
#pragma unroll
                for (int q = 0; q < PARTS; ++q) {
                    if (!(SHARED || q == mine) || g.part_begin<PARTS>(q) + j >= g.part_begin<PARTS>(q + 1)) continue;
                    const int from = SHARED ? q * RB : 0;                // + grp: the group whose step it is
                    const int stage = ring + px.s;
                    const bool issues = elect_one();
                    ok = ok && mbar_wait(full_x + 8 * stage, px.phase, p.status) && mbar_wait(full_a + 8 * (grp + from), SHARED ? (a_phase >> q) & 1u : a_phase, p.status);
                    a_phase ^= SHARED ? 1u << q : 1u;
                    tc_fence_after();
                    const uint32_t a_tmem = a_first + 32u * (uint32_t)from;
                    const uint64_t xb = umma_desc_sw128(p.x_addr + (uint32_t)stage * bytes);
                    if (issues && ok) {
                        // + 32 bytes of shared memory, + 8 columns of tensor memory per K = 16
                        tc_mma_f16_ta(d_tmem, a_tmem, xb, idesc, accumulate);
                        tc_mma_f16_ta(d_tmem + d1, a_tmem + 8u, xb + 2u, idesc, accumulate | (uint32_t)(p.n_sums == 1));
                        tc_mma_f16_ta(d_tmem, a_tmem + 16u, xb + 4u, idesc, 1u);
                        tc_mma_f16_ta(d_tmem + d1, a_tmem + 24u, xb + 6u, idesc, 1u);
                        tc_commit(empty_a + 8 * (grp + from));
                        tc_commit(empty_x + 8 * stage);
                    }
                    accumulate = 1u;
                    px.advance(p.n_xstages);
                }
            if (elect_one() && ok) {
                if (accumulate) tc_commit(sums);
                else mbar_arrive(sums);          // no step of this segment
            }
            __syncwarp();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kFewMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kFewTmemCols) : "memory");
    }
}

template <int CODE, int K, int RB, bool SHARED, bool ORDERED>
static int launch_few(const FewParams &p, const CUtensorMap &map, unsigned grid, cudaStream_t stream) {
    static SmemOptIn opted;
    auto kern = gemv_few_kernel<CODE, K, RB, SHARED, ORDERED>;
    static SmemOptIn preferred;
    if (int e = allow_max_smem(kern, opted)) return e;
    if (int e = prefer_shared_memory(kern, preferred)) return e;
    return launch(kern, dim3(grid), dim3(kFewThreads), p.x_addr + (uint32_t)(p.n_xstages * (SHARED ? 1 : 4 / RB)) * 128u * (uint32_t)p.n_cols, stream, p, map);
}

template <int CODE, int K, bool ORDERED>
static int launch_few_rb(int rb, const FewParams &p, const CUtensorMap &map, unsigned grid, cudaStream_t s) {
    if (p.shared) return rb == 1 ? launch_few<CODE, K, 1, true, ORDERED>(p, map, grid, s) : launch_few<CODE, K, 2, true, ORDERED>(p, map, grid, s);
    switch (rb) {
        case 1: return launch_few<CODE, K, 1, false, ORDERED>(p, map, grid, s);
        case 2: return launch_few<CODE, K, 2, false, ORDERED>(p, map, grid, s);
    }
    return launch_few<CODE, K, 4, false, ORDERED>(p, map, grid, s);
}
template <int CODE, int K>
static int launch_few_sums(int rb, const FewParams &p, const CUtensorMap &map, unsigned grid, cudaStream_t s, bool ordered) {
    return ordered ? launch_few_rb<CODE, K, true>(rb, p, map, grid, s) : launch_few_rb<CODE, K, false>(rb, p, map, grid, s);
}

// acc[token][column] = the partial sums of the column's tile, first segment first.  One thread per four columns of a token (of one tile and
// bank: m is a multiple of 32); where they lie is worked out under the product.  Bound: one or two trips to L2.
struct SumParams {
    const float *partial;                            // [CTA within the tile][token][ld]
    float *acc;
    int64_t ld;
    GemvSums sums;
    int32_t columns, m;
};
__global__ void __launch_bounds__(128) ordered_sum_kernel(const SumParams p) {
    constexpr int kAhead = 8;
    pdl_allow_next_grid();
    const int col = 4 * (blockIdx.x * 128 + threadIdx.x), token = blockIdx.y;
    const int slots = p.sums.count((uint32_t)(col % p.m), (uint32_t)token);
    const float *src = p.partial + (int64_t)token * p.ld + col;
    pdl_wait_prior_grids();
    if (col >= p.columns) return;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < slots; s += kAhead, src += kAhead * p.sums.plane) {
        float4 v[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i) v[i] = s + i < slots ? __ldcg(reinterpret_cast<const float4 *>(src + i * p.sums.plane)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < kAhead; ++i) sum.x += v[i].x, sum.y += v[i].y, sum.z += v[i].z, sum.w += v[i].w;
    }
    *reinterpret_cast<float4 *>(p.acc + (int64_t)token * p.ld + col) = sum;
}

// Row blocks per tile up to kFewOwnTokens activation rows.  With four of them a step of activations is loaded, waited for and handed back once per 512 rows;
// the relative times of a 128-row block are measured (28672 x 8192, 8 tokens: 31.0 us with four, 33.9 with two, 47.0
// with one).  A bank that is not a whole number of tiles leaves groups without rows: count the blocks that are walked.
static int few_row_blocks(int64_t m) {
    const int64_t blocks = (m + 127) / 128;
    int best = 4;
    double best_cost = 0;
    for (int rb = 4; rb >= 1; rb >>= 1) {
        const double cost = (double)((blocks + rb - 1) / rb * rb) * (rb == 4 ? 1.0 : rb == 2 ? 1.1 : 1.5);
        if (rb == 4 || cost < best_cost) best = rb, best_cost = cost;
    }
    return best;
}
// The same for ordered sums: every CTA that has a part of a tile puts down sums for all of its rows, so narrow tiles leave fewer of
// them to write and read.  Layers of 4096 x 4096, HASH, one, two and four row blocks: 16 rows 17.0, 19.7, 18.8 us, 64 rows 25.8, 31.3, 36.9;
// 22016 x 4096: 31.4, 29.2, 27.7 and 44.0, 43.3, 50.6.  The table code, bound by its look-ups, takes one: 11008 x 4096 in 32 banks, 16 rows
// 35.1, 40.0, 40.9.
static int ordered_row_blocks(int64_t m, int64_t tokens, int code) {
    return code == RPTC_CODE_LUT || m <= 32 * 128 || tokens > 48 ? 1 : 2;
}
// SHARED: microseconds of a 64-column step of a tile.  The decode (tables: bank conflicts, of 65,536 entries a little more), the tensor
// core (four clocks per token and pair of row blocks), or one thread's issue of the step.
static double shared_step_us(int rb, int n_cols, const rptc_format &f) {
    const double decode = rb * (f.code != RPTC_CODE_LUT ? 0.14 : f.L == 16 ? 0.60 : 0.55), mma = rb * n_cols * 2 / 1900.0, issue = 0.34;
    return decode > mma ? (decode > issue ? decode : issue) : (mma > issue ? mma : issue);
}

// Tile of `rb` row blocks, where the table and the activation ring go; false when they do not fit.
static bool few_plan(FewParams &p, const rptc_format &f, int64_t tokens, int rb, int64_t most_cols) {
    p.shared = tokens > kFewOwnTokens;
    const uint32_t codes_end = kFewCodes + kFewWarps * few_ahead(f.code, p.shared) * (f.K / 2) * 512;
    uint32_t free;
    if (f.code == RPTC_CODE_HASH) {
        p.lut_addr = kHashLutWindow;
        free = kHashLutWindow + kHashLutBytes;
    } else {
        p.lut_addr = codes_end;
        free = (codes_end + (f.code == RPTC_CODE_LUT ? (2u << f.L) : (128u << f.S)) + 1023u) & ~1023u;
    }
    if (free >= kFewTop) return false;
    p.x_addr = free;
    p.token_tiles = 1;
    if (p.shared) {      // three stages of activations (two under a table's slower look-ups), and the accumulators beside the decoded weights, bound the tile
        const int64_t fit = (kFewTop - free) / ((f.code == RPTC_CODE_LUT ? 2 : 3) * 128) / 16 * 16, most = rb == 1 ? most_cols : std::min<int64_t>(most_cols, 192), cols = fit < most ? fit : most;
        if (cols < 16) return false;
        p.token_tiles = (int32_t)((tokens + cols - 1) / cols);
    }
    p.n_cols = (int32_t)(((tokens + p.token_tiles - 1) / p.token_tiles + 15) / 16 * 16);
    int32_t stages = (int32_t)((kFewTop - free) / (128u * (uint32_t)p.n_cols));
    if (stages > kFewMaxXStages) stages = kFewMaxXStages;
    p.n_xstages = p.shared ? stages : stages / (4 / rb);      // four, two or one part: a ring each
    return stages >= 2 && p.n_xstages >= 1;
}
static int64_t few_tiles(int64_t m, int rb) { return (m + rb * 128 - 1) / (rb * 128); }
// The plan for `tokens` activation rows: row blocks per tile, or 0 where there is none.
static int few_choose(FewParams &p, const rptc_format &f, int64_t m, int64_t n, int64_t tokens, const Banks &banks, bool ordered) {
    // Beside a table of 128 KiB a weight is looked up once per tile of tokens, but a CTA of two steps looks up little, and tiles of more tokens leave
    // more CTAs to put down sums of a value: 1024 x 2048 in 8 banks, 192 and 256 tokens in two tiles 16.8 and 16.7 us, in one 17.5 and 17.6.
    const int64_t ctas = num_sms() / banks.banks > 0 ? num_sms() / banks.banks : 1;
    const int64_t most_cols = f.code == RPTC_CODE_LUT && f.L == 16 && few_tiles(m, 1) * (n / 64) < 3 * ctas ? 144 : 256;
    int rb = ordered ? ordered_row_blocks(m, tokens, f.code) : few_row_blocks(m);
    if (tokens > kFewOwnTokens) {
        FewParams one, two;
        const bool has_one = few_plan(one, f, tokens, 1, most_cols), has_two = few_plan(two, f, tokens, 2, most_cols);
        if (!has_one && !has_two) return 0;
        rb = !has_two || (has_one && few_tiles(m, 1) * one.token_tiles * shared_step_us(1, one.n_cols, f) <
                                         few_tiles(m, 2) * two.token_tiles * shared_step_us(2, two.n_cols, f))
                 ? 1
                 : 2;
    }
    // a table and tokens that leave no stage for each of the parts take tiles of more row blocks, which have fewer of them
    for (; rb <= 4; rb *= 2) {
        if (few_plan(p, f, tokens, rb, most_cols)) return rb;
        if (p.shared) break;
    }
    return 0;
}

// How the chosen plan's steps are cut into CTAs and segments.
static int few_ranges(FewParams &p, int rb, int64_t m, int64_t n, const Banks &banks) {
    p.n_steps = (int32_t)(n / 64);
    p.tiles = (int32_t)few_tiles(m, rb);
    const int64_t steps = (int64_t)p.tiles * p.token_tiles * p.n_steps;
    if (steps >= (int64_t(1) << 31)) return RPTC_ERR_TOO_LARGE;
    // one bank's table per CTA: the SMs are dealt out to the banks
    p.ctas = num_sms() / banks.banks > 0 ? num_sms() / banks.banks : 1;
    if (p.ctas > steps) p.ctas = (int32_t)steps;
    // The tensor core rounds its running sums towards zero, so the error of a sum grows with the number of MMAs behind it.
    // Two accumulators per group keep it where the mma.sync kernel had it (22016 x 4096, 16 rows: relative error 0.7e-6
    // against 1.3e-6 with one); where there is room for one only, a CTA's range goes into the result in two halves.
    // SHARED: no chain is longer than those of the fused GEMM, whose place it takes.
    p.n_sums = !p.shared && p.n_cols <= 48 ? 2 : 1;
    const int64_t range = (steps + p.ctas - 1) / p.ctas;
    p.max_steps = (int32_t)(p.n_sums == 2 || p.shared ? range : (range + 1) / 2);
    return RPTC_OK;
}

int64_t gemv_few_partials(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f) {
    FewParams p;
    const int rb = few_choose(p, f, m, n, tokens, banks, true);
    if (!rb || few_ranges(p, rb, m, n, banks)) return 0;
    // CTAs that meet in a tile: its first step may be a range's last, unless whole ranges make up a tile; those behind are full ones
    const int64_t steps = (int64_t)p.tiles * p.token_tiles * p.n_steps, per = steps / p.ctas;
    const bool whole = steps % p.ctas == 0 && p.n_steps % per == 0;
    const int64_t slots = whole ? p.n_steps / per : 1 + (p.n_steps - 1 + per - 1) / per;
    const bool two_each = p.max_steps < (steps + p.ctas - 1) / p.ctas;
    return slots * (two_each ? 2 : 1) <= 2 ? 0 : slots * tokens * banks.banks * m;
}

// Up to kFewOwnTokens activation rows always (a step costs its decode), beyond that where it is estimated to finish before
// the fused GEMM: a GEMM tile of 256 x 256 feeds the tensor core better and its result is fp16, but its decode goes through
// shared memory and half of its SMs are idle for a few hundred tokens.  Here a CTA has its equal share of the steps, takes
// its tiles' sums to memory (0.021 us per token and pair of row blocks, 1 us for every further tile of tokens), where more than two of them for a
// tile cost about 2.5 us and 0.3 per million values (they are added up in order by a second kernel), and the fp32 result is read behind.  The time
// around the steps is fitted to whole layers of both codes, and so is what a layer takes around the tiled product beyond that product's
// estimate: 1.7 us with a table, 4 with the others, whose layers have transforms on both sides that do not run under the start of this product.
// 2301 layers of 256 to 18176 rows and 512 to 14336 columns, 97 to 512 tokens, all codes, by both products: the choice costs 0.6 % over the better
// one; without the last three terms 1.2 (1280 x 3584 in 32 banks, L = 14, 158 tokens 17.0 here and 22.8; 4096 x 4096 in 32, L = 10, 128 21.8 and 24.6;
// 1024 x 3840 LITE, 512 25.2 and 28.7; on the other side 640 x 2752 in 8, L = 8, 500 23.0 and 18.7; 1024 x 2048 in 8, L = 10, 256 17.3 and 15.8).  Measured, whole layers, GEMM against this: 4096 x 11008 HASH, 128 tokens 44.5 and 31.6 us, 512
// 57.1 and 58.6; 22016 x 4096, 192 tokens 67.4 and 57.6; 1024 x 14336, 256 tokens 53.8 and 34; on the other side of the line 14336 x 1024, 512 tokens 38.7 and 51.7, 22016 x 4096, 2048 tokens 350 and 406.
static bool few_is_faster(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f) {
    FewParams p;
    const int rb = few_choose(p, f, m, n, tokens, banks, true);
    if (!rb || !p.shared) return rb != 0;
    const int64_t ctas = num_sms() / banks.banks > 0 ? num_sms() / banks.banks : 1, waves = (banks.banks * ctas + num_sms() - 1) / num_sms();
    const int64_t n_steps = n / 64, steps = (few_tiles(m, rb) * p.token_tiles * n_steps + ctas - 1) / ctas;
    const double drains = 1 + steps / n_steps;
    const int64_t partials = gemv_few_partials(m, n, tokens, banks, f);
    const double us = waves * ((f.code == RPTC_CODE_LUT ? 8.0 : 12.0) + steps * shared_step_us(rb, p.n_cols, f) + drains * 0.0105 * rb * p.n_cols) +
                      (double)banks.banks * m * tokens * 8 / 4.5e6 + (partials ? 2.5 + 0.3e-6 * (double)partials : 0.0) + (p.token_tiles - 1);
    const double gemm = gemm_us(m, n, tokens, banks, f);
    return gemm == 0 || us < gemm + (f.code == RPTC_CODE_LUT ? 1.7 : 4.0);
}

bool gemv_few_takes(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f, const void *x, int64_t ld_x) {
    if (f.layout != RPTC_LAYOUT_TILED || f.quirk != RPTC_QUIRK_NONE || (f.K != 2 && f.K != 4) || n % 64 || (reinterpret_cast<uintptr_t>(x) & 15) || ld_x % 8)
        return false;
    // a layer asks several times per call, and mostly the question of the call before
    struct Question {
        int64_t m, n, tokens;
        int32_t banks, code, K, L, S, device;      // device: its SMs, and the clusters that fit on them
        bool may_split;
        bool operator==(const Question &o) const {
            return m == o.m && n == o.n && tokens == o.tokens && banks == o.banks && code == o.code && K == o.K && L == o.L && S == o.S && device == o.device &&
                   may_split == o.may_split;
        }
    };
    static thread_local Question last = {};
    static thread_local bool last_answer = false;
    const Question q = {m, n, tokens, banks.banks, f.code, f.K, f.L, f.S, current_device(), banks.may_split};
    if (q == last) return last_answer;
    last_answer = few_is_faster(m, n, tokens, banks, f);
    last = q;
    return last_answer;
}

int gemv_few(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x, float *acc, int64_t ld_acc, int64_t m,
             int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f, cudaStream_t s, bool ordered, float *partial, GemvSums *parts) {
    FewParams p;
    const int rb = few_choose(p, f, m, n, tokens, banks, ordered);
    if (!rb) return RPTC_ERR_UNSUPPORTED;
    if (int e = few_ranges(p, rb, m, n, banks)) return e;
    CUtensorMap map;
    if (int e = encode_map(map, x, n, tokens, ld_x, p.n_cols)) return e;
    p.codes = static_cast<const uint4 *>(codes);
    p.lut = static_cast<const __half *>(lut);
    p.carry_in = carry_in;
    p.acc = acc;
    p.ld_acc = ld_acc;
    p.m = m;
    p.lut_stride = banks.lut_stride;
    p.n_units = (int32_t)(n * f.K / 128);
    p.tokens = (int32_t)tokens;
    if (partial) p.acc = partial;
    p.L = f.L;
    p.S = f.S;
    p.status = device_status_word();
    if (!p.status) return RPTC_ERR_CUDA;
    const unsigned grid = (unsigned)(banks.banks * p.ctas);
    const bool apart = partial != nullptr;
    int e = RPTC_ERR_UNSUPPORTED;
    switch (f.code) {
        case RPTC_CODE_LUT:
            e = f.K == 2 ? launch_few_sums<RPTC_CODE_LUT, 2>(rb, p, map, grid, s, apart) : launch_few_sums<RPTC_CODE_LUT, 4>(rb, p, map, grid, s, apart);
            break;
        case RPTC_CODE_HASH: e = launch_few_sums<RPTC_CODE_HASH, 2>(rb, p, map, grid, s, apart); break;
        case RPTC_CODE_LITE:
            e = f.K == 2 ? launch_few_sums<RPTC_CODE_LITE, 2>(rb, p, map, grid, s, apart) : launch_few_sums<RPTC_CODE_LITE, 4>(rb, p, map, grid, s, apart);
            break;
    }
    if (e || !apart) return e;
    const int64_t steps = (int64_t)p.tiles * p.token_tiles * p.n_steps;
    GemvSums sums = {};
    sums.plane = tokens * ld_acc;
    sums.per = (uint32_t)(steps / p.ctas);
    sums.extra = (uint32_t)(steps % p.ctas);
    sums.units = (uint32_t)p.n_steps;
    sums.tile_rows = rb * 128;
    sums.token_tiles = p.token_tiles;
    sums.n_cols = p.n_cols;
    if (parts) {
        *parts = sums;
        return RPTC_OK;
    }
    SumParams q;
    q.partial = partial;
    q.acc = acc;
    q.ld = ld_acc;
    q.sums = sums;
    q.columns = (int32_t)(banks.banks * m);
    q.m = (int32_t)m;
    return launch(ordered_sum_kernel, dim3((unsigned)((q.columns + 511) / 512), (unsigned)tokens), dim3(128), 0, s, q);
}

}  // namespace rptc
