// Fused RPTC decode + GEMM for prefill on the sm_100a tensor cores (tcgen05 + TMEM).
//
//   y[t][row] = sum_c x[t][c] * W[row][c]        x: [tokens][n] fp16,  W decoded on the fly
//
// One CTA owns an output tile of TOKENS (128 or 256) x NROWS (256, 128, or with 128 tokens 64 or 32) and walks the reduction dimension in steps of 64
// columns.  With both operands read from shared memory a 128 x 128 x 16 MMA needs 8 KiB of operand reads per 64
// tensor-core cycles -- exactly the 128 B/clk a SM's shared memory delivers -- so the wide tile (N = 256, 12 KiB per 128
// cycles) is what lets the tensor pipe run ahead of shared memory.  The two operands travel through separate
// shared-memory rings (activations: up to four stages of 16 KiB per 128 tokens; decoded weights: two or three stages of
// 128 bytes per tile row), each with its own full/empty barriers.  Warp roles:
//   warps 0-7  decode producers: thread r owns weight row r of the tile (256-row tiles: every thread takes every step;
//              narrower ones: two, four or eight groups of threads take the steps in turn).  Per step a thread takes its row's next
//              128 * K / 2 code bits with 128-bit loads (coalesced per 32-row block of the TILED layout), rebuilds the
//              shift-register windows with funnel shifts and looks the 64 weights up INTO REGISTERS; only then does it
//              wait for the stage, and writes its 128-byte row of the B operand straight into the 128-byte-swizzled
//              K-major layout the tensor core reads.  After the last step the same warps run the epilogue.
//   warp 8     one lane issues the 2-D TMA loads of the activation tile (128 tokens each), as far ahead as the
//              activation ring allows.
//   warp 9     owns the TMEM allocation; one lane (small tiles: an elected one of a warp that waits) issues tcgen05.mma (M = 128, N = NROWS,
//              K = 16, fp32 accumulators in TMEM, one or two token halves) and commits each stage back to its producer.
//              Small tiles were bound by this one thread: a step of a 128 x 128 tile 0.48 us with a lane that waits and
//              issues by itself (its operands are then not known to be uniform); 0.39 with one ring instead of two, one wait and one
//              commit less; 0.36 with the elected lane, where decoding and shared memory bound it.
//              Wide tiles, bound by the tensor core, lose by 31 more lanes that wait: prefill of 2048 tokens 29.25 -> 29.66 ms.
// Narrow tiles are for few tokens, whose wide tiles leave most SMs idle, where the order of additions must stay the wide ones'
// (invariant products, so the prompts of a model) or splitting gives less: 4096 x 11008, 22 tokens, 32 tiles of 128 rows 65.6 us, 64 of 64
// rows 45.5, 128 of 32 rows 43.5; of tables without bank conflicts 64 rows take a step in 0.24 us and 32 in 0.21.  Their ring
// is up to eight stages deep, and one copy of activations has the tokens that there are instead of 128.
// Where there are fewer tiles than SMs, a cluster of two or four CTAs shares a tile and each takes a part of the
// reduction; the partial sums meet in fp32 through distributed shared memory (`exchange_partials`) and each CTA stores
// its share of the tile's rows.
// Epilogue: tcgen05.ld 32 lanes x 32 columns at a time -> fp16 -> swizzled panels in shared memory -> TMA stores.
// The HASH code's table is kept in its packed form here (32 KiB instead of the GEMV kernels' 64 KiB), which is what
// makes room for the third activation stage beside two 32 KiB weight stages.
// Every wait on an mbarrier is bounded; a wait that runs out raises the device status word and the CTA drains and
// returns (TMEM is still released).
#include "common.cuh"
#include "matmul.cuh"
#include "tc_ptx.cuh"

namespace rptc {

constexpr int kStepCols = 64;          // one 128-byte swizzle atom of fp16
constexpr uint32_t kXHalfBytes = 128 * kStepCols * 2;          // 16 KiB: 128 tokens of a step
constexpr int kMaxGemmStages = 8;      // per ring
constexpr int kGemmThreads = 320;
constexpr int kProducerWarps = 8, kTmaWarp = 8, kMmaWarp = 9;

// The decoded-weight ring and the activation ring are separate: a TMA load takes about a microsecond to land and so
// wants the deeper ring, while a weight stage is refilled within a few hundred cycles of being handed back (the
// producers decode into registers ahead of time and only store once the stage is free).
struct GemmParams {
    const uint4 *codes;
    const __half *lut;
    const uint32_t *carry_in;
    __half *y;
    int64_t ld_y;
    int64_t m, n, tokens;             // m: rows of a bank
    int32_t n_units;                  // units per row
    int32_t L, S;
    int32_t tiles_per_bank, n_split;  // tiles that a bank's rows are rounded up to; CTAs that share a tile's reduction
    int64_t lut_stride;               // fp16 elements from one bank's table to the next
    int32_t n_xstages, n_wstages;
    uint32_t x_bytes;                 // of one copy of activations
    uint32_t bar_addr, lut_addr;      // offsets in the CTA's shared window
    uint32_t xa_addr[kMaxGemmStages], xb_addr[kMaxGemmStages];   // activation ring: two 128-token halves per stage
    uint32_t w_addr[kMaxGemmStages];                             // decoded-weight ring
    uint32_t epi_addr;                // epilogue: what it keeps in shared memory, laid over rings and table
    unsigned int *status;
};

// Barrier block (8 bytes each) at GemmParams::bar_addr.
struct GemmBars {
    uint32_t full_w, full_x, empty_w, empty_x, accum, tmem_slot, table;
};
__device__ __forceinline__ GemmBars gemm_bars(uint32_t base) {
    GemmBars b;
    b.full_w = base;
    b.full_x = base + 8 * kMaxGemmStages;
    b.empty_w = base + 16 * kMaxGemmStages;
    b.empty_x = base + 24 * kMaxGemmStages;
    b.accum = base + 32 * kMaxGemmStages;
    b.tmem_slot = b.accum + 8;
    b.table = b.accum + 16;                       // the lookup table, where the copy engine brings it in
    return b;
}

// Tiles of up to 128 x 128: activations and weights of a step share a stage and its barriers.  Wide ones have a ring each, the
// activations' a deeper one (22016 x 4096, 22 tokens in tiles of 256 rows: 45.7 us, 47.5 with one ring), and so have tiles of 128 rows beside a
// table of 128 KiB, which leaves three stages: 15616 x 1536, 100 tokens 25.5 us, 26.1 with one ring (32 KiB and K = 4, 128 tokens: 25.1 and 24.6).
constexpr bool one_ring(int rows, int halves, int table_bytes) { return halves == 1 && rows <= (table_bytes > 64 << 10 ? 64 : 128); }

// The HASH code is looked up in the packed table (128-byte rows) here: 32 KiB instead of 64 KiB leaves room for one more
// ring stage, and the extra shift per lookup is hidden behind the tensor pipe.
template <int CODE>
struct GemmDecode {
    static constexpr int kCode = CODE == RPTC_CODE_HASH ? kCodeHashPacked : CODE;
};

// `window` in the functions below: bits to OR onto every planned shared-memory offset (0 outside a cluster; inside one,
// the upper address bits that select this CTA's window in the cluster's).
// ---- decode producers ------------------------------------------------------------------------------------------------
// GROUPS groups of 256 / GROUPS threads take the steps in turn; thread r of a group owns row `row` of the bank whose codes
// start at `codes`.  A step's 64 weights are decoded into registers BEFORE the wait for the stage, so that between the
// tensor cores handing a stage back and its next contents being announced lie only eight 128-bit stores and a fence.
template <int CODE, int K, int GROUPS>
__device__ __forceinline__ bool produce_weights(const GemmParams &p, uint32_t window, const GemmBars &bars, const uint4 *codes, int64_t row,
                                                int step0, int n_steps) {
    constexpr int DC = GemmDecode<CODE>::kCode;
    constexpr int UPS = K / 2;                 // 128-bit units per 64-column step
    constexpr int kPairs = GroupShape<K>::kPairs;
    static_assert(UPS * kPairs == 32, "a step is 32 weight pairs per row");
    const int tid = threadIdx.x;
    const Lut<DC> lut = lut_view<DC>(p.lut_addr | window, p.L, p.S);
    const int group = tid / (256 / GROUPS);              // takes steps it = group, group + GROUPS, ...
    const int r = tid % (256 / GROUPS);                  // row of the tile
    // TILED layout: unit u of row -> ((row >> 5) * n_units + u) * 32 + (row & 31)
    const uint4 *src = codes + ((row >> 5) * (int64_t)p.n_units + (int64_t)step0 * UPS) * 32 + (row & 31);
    auto history = [&](int it) -> uint32_t {             // last word before step `it` of this CTA's part
        if (step0 + it == 0) return p.carry_in ? __ldg(p.carry_in + row) : 0u;
        return __ldg(reinterpret_cast<const uint32_t *>(src + ((int64_t)it * UPS - 1) * 32) + 3);
    };
    uint4 nxt[UPS];
    uint32_t nxt_prev = 0, carry = 0;                    // carry: last word of the previous step when this thread decoded it
    if (group < n_steps) {
#pragma unroll
        for (int q = 0; q < UPS; ++q) nxt[q] = ldg128_stream(src + ((int64_t)group * UPS + q) * 32);
        nxt_prev = history(group);
    }
    // the table, where the copy engine brings it in; the first step's codes are on their way
    if (CODE == RPTC_CODE_LUT && !mbar_wait(bars.table, 0, p.status)) return false;
    RingPos pos = {0, 1u};                               // waits on `empty` pass at once the first time round
    pos.advance_by(group, p.n_wstages);
    for (int it = group; it < n_steps; it += GROUPS) {
        uint4 cur[UPS];
#pragma unroll
        for (int q = 0; q < UPS; ++q) cur[q] = nxt[q];
        uint32_t prevw = (GROUPS > 1 || it == 0) ? nxt_prev : carry;
        if (it + GROUPS < n_steps) {
#pragma unroll
            for (int q = 0; q < UPS; ++q) nxt[q] = ldg128_stream(src + ((int64_t)(it + GROUPS) * UPS + q) * 32);
            nxt_prev = GROUPS > 1 ? history(it + GROUPS) : 0u;
        }
        uint32_t out[32];
#pragma unroll
        for (int q = 0; q < UPS; ++q) {
            const uint32_t w[4] = {cur[q].x, cur[q].y, cur[q].z, cur[q].w};
            decode_group<DC, K>(w, prevw, lut, [&](int pi, __half2 wp) { out[q * kPairs + pi] = half2_as_u32(wp); });
            prevw = cur[q].w;
        }
        carry = prevw;
        if (!mbar_wait(bars.empty_w + 8 * pos.s, pos.phase, p.status)) return false;      // the MMAs are done with the stage's old contents
        const uint32_t wrow = (p.w_addr[pos.s] | window) + (uint32_t)r * 128u;
#pragma unroll
        for (uint32_t chunk = 0; chunk < 8; ++chunk)         // 16-byte chunks of the row, 128-byte swizzle
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(wrow + 16u * (chunk ^ ((uint32_t)r & 7u))), "r"(out[4 * chunk]),
                         "r"(out[4 * chunk + 1]), "r"(out[4 * chunk + 2]), "r"(out[4 * chunk + 3])
                         : "memory");
        fence_proxy_async_smem();               // make the generic-proxy stores visible to the tensor cores' reads
        mbar_arrive(bars.full_w + 8 * pos.s);
        pos.advance_by(GROUPS, p.n_wstages);
    }
    return true;
}

// ---- activation loads (one thread) ----------------------------------------------------------------------------------
template <int HALVES, bool ONE_RING>
__device__ __forceinline__ bool load_activations(const GemmParams &p, uint32_t window, const GemmBars &bars, const CUtensorMap *x_map, int tok0,
                                                 int step0, int n_steps) {
    RingPos pos = {0, 1u};
    for (int it = 0; it < n_steps; ++it) {
        if (!mbar_wait((ONE_RING ? bars.empty_w : bars.empty_x) + 8 * pos.s, pos.phase, p.status)) return false;
        const uint32_t bar = (ONE_RING ? bars.full_w : bars.full_x) + 8 * pos.s;
        mbar_expect_tx(bar, HALVES * p.x_bytes);
        tma_load_2d(p.xa_addr[pos.s] | window, x_map, (step0 + it) * kStepCols, tok0, bar);
        if (HALVES == 2) tma_load_2d(p.xb_addr[pos.s] | window, x_map, (step0 + it) * kStepCols, tok0 + 128, bar);
        pos.advance(p.n_xstages);
    }
    return true;
}

// ---- epilogue (warps 0-7): TMEM -> fp16 -> shared memory -> global ----------------------------------------------------
// 32 accumulator columns from `col` on of this thread's token.  A warp may only touch TMEM lanes 32 * (warp % 4) ...
__device__ __forceinline__ void load_accumulators(uint32_t tmem_base, int col, uint32_t (&v)[32]) {
    const uint32_t taddr = tmem_base + ((uint32_t)((threadIdx.x >> 5 & 3) * 32) << 16) + (uint32_t)col;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Which accumulators an epilogue thread handles: with two token halves, warps 0-3 the first and 4-7 the second, every
// 32-column piece; with one half, both groups of four warps the same tokens and alternate pieces.
template <int HALVES>
struct EpilogueThread {
    int half, piece0, pieces_step;
    uint32_t token;               // inside the tile
    __device__ __forceinline__ EpilogueThread() {
        const int warp = threadIdx.x >> 5;
        half = HALVES == 2 ? warp >> 2 : 0;
        piece0 = HALVES == 2 ? 0 : warp >> 2;
        pieces_step = HALVES == 2 ? 1 : 2;
        token = (uint32_t)(half * 128 + (warp & 3) * 32 + (threadIdx.x & 31));
    }
};

// Split reduction: CTA j of the cluster is to finish columns [j C, (j + 1) C) of the tile, C = NROWS / n_split.  Every CTA
// sends each other one its partial sums of that one's columns, fp32, into the slot reserved for the sender: 16-byte
// pieces in the order [piece][token], so that a warp's stores are 512 contiguous bytes and the reader, the thread of the
// same number, finds them without bank conflicts.  Against partial sums through global memory (atomics, a cleared
// buffer and a pass that reads it) nothing leaves the chip.
template <int NROWS, int HALVES>
__device__ __forceinline__ void exchange_partials(const GemmParams &p, uint32_t window, uint32_t tmem_base, uint32_t rank) {
    const EpilogueThread<HALVES> me;
    const int C = NROWS / p.n_split;
    const uint32_t slot_bytes = (uint32_t)(HALVES * 128 * C * 4);
#pragma unroll 1
    for (uint32_t hop = 1; hop < (uint32_t)p.n_split; ++hop) {
        const uint32_t to = (rank + hop) % (uint32_t)p.n_split;
        const uint32_t slot = (p.epi_addr | window) + (uint32_t)(p.n_split - 1 - (int)hop) * slot_bytes + me.token * 16u;
        uint32_t dst;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(slot), "r"(to));
#pragma unroll 1
        for (int c = me.piece0; c < C / 32; c += me.pieces_step) {
            uint32_t v[32];
            load_accumulators(tmem_base, me.half * NROWS + (int)to * C + c * 32, v);
#pragma unroll
            for (int q = 0; q < 8; ++q)
                asm volatile("st.shared::cluster.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + (uint32_t)(c * 8 + q) * (HALVES * 128 * 16)),
                             "r"(v[4 * q]), "r"(v[4 * q + 1]), "r"(v[4 * q + 2]), "r"(v[4 * q + 3])
                             : "memory");
        }
    }
}

// `tok0` is this CTA's first token, `row0` its first output column (of C = NROWS / n_split).  The rings are free once the
// last MMA has been committed, so the tile is laid over them as panels of 128 tokens x 64 columns in the
// 128-byte-swizzled form a TMA store reads (a thread owns a token: its 16-byte chunks land in four-way-interleaved banks,
// the minimum for 512 bytes per warp), and one thread sends the panels off.  Against per-thread global stores (32 different
// lines per instruction) this cut the epilogue from 8.3 us to the time the tile takes to leave through the copy engine.
template <int NROWS, int HALVES>
__device__ __forceinline__ void drain_accumulators(const GemmParams &p, uint32_t window, uint32_t tmem_base, uint32_t rank, int tok0, int64_t row0,
                                                   int64_t col_end, const CUtensorMap *y_map, bool ok) {
    const EpilogueThread<HALVES> me;
    const int C = NROWS / p.n_split;
    const uint32_t slot_bytes = (uint32_t)(HALVES * 128 * C * 4);
    const uint32_t slots = p.epi_addr | window, panels = slots + (uint32_t)(p.n_split - 1) * slot_bytes;
    const uint32_t t = me.token & 127u;                       // row of the panel
    // All eight warps come here, also one whose wait ran out (`ok` false: it skips its part, and nothing is sent).
#pragma unroll 1
    for (int c = me.piece0; ok && c < C / 32; c += me.pieces_step) {
        uint32_t v[32];
        load_accumulators(tmem_base, me.half * NROWS + (int)rank * C + c * 32, v);
#pragma unroll 1
        for (int j = 0; j < p.n_split - 1; ++j) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint4 o = lds128(slots + (uint32_t)j * slot_bytes + (uint32_t)(c * 8 + q) * (HALVES * 128 * 16) + me.token * 16u);
                v[4 * q] = __float_as_uint(__uint_as_float(v[4 * q]) + __uint_as_float(o.x));
                v[4 * q + 1] = __float_as_uint(__uint_as_float(v[4 * q + 1]) + __uint_as_float(o.y));
                v[4 * q + 2] = __float_as_uint(__uint_as_float(v[4 * q + 2]) + __uint_as_float(o.z));
                v[4 * q + 3] = __float_as_uint(__uint_as_float(v[4 * q + 3]) + __uint_as_float(o.w));
            }
        }
        // tiles of 32 rows: a panel of 32 columns, 64-byte rows with the 64-byte swizzle
        const uint32_t prow = NROWS == 32 ? panels + t * 64u : panels + (uint32_t)(me.half * (C / 64) + (c >> 1)) * kXHalfBytes + t * 128u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                o[e] = half2_as_u32(__floats2half2_rn(__uint_as_float(v[8 * j + 2 * e]), __uint_as_float(v[8 * j + 2 * e + 1])));
            const uint32_t chunk = (uint32_t)((c & 1) * 4 + j) ^ (NROWS == 32 ? t >> 1 & 3u : t & 7u);
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(prow + 16u * chunk), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3])
                         : "memory");
        }
    }
    fence_proxy_async_smem();                                 // the stores above are read by the copy engine
    uint32_t all_ok;                                          // barrier of the eight epilogue warps, AND of their `ok`
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "barrier.cta.red.and.pred p, 1, 256, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(all_ok)
        : "r"((uint32_t)ok)
        : "memory");
    if (threadIdx.x == 0 && all_ok) {
#pragma unroll 1
        for (int hh = 0; hh < HALVES; ++hh) {
            if ((int64_t)tok0 + hh * 128 >= p.tokens) break;  // a half with no tokens at all (rows beyond `tokens` inside a half are clipped)
#pragma unroll 1
            for (int q = 0; q < (NROWS == 32 ? 1 : C / 64) && row0 + q * 64 < col_end; ++q)
                tma_store_2d(y_map, (int)row0 + q * 64, tok0 + hh * 128, panels + (uint32_t)(hh * (C / 64) + q) * kXHalfBytes);
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");     // the tile has left before the CTA (and its shared memory) goes
    }
}

// Of the stages in use: one thread does it, in front of everything.
__device__ __forceinline__ void init_ring_barriers(const GemmBars &bars, int x_stages, int w_stages, uint32_t w_arrivals) {
    for (int s = 0; s < w_stages; ++s) {
        mbar_init(bars.full_w + 8 * s, w_arrivals);
        mbar_init(bars.empty_w + 8 * s, 1);
    }
    for (int s = 0; s < x_stages; ++s) {
        mbar_init(bars.full_x + 8 * s, 1);
        mbar_init(bars.empty_x + 8 * s, 1);
    }
    mbar_init(bars.accum, 1);
    mbar_init(bars.table, 1);
    mbar_fence_init();
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int CODE, int K, int NROWS, int HALVES, bool ONE_RING>
__global__ void __launch_bounds__(kGemmThreads, 1)
    gemm_kernel(const GemmParams p, const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap y_map) {
    constexpr int DC = GemmDecode<CODE>::kCode;
    constexpr uint32_t kTmemCols = HALVES * NROWS;       // NROWS fp32 columns per 128 tokens
    constexpr uint32_t kInstrDesc = instr_desc(NROWS);
    constexpr int kGroups = 256 / NROWS;                 // producer groups taking the steps in turn
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // In a cluster every CTA's shared-memory window sits at its own place in the cluster's window: shared addresses of
    // this CTA's memory carry the CTA's rank in their upper bits (rank 1 starts at 0x01000000).  The host's plan holds
    // offsets inside a CTA's window, so those bits are ORed onto every planned address that a load, store, copy or
    // barrier instruction gets; the tensor-core descriptors keep only the offset bits.
    const uint32_t s_raw = smem_addr(smem_raw);
    const uint32_t s0 = s_raw & 0x00FFFFFFu, window = s_raw & 0xFF000000u;
    if (s0 > p.bar_addr) {                     // the dynamic area starts later than the host planned for (in every CTA alike)
        if (tid == 0) atomicExch(p.status, kStatusSmemPlan);
        return;
    }
    const GemmBars bars = gemm_bars(p.bar_addr | window);
    // this CTA's part of the reduction: step0 .. step0 + n_steps
    const uint32_t rank = blockIdx.z;          // also the CTA's rank in its cluster
    const int all_steps = (int)(p.n / kStepCols);
    const int step0 = (int)((int64_t)all_steps * rank / p.n_split), n_steps = (int)((int64_t)all_steps * (rank + 1) / p.n_split) - step0;
    const int tok0 = blockIdx.y * (HALVES * 128);
    // rows of the bank, and where the bank's codes and table are
    const int bank = blockIdx.x / p.tiles_per_bank;
    const int64_t tile_row = (int64_t)(blockIdx.x - bank * p.tiles_per_bank) * NROWS;
    const uint4 *codes = p.codes + (int64_t)bank * p.m * p.n_units;

    if (tid == 0) init_ring_barriers(bars, ONE_RING ? 0 : p.n_xstages, p.n_wstages, NROWS + (ONE_RING ? 1 : 0));
    if (warp == kMmaWarp) {                     // TMEM: fp32 accumulators of NROWS columns per 128 tokens
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bars.tmem_slot), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const __half *table = p.lut + (int64_t)bank * p.lut_stride;
    if (CODE == RPTC_CODE_LUT) {
        // a plain image of the codebook (128 KiB at L = 16): one bulk copy, awaited by the producers
        if (tid == 0) {
            mbar_expect_tx(bars.table, 2u << p.L);
            bulk_g2s(p.lut_addr | window, table, 2u << p.L, bars.table);
        }
    } else {
        lut_fill<DC>(p.lut_addr | window, table, p.L, p.S);      // only the producer warps read the table, but everyone helps to fill it
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_allow_next_grid();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(bars.tmem_slot));
    bool ok = true;

    if (warp < kProducerWarps) {
        // rows beyond the bank's end decode its last row; their columns of the output hold no result
        const int64_t row = tile_row + tid % NROWS;
        ok = produce_weights<CODE, K, kGroups>(p, window, bars, codes, row < p.m ? row : p.m - 1, step0, n_steps);
    } else if (warp == kTmaWarp) {
        pdl_wait_prior_grids();
        if (lane == 0) load_activations<HALVES, ONE_RING>(p, window, bars, &x_map, tok0, step0, n_steps);
    } else if (ONE_RING || lane == 0) {
        // ================= MMA issue =================
        RingPos px = {0, 0u}, pw = {0, 0u};
        for (int it = 0; it < n_steps; ++it) {
            const bool issues = !ONE_RING || elect_one();
            if (ONE_RING) {
                ok = ok && mbar_wait(bars.full_w + 8 * pw.s, pw.phase, p.status);
            } else {
                ok = mbar_wait(bars.full_x + 8 * px.s, px.phase, p.status) && mbar_wait(bars.full_w + 8 * pw.s, pw.phase, p.status);
                if (!ok) break;
            }
            tc_fence_after();
            const uint64_t xa = umma_desc_sw128(p.xa_addr[px.s]), xb = umma_desc_sw128(p.xb_addr[px.s]), wd = umma_desc_sw128(p.w_addr[pw.s]);
            if (!ONE_RING && CODE == RPTC_CODE_LUT) {
                // Descriptors made MMA by MMA: look-ups bind these tiles, and with the additions below they take 1 to 2 % more time (4096 x 11008, L = 16,
                // 900 tokens 165.7 and 168.2 us); the other codes' 0.6 % less (HASH, 22016 x 4096, 2048 tokens 271.6 and 270.1).
#pragma unroll
                for (uint32_t k = 0; k < kStepCols / 16; ++k) {
                    const uint64_t w_desc = umma_desc_sw128(p.w_addr[pw.s] + 32u * k);
                    tc_mma_f16(tmem_base, umma_desc_sw128(p.xa_addr[px.s] + 32u * k), w_desc, kInstrDesc, (it | k) != 0);
                    if (HALVES == 2) tc_mma_f16(tmem_base + (uint32_t)NROWS, umma_desc_sw128(p.xb_addr[px.s] + 32u * k), w_desc, kInstrDesc, (it | k) != 0);
                }
                tc_commit(bars.empty_x + 8 * px.s);
                tc_commit(bars.empty_w + 8 * pw.s);
            } else if (issues && ok) {
#pragma unroll
                for (uint32_t k = 0; k < kStepCols / 16; ++k) {           // + 32 bytes per K = 16
                    tc_mma_f16(tmem_base, xa + 2u * k, wd + 2u * k, kInstrDesc, (it | k) != 0);
                    if (HALVES == 2) tc_mma_f16(tmem_base + (uint32_t)NROWS, xb + 2u * k, wd + 2u * k, kInstrDesc, (it | k) != 0);
                }
                if (!ONE_RING) tc_commit(bars.empty_x + 8 * px.s);      // each arrives when the MMAs above have read the stage
                tc_commit(bars.empty_w + 8 * pw.s);
            }
            if (ONE_RING) __syncwarp();
            px.advance(p.n_xstages);
            pw.advance(p.n_wstages);
        }
        if ((!ONE_RING || elect_one()) && ok) tc_commit(bars.accum);   // arrives when every MMA has written its accumulator
    }
    __syncwarp();

    if (warp < kProducerWarps) {
        if (ok) ok = mbar_wait(bars.accum, 0, p.status);
        tc_fence_after();
    }
    if (p.n_split > 1) {
        cluster_sync_all();                         // every CTA of the cluster is done with its rings: partial sums may land on them
        if (warp < kProducerWarps && ok) exchange_partials<NROWS, HALVES>(p, window, tmem_base, rank);
        __syncwarp();
        cluster_sync_all();                         // ... and have landed
    }
    if (warp < kProducerWarps)
        drain_accumulators<NROWS, HALVES>(p, window, tmem_base, rank, tok0, (int64_t)blockIdx.x * NROWS + rank * (NROWS / p.n_split),
                                          (int64_t)bank * p.tiles_per_bank * NROWS + p.m, &y_map, ok);
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

// ---- host -----------------------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 encode_tiled_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    }
    return fn;
}

int encode_map(CUtensorMap &map, const void *base, int64_t cols, int64_t rows, int64_t ld, int box_rows, int box_cols) {
    auto encode = encode_tiled_fn();
    if (!encode) return RPTC_ERR_CUDA;
    const cuuint64_t dim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t stride[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, estride[2] = {1, 1};
    const CUresult r = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dim, stride, box, estride,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS) return RPTC_OK;
    g_last_cuda_error = (int)r;
    return RPTC_ERR_CUDA;
}

// How a product is cut into CTAs.
struct GemmShape {
    int rows, halves, split;      // weight rows and 128-token halves of a tile, CTAs that share a tile's reduction
};

template <int CODE, int K, int NROWS, int HALVES, bool ONE_RING>
static int launch_gemm(const GemmParams &p, const CUtensorMap &map, const CUtensorMap &ymap, size_t smem, dim3 grid, cudaStream_t stream) {
    static SmemOptIn opted;
    auto kern = gemm_kernel<CODE, K, NROWS, HALVES, ONE_RING>;
    if (int e = allow_max_smem(kern, opted)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (grid.z > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = grid.z;
    }
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    RPTC_CUDA(cudaLaunchKernelEx(&cfg, kern, p, map, ymap));
    return RPTC_OK;
}

template <int CODE, int K>
static int launch_gemm_shape(const GemmShape &g, const GemmParams &p, const CUtensorMap &map, const CUtensorMap &ymap, size_t smem, dim3 grid,
                             cudaStream_t stream) {
    if (g.rows == 256)
        return g.halves == 2 ? launch_gemm<CODE, K, 256, 2, false>(p, map, ymap, smem, grid, stream) : launch_gemm<CODE, K, 256, 1, false>(p, map, ymap, smem, grid, stream);
    if (g.rows == 64) return launch_gemm<CODE, K, 64, 1, true>(p, map, ymap, smem, grid, stream);
    if (g.rows == 32) return launch_gemm<CODE, K, 32, 1, true>(p, map, ymap, smem, grid, stream);
    if (g.halves == 2) return launch_gemm<CODE, K, 128, 2, false>(p, map, ymap, smem, grid, stream);
    if constexpr (CODE == RPTC_CODE_LUT)
        if (!one_ring(128, 1, 2 << p.L)) return launch_gemm<CODE, K, 128, 1, false>(p, map, ymap, smem, grid, stream);
    return launch_gemm<CODE, K, 128, 1, true>(p, map, ymap, smem, grid, stream);
}

// Shared-window plan (offsets in the CTA's window; the dynamic area is expected to start at or below 0x400).  The packed
// HASH table sits on its 32 KiB boundary; ring stages go first-fit into the space around the table: first two stages of
// each ring, then alternately one more of each (the activation ring, the slower to refill, first).  The epilogue lays
// its slots and panels over everything but the barriers.  False when the tile does not fit beside this table.
constexpr uint32_t kGemmTop = 0x38800;       // 226 KiB: the last byte any plan may touch (dynamic limit is 227 KiB)
static bool plan_gemm(GemmParams &p, const GemmShape &g, const rptc_format &f) {
    const uint32_t kHashAt = 0x8000;
    uint32_t free_lo[2], free_hi[2];
    int n_free;
    p.bar_addr = 0x400;
    p.epi_addr = 0x800;
    if (f.code == RPTC_CODE_HASH) {
        p.lut_addr = kHashAt;
        free_lo[0] = 0x800, free_hi[0] = kHashAt;
        free_lo[1] = kHashAt + kHashPackedLutBytes, free_hi[1] = kGemmTop;
        n_free = 2;
    } else {
        p.lut_addr = 0x800;
        const uint32_t lb = f.code == RPTC_CODE_LUT ? (2u << f.L) : (128u << f.S);
        free_lo[0] = (0x800 + lb + 1023u) & ~1023u, free_hi[0] = kGemmTop;
        n_free = 1;
    }
    auto take = [&](uint32_t bytes) -> uint32_t {
        for (int i = 0; i < n_free; ++i)
            if (free_lo[i] + bytes <= free_hi[i]) {
                const uint32_t a = free_lo[i];
                free_lo[i] += bytes;
                return a;
            }
        return 0;
    };
    int xs = 0, ws = 0;
    const bool one = one_ring(g.rows, g.halves, f.code == RPTC_CODE_LUT ? 2 << f.L : 0);
    const int most_x = g.rows < 128 ? kMaxGemmStages : 4, most_w = one ? most_x : 3;
    auto add_x = [&]() -> bool {
        if (xs == most_x) return false;
        const uint32_t save0 = free_lo[0], save1 = free_lo[1];
        const uint32_t xa = take(kXHalfBytes), xb = g.halves == 2 ? take(kXHalfBytes) : xa;
        if (!xa || !xb) {
            free_lo[0] = save0, free_lo[1] = save1;
            return false;
        }
        p.xa_addr[xs] = xa, p.xb_addr[xs] = xb;
        ++xs;
        return true;
    };
    auto add_w = [&]() -> bool {
        if (ws == most_w) return false;
        const uint32_t w = take((uint32_t)g.rows * 128u);
        if (!w) return false;
        p.w_addr[ws++] = w;
        return true;
    };
    add_w(), add_w(), add_x(), add_x();
    if (xs < 2 || ws < 2) return false;
    for (bool grew = true; grew;) {
        grew = add_x();
        grew = add_w() || grew;
    }
    for (int s = xs; s < kMaxGemmStages; ++s) p.xa_addr[s] = p.xb_addr[s] = 0;
    for (int s = ws; s < kMaxGemmStages; ++s) p.w_addr[s] = 0;
    p.n_xstages = one && ws < xs ? ws : xs;
    p.n_wstages = one && xs < ws ? xs : ws;
    // A group must find no stage two uses behind: a wait tells the uses' parity only.
    return p.n_wstages >= 256 / g.rows;
}

// Microseconds of one 64-column step of a tile, and of a CTA around its steps (start, table, epilogue, and where a tile is
// shared the exchange of partial sums).  Measured on 4096 rows x 4096 and 11008 columns; what matters is their ratio.
static double step_us(int rows, int halves, int code) {
    if (rows == 64) return code == RPTC_CODE_LUT ? 0.42 : 0.235;
    if (rows == 32) return code == RPTC_CODE_LUT ? 0.25 : 0.21;
    if (code == RPTC_CODE_LUT) return rows == 256 ? 1.43 : halves == 2 ? 0.92 : 0.77;
    if (halves == 2) return rows == 256 ? 0.61 : 0.56;
    return rows == 256 ? 0.58 : 0.36;
}
static double around_us(int rows, int halves, int split) {
    const double tile = rows / 256.0 * halves;               // in wide tiles of one half
    return 5.0 + 1.5 * tile + (split > 1 ? 1.5 + 1.3 * tile * (split == 4 ? 2.0 : 1.0) : 0.0);
}

// Clusters of `split` CTAs that fit the device at once (one CTA per SM, and a cluster stays within one group of SMs, so
// fewer than SMs / split).
static int64_t cluster_places(int split) {
    static int cached[kMaxDevices][2];
    const int dev = current_device();
    if (split == 1 || dev < 0) return num_sms() / split;
    int &places = cached[dev][split == 4];
    if (!places) {
        auto kern = gemm_kernel<RPTC_CODE_HASH, 2, 256, 2, false>;
        SmemOptIn first;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, 1, (unsigned)split);
        cfg.blockDim = dim3(kGemmThreads);
        cfg.dynamicSmemBytes = kGemmTop;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = (unsigned)split;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (allow_max_smem(kern, first) || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            n = num_sms() / split;
        }
        places = n;
    }
    return places;
}

// Tile and split: the combination whose slowest CTA finishes first, counted in whole waves of CTAs over the SMs.  The wide
// tile feeds the tensor pipe about 1.35 times faster per weight row, but there are half as many of it; sharing a tile's
// reduction over two or four CTAs fills SMs that would be idle (4096 rows x 512 tokens are 32 wide tiles for 148 SMs)
// at the price of the exchange.  A CTA keeps at least eight steps.
static GemmShape choose_shape(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f, double *estimate = nullptr) {
    GemmShape best = {0, 0, 0};
    double best_us = 0;
    const int64_t steps = n / kStepCols;
    for (int rows = 256; rows >= 32; rows >>= 1) {
        for (int halves = tokens > 128 && rows >= 128 ? 2 : 1; halves >= 1; --halves) {
            GemmParams probe;
            if (!plan_gemm(probe, {rows, halves, 1}, f) || tokens > 65535 * 128 * (int64_t)halves) continue;      // a grid row per tile of tokens
            const int64_t tiles = banks.banks * ((m + rows - 1) / rows) * ((tokens + halves * 128 - 1) / (halves * 128));
            for (int split = 1; split <= (banks.may_split && rows >= 128 ? rows / 64 : 1) && (split == 1 || steps >= 8 * split); split *= 2) {
                const int64_t places = cluster_places(split);
                const int64_t waves = (tiles + places - 1) / places;
                const double us = waves * ((double)((steps + split - 1) / split) * step_us(rows, halves, f.code) + around_us(rows, halves, split));
                if (!best.rows || us < best_us) best = {rows, halves, split}, best_us = us;
            }
        }
    }
    if (estimate) *estimate = best_us;
    return best;
}

double gemm_us(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f) {
    double us;
    choose_shape(m, n, tokens, banks, f, &us);
    return us;
}

int64_t gemm_bank_columns(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f) {
    const GemmShape g = choose_shape(m, n, tokens, banks, f);
    return g.rows ? (m + g.rows - 1) / g.rows * g.rows : 0;
}

int gemm_banked(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x, void *y, int64_t ld_y, int64_t m,
                int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f, cudaStream_t s) {
    const GemmShape g = choose_shape(m, n, tokens, banks, f);
    GemmParams p;
    if (!g.rows || !plan_gemm(p, g, f)) return RPTC_ERR_UNSUPPORTED;
    p.tiles_per_bank = (int32_t)((m + g.rows - 1) / g.rows);
    CUtensorMap map, ymap;
    const int x_rows = g.halves == 1 && tokens < 128 ? (int)((tokens + 7) / 8 * 8) : 128;      // what lies in a stage's other rows does not mix with these
    p.x_bytes = (uint32_t)x_rows * kStepCols * 2;
    if (int e = encode_map(map, x, n, tokens, ld_x, x_rows)) return e;
    if (int e = encode_map(ymap, y, banks.banks == 1 ? m : (int64_t)banks.banks * p.tiles_per_bank * g.rows, tokens, ld_y, 128, g.rows == 32 ? 32 : 64)) return e;
    p.codes = static_cast<const uint4 *>(codes);
    p.lut = static_cast<const __half *>(lut);
    p.carry_in = carry_in;
    p.m = m;
    p.n = n;
    p.tokens = tokens;
    p.n_units = (int32_t)(n * f.K / 128);
    p.L = f.L;
    p.S = f.S;
    p.n_split = g.split;
    p.lut_stride = banks.lut_stride;
    p.status = device_status_word();
    if (!p.status) return RPTC_ERR_CUDA;
    const size_t smem = kGemmTop;            // covers every planned address whatever the start of the dynamic area
    const dim3 grid((unsigned)(banks.banks * p.tiles_per_bank), (unsigned)((tokens + g.halves * 128 - 1) / (g.halves * 128)), (unsigned)g.split);
    switch (f.code) {
        case RPTC_CODE_LUT:
            return f.K == 2 ? launch_gemm_shape<RPTC_CODE_LUT, 2>(g, p, map, ymap, smem, grid, s)
                            : launch_gemm_shape<RPTC_CODE_LUT, 4>(g, p, map, ymap, smem, grid, s);
        case RPTC_CODE_HASH:
            return launch_gemm_shape<RPTC_CODE_HASH, 2>(g, p, map, ymap, smem, grid, s);
        case RPTC_CODE_LITE:
            return f.K == 2 ? launch_gemm_shape<RPTC_CODE_LITE, 2>(g, p, map, ymap, smem, grid, s)
                            : launch_gemm_shape<RPTC_CODE_LITE, 4>(g, p, map, ymap, smem, grid, s);
    }
    return RPTC_ERR_UNSUPPORTED;
}

int check_format(const rptc_format *f);   // api.cu

}  // namespace rptc

using namespace rptc;

static int gemm_checked(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x, void *y, int64_t ld_y, int64_t m,
                        int64_t n, int64_t tokens, const Banks &banks, const rptc_format *fmt, rptc_stream_t stream) {
    if (!codes || !lut || !x || !y || !fmt) return RPTC_ERR_ARG;
    if (int e = check_format(fmt)) return e;
    if (fmt->layout != RPTC_LAYOUT_TILED || fmt->quirk != RPTC_QUIRK_NONE) return RPTC_ERR_UNSUPPORTED;
    if (fmt->K != 2 && fmt->K != 4) return RPTC_ERR_UNSUPPORTED;
    if (m <= 0 || n <= 0 || tokens <= 0 || (m % 128) || (n % kStepCols) || ld_x < n || ld_y < m) return RPTC_ERR_SHAPE;
    if (m > (int64_t(1) << 30) || n > (int64_t(1) << 30) || tokens > (int64_t(1) << 24)) return RPTC_ERR_TOO_LARGE;
    if ((reinterpret_cast<uintptr_t>(codes) & 15) || (reinterpret_cast<uintptr_t>(lut) & 15) || (reinterpret_cast<uintptr_t>(x) & 15) ||
        (reinterpret_cast<uintptr_t>(y) & 15) || (ld_x % 8) || (ld_y % 8))
        return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    return gemm_banked(codes, lut, carry_in, x, ld_x, y, ld_y, m, n, tokens, banks, *fmt, static_cast<cudaStream_t>(stream));
}

extern "C" int rptc_gemm(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x, void *y,
                         int64_t ld_y, int64_t m, int64_t n, int64_t tokens, const rptc_format *fmt, rptc_stream_t stream) {
    return gemm_checked(codes, lut, carry_in, x, ld_x, y, ld_y, m, n, tokens, Banks(), fmt, stream);
}

extern "C" int rptc_gemm_invariant(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x, void *y,
                                   int64_t ld_y, int64_t m, int64_t n, int64_t tokens, const rptc_format *fmt, rptc_stream_t stream) {
    Banks banks;
    banks.may_split = false;
    return gemm_checked(codes, lut, carry_in, x, ld_x, y, ld_y, m, n, tokens, banks, fmt, stream);
}
