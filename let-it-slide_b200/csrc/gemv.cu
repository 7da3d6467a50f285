// Fused RPTC decode + matvec for one or two activation rows on sm_100a (more of them: gemv_tcgen05.cu).
//
// The kernel for the native layout is in gemv_rows.cuh.  Other layouts (and the reference-quirk modes) take plain 128-bit loads in
// kernels of their own.
#include "gemv_rows.cuh"

namespace rptc {

// The general kernel: any layout (strided 128-bit loads straight from memory, one unit of one row block per
// step), the reference kernels' lane-0 deviations, batch 1.  It is left with the layouts whose 32 rows of a unit lie
// together (UNITMAJOR, TILED with a deviation); the others have kernels of their own below.
template <int CODE, int K>
__global__ void __launch_bounds__(kGemvThreads, 1) gemv_kernel(const GemvParams p) {
    constexpr int WPU = 128 / K;          // weights per unit
    constexpr int PAIRS = WPU / 2;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t s0 = smem_addr(smem_raw);
    uint32_t lut_tab, xs;
    if (CODE == RPTC_CODE_HASH) {
        lut_tab = kHashLutWindow;
        xs = kHashLutWindow + kHashLutBytes;
    } else {
        lut_tab = s0 + kBarBytes;
        xs = lut_tab + lut_bytes<CODE>(p.L, p.S);
    }
    // ---- prologue: nothing here depends on the kernels before this one ----
    lut_fill<CODE>(lut_tab, p.lut, p.L, p.S);
    const Lut<CODE> lut = lut_view<CODE>(lut_tab, p.L, p.S);
    pdl_allow_next_grid();

    const uint32_t n_rb = (uint32_t)(p.m >> 5);
    const uint32_t gw = blockIdx.x * kGemvWarps + warp, GW = gridDim.x * kGemvWarps;
    bool waited_prior = false;

    for (int32_t useg0 = 0; useg0 < p.n_units; useg0 += p.seg_units) {
        const int32_t nu = min(p.seg_units, p.n_units - useg0);
        // Balanced contiguous split of the T = row blocks x units steps over the GW warps of the grid, in 32-bit
        // arithmetic: the first T % GW warps take one step more than the others.
        const uint32_t T = (uint32_t)n_rb * (uint32_t)nu;
        const uint32_t per = T / GW, extra = T - per * GW;
        const uint32_t g0 = gw * per + min(gw, extra);
        const uint32_t count = per + (gw < extra ? 1u : 0u);
        const uint32_t rb0 = count ? g0 / (uint32_t)nu : 0u;
        const int32_t gi0 = count ? (int32_t)(g0 - rb0 * (uint32_t)nu) : 0;

        int64_t frb = rb0;          // fetch cursor, one step ahead of the decode
        int32_t fgi = gi0;
        auto next_unit_ptr = [&]() -> const uint4 * {
            const uint4 *ptr = p.codes + unit_index(p.st, useg0 + fgi, (frb << 5) + lane);
            if (++fgi == nu) {
                fgi = 0;
                ++frb;
            }
            return ptr;
        };

        // ---- activations of this column segment -> shared memory ----
        if (!waited_prior) {
            pdl_wait_prior_grids();
            waited_prior = true;
        }
        if (useg0 > 0) __syncthreads();          // everyone is done with the previous segment's x
        {
            const int64_t col0 = (int64_t)useg0 * WPU;
            const int pairs = nu * PAIRS;
            for (int i = threadIdx.x; i < pairs; i += kGemvThreads) {
                int64_t src = (col0 >> 1) + i;
                if (p.x_order == RPTC_XORDER_K2_LEGACY) src = k2_legacy_pair(src, p.n);
                const uint32_t v = ld_ordered_u32(reinterpret_cast<const uint32_t *>(p.x) + src);
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(xs + 4u * i), "r"(v) : "memory");
            }
        }
        __syncthreads();

        // ---- main loop over this warp's steps ----
        int64_t rb = rb0;
        int32_t gi = gi0;
        bool fresh = true;                        // the next step starts a run: fetch its history, zero the sum
        uint32_t prevw = 0;
        float facc = 0.f;
        uint4 nextv = make_uint4(0, 0, 0, 0);
        if (count > 0) nextv = ldg128_stream(next_unit_ptr());

#pragma unroll 1
        for (uint32_t k = 0; k < count; ++k) {
            const int64_t row = (rb << 5) + lane;
            const int32_t u = useg0 + gi;
            if (fresh) {
                fresh = false;
                if (u == 0)
                    prevw = p.carry_in ? __ldg(p.carry_in + row) : 0u;
                else
                    prevw = __ldg(reinterpret_cast<const uint32_t *>(p.codes + unit_index(p.st, u - 1, row)) + 3);
                facc = 0.f;
            }
            const bool last_of_block = gi == nu - 1;
            const uint4 v = nextv;
            if (k + 1 < count) nextv = ldg128_stream(next_unit_ptr());
            uint32_t halo = prevw;
            if (p.quirk != RPTC_QUIRK_NONE && (u & 31) == 0) {        // the reference kernels' lane-0 deviations
                if (p.quirk == RPTC_QUIRK_K2_LANE0_CARRY) halo = v.w;
                else if (u > 0) halo = prevw >> 16;
            }
            prevw = v.w;
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            const uint32_t xu = xs + (uint32_t)gi * (WPU * 2u);
            __half2 hacc[4];
            uint4 xv;
            decode_group<CODE, K>(w, halo, lut, [&](int pi, __half2 wp) {
                if ((pi & 3) == 0) xv = lds128(xu + 4u * pi);
                const uint32_t xq = (pi & 3) == 0 ? xv.x : (pi & 3) == 1 ? xv.y : (pi & 3) == 2 ? xv.z : xv.w;
                hacc[pi & 3] = pi < 4 ? __hmul2(wp, u32_as_half2(xq)) : __hfma2(wp, u32_as_half2(xq), hacc[pi & 3]);
            });
            const float2 f2 = __half22float2(__hadd2(__hadd2(hacc[0], hacc[1]), __hadd2(hacc[2], hacc[3])));
            facc += f2.x + f2.y;
            if (last_of_block || k + 1 == count) {
                atomicAdd(p.acc + row, facc);
                fresh = true;
            }
            if (last_of_block) {
                gi = 0;
                ++rb;
            } else {
                ++gi;
            }
        }
    }
    if (!waited_prior) pdl_wait_prior_grids();
}

// ---- layouts whose units of a row lie together (ROWMAJOR, CHUNKED), batch 1 ------------------------------------------------
// lane = unit: a warp takes one row of a chunk of 32 units (2048 columns at two bits) per step, a single 512-byte request where
// lane = row would touch 32 places 512 bytes or more apart (16384 x 16384, CHUNKED: 70 us).  The activations of a lane's
// unit stay in registers while the warp walks down the rows of the chunk; the 16 bits in front of a unit come from the lane
// to the left, in front of the chunk from memory.  Codes arrive through a private ring of asynchronous copies, four rows
// ahead.  fp16 pair products per unit, fp32 sums across the lanes.  Bound by the table look-ups; against lane = row, 16384 x
// 16384: HASH 65 -> 54 us, LUT 145 -> 134 us, LITE 73 -> 66 us; 4096 x 4096 HASH in a drop-in call 32.4 -> 31 us.
constexpr int kUnitsAhead = 4;
constexpr uint32_t kUnitsRing = kGemvWarps * kUnitsAhead * 512, kUnitsHist = kGemvWarps * kUnitsAhead * 4;
static_assert(kBarBytes + kUnitsRing + kUnitsHist + 1024 <= kHashLutWindow, "ring must fit below the HASH table window");
template <int CODE, int K>
__global__ void __launch_bounds__(kGemvThreads, 1) gemv_units_kernel(const GemvParams p) {
    constexpr int PAIRS = 64 / K, PPU = PAIRS / 4;            // activation pairs, 16-byte pieces of them, per unit
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t s0 = smem_addr(smem_raw);
    const uint32_t ring = s0 + kBarBytes + (uint32_t)warp * (kUnitsAhead * 512) + 16u * lane;
    const uint32_t hist = s0 + kBarBytes + kUnitsRing + (uint32_t)warp * (kUnitsAhead * 4);
    const uint32_t lut_tab = CODE == RPTC_CODE_HASH ? kHashLutWindow : s0 + kBarBytes + kUnitsRing + kUnitsHist;
    const uint32_t xs = lut_tab + lut_bytes<CODE>(p.L, p.S);
    if (CODE == RPTC_CODE_LUT) {
        if (threadIdx.x == 0) {
            mbar_init(s0, 1);
            mbar_fence_init();
            mbar_expect_tx(s0, 2u << p.L);
            bulk_g2s(lut_tab, p.lut, 2u << p.L, s0);
        }
    } else {
        lut_fill<CODE>(lut_tab, p.lut, p.L, p.S);
    }
    const Lut<CODE> lut = lut_view<CODE>(lut_tab, p.L, p.S);
    pdl_allow_next_grid();
    // (chunk, row) pairs, chunk by chunk, in equal ranges per CTA; a warp takes every sixteenth row of the range
    const uint32_t m = (uint32_t)p.m, chunks = (uint32_t)(p.n_units + 31) >> 5, T = chunks * m;
    const uint32_t per = T / gridDim.x, extra = T - per * gridDim.x;
    const uint32_t c0 = blockIdx.x * per + min(blockIdx.x, extra), c1 = c0 + per + (blockIdx.x < extra ? 1u : 0u);
    bool first = true;
    for (uint32_t pos = c0; pos < c1;) {
        const uint32_t chunk = pos / m, r0 = pos - chunk * m, r1 = min(m, r0 + (c1 - pos));
        pos += r1 - r0;
        const int32_t u = (int32_t)(chunk * 32) + lane;
        const bool active = u < p.n_units;
        const uint4 *base = p.codes + (int64_t)chunk * p.st.hi + lane;
        uint32_t f_row = r0 + warp, f_slot = 0;               // fetch cursor
        auto fetch = [&]() {
            if (f_row < r1) {
                const uint4 *src = base + (int64_t)f_row * p.st.row;
                if (active) cp_async16(ring + f_slot * 512u, src);
                if (lane == 0) {
                    if (chunk == 0) {
                        const uint32_t v = p.carry_in ? __ldg(p.carry_in + f_row) : 0u;
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(hist + 4u * f_slot), "r"(v) : "memory");
                    } else {      // the last word of the row's unit in front of the chunk
                        const uint32_t *last = reinterpret_cast<const uint32_t *>(p.codes + (int64_t)(chunk - 1) * p.st.hi + 31 + (int64_t)f_row * p.st.row) + 3;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(hist + 4u * f_slot), "l"(last) : "memory");
                    }
                }
            }
            cp_async_commit();                                // an empty group when nothing is left keeps the count constant
            f_row += kGemvWarps;
            f_slot = (f_slot + 1) % kUnitsAhead;
        };
#pragma unroll 1
        for (int i = 0; i < kUnitsAhead; ++i) fetch();
        if (first) pdl_wait_prior_grids();
        else __syncthreads();                                 // everyone is done with the chunk before
        // activations of the chunk; piece j of unit q sits at piece j ^ swz(q), so that 32 lanes read theirs without conflicts
        auto swz = [](int q) { return (uint32_t)(PPU == 8 ? q & 7 : (q >> 1) & 3); };
        for (int i = threadIdx.x; i < 32 * PAIRS; i += kGemvThreads) {
            const int q = i / PAIRS, w = i % PAIRS;
            const int64_t s = (int64_t)chunk * (32 * PAIRS) + i;
            uint32_t v = 0;
            if (2 * s < p.n) v = ld_ordered_u32(reinterpret_cast<const uint32_t *>(p.x) + (p.x_order == RPTC_XORDER_K2_LEGACY ? k2_legacy_pair(s, p.n) : s));
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(xs + (((uint32_t)(q * PPU) + ((uint32_t)(w >> 2) ^ swz(q))) << 4) + 4u * (w & 3)), "r"(v) : "memory");
        }
        __syncthreads();
        if (CODE == RPTC_CODE_LUT && first && !mbar_wait(s0, 0, p.status)) {
            cp_async_wait<0>();
            return;
        }
        first = false;
        uint32_t xr[PAIRS];
#pragma unroll
        for (int j = 0; j < PPU; ++j) {
            const uint4 v = lds128(xs + (((uint32_t)(lane * PPU) + ((uint32_t)j ^ swz(lane))) << 4));
            xr[4 * j] = v.x, xr[4 * j + 1] = v.y, xr[4 * j + 2] = v.z, xr[4 * j + 3] = v.w;
        }
        uint32_t slot = 0;
#pragma unroll 1
        for (uint32_t row = r0 + warp; row < r1; row += kGemvWarps) {
            cp_async_wait<kUnitsAhead - 1>();
            const uint4 v = lds128(ring + slot * 512u);
            uint32_t halo = __shfl_up_sync(0xFFFFFFFFu, v.w, 1);
            if (lane == 0) {
                halo = lds32(hist + 4u * slot);
                if (p.quirk == RPTC_QUIRK_K2_LANE0_CARRY) halo = v.w;      // the reference kernels' lane-0 deviations
                else if (p.quirk == RPTC_QUIRK_K1_LANE0_SEED && u > 0) halo >>= 16;
            }
            fetch();                                          // the words are in registers
            slot = (slot + 1) % kUnitsAhead;
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            __half2 hacc[4];
            decode_group<CODE, K>(w, halo, lut, [&](int pi, __half2 wp) {
                const __half2 x2 = u32_as_half2(xr[pi]);
                hacc[pi & 3] = pi < 4 ? __hmul2(wp, x2) : __hfma2(wp, x2, hacc[pi & 3]);
            });
            const float2 f2 = __half22float2(__hadd2(__hadd2(hacc[0], hacc[1]), __hadd2(hacc[2], hacc[3])));
            float sum = active ? f2.x + f2.y : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
            if (lane == 0) atomicAdd(p.acc + row, sum);
        }
        cp_async_wait<0>();
    }
    if (first) {                                              // a CTA without work
        pdl_wait_prior_grids();
        if (CODE == RPTC_CODE_LUT && threadIdx.x == 0) mbar_wait(s0, 0, p.status);      // its table must not land in memory given back
    }
}

__global__ void gemv_finish_kernel(float *__restrict__ acc, int64_t ld_acc, __half *__restrict__ y, int64_t ld_y,
                                   int64_t m, int batch, float scale, int accumulate, int clear) {
    pdl_allow_next_grid();
    pdl_wait_prior_grids();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m * batch) return;
    const int64_t b = i / m, r = i - b * m;
    float v = acc[b * ld_acc + r] * scale;
    if (accumulate) {
        // the reference accumulates in fp16: out = out + delta (inference_t.cu:170-171)
        y[b * ld_y + r] = __hadd(y[b * ld_y + r], __float2half_rn(v));
    } else {
        y[b * ld_y + r] = __float2half_rn(v);
    }
    if (clear) acc[b * ld_acc + r] = 0.f;
}

template <int CODE, int K>
static int launch_gemv(const GemvParams &p, size_t smem, cudaStream_t stream) {
    static SmemOptIn opted;
    auto kern = gemv_kernel<CODE, K>;
    if (int e = allow_max_smem(kern, opted)) return e;
    return launch(kern, dim3(num_sms()), dim3(kGemvThreads), smem, stream, p);
}

template <int CODE, int K>
static int launch_gemv_units(const GemvParams &p, cudaStream_t stream) {
    static SmemOptIn opted;
    auto kern = gemv_units_kernel<CODE, K>;
    if (int e = allow_max_smem(kern, opted)) return e;
    const size_t x = 32 * (128 / K) * 2;                              // one chunk of activations
    const size_t smem = CODE == RPTC_CODE_HASH ? kHashLutWindow + kHashLutBytes + x
                                               : kBarBytes + kUnitsRing + kUnitsHist + (CODE == RPTC_CODE_LUT ? size_t(2) << p.L : size_t(128) << p.S) + x + 128;
    return launch(kern, dim3(num_sms()), dim3(kGemvThreads), smem, stream, p);
}

template <int CODE, int K>
static int dispatch(const GemvParams &p, int batch, bool tiled, size_t smem, dim3 grid, cudaStream_t stream) {
    if (!tiled) {
        if (batch != 1 || p.in.h_in) return RPTC_ERR_UNSUPPORTED;
        return p.st.lo == 1 ? launch_gemv_units<CODE, K>(p, stream) : launch_gemv<CODE, K>(p, smem, stream);
    }
    if (p.in.h_in) {
        if (batch > 2) return RPTC_ERR_UNSUPPORTED;
        return batch == 1 ? launch_gemv_rows<CODE, K, 1, 1>(p, smem, stream) : launch_gemv_rows<CODE, K, 2, 1>(p, smem, stream);
    }
    switch (batch) {
        case 1: return launch_gemv_rows<CODE, K, 1, 0>(p, smem, stream, grid);
        case 2: return launch_gemv_rows<CODE, K, 2, 0>(p, smem, stream, grid);
    }
    return RPTC_ERR_ARG;
}

// One launch for batch in {1,2}.
static int gemv_one(const void *codes, const void *lut, const uint32_t *carry_in, const __half *x, int64_t ld_x, float *acc,
                    int64_t ld_acc, int64_t m, int64_t n, int batch, int x_order, const rptc_format &f, cudaStream_t stream,
                    const rptc_gemv_input *in = nullptr, const Banks &banks = Banks()) {
    const int K = f.K;
    const int wpu = 128 / K;
    GemvParams p;
    p.codes = static_cast<const uint4 *>(codes);
    p.n_units = (int32_t)(n / wpu);
    p.st = unit_strides(f.layout, m, p.n_units);
    p.lut = static_cast<const __half *>(lut);
    p.carry_in = carry_in;
    p.x = x;
    p.ld_x = ld_x;
    p.acc = acc;
    p.ld_acc = ld_acc;
    p.m = m;
    p.n = n;
    p.L = f.L;
    p.S = f.S;
    p.quirk = f.quirk;
    p.x_order = x_order;
    p.status = device_status_word();
    if (!p.status) return RPTC_ERR_CUDA;
    const bool tma = f.layout == RPTC_LAYOUT_TILED && f.quirk == RPTC_QUIRK_NONE;
    p.in = in ? *in : rptc_gemv_input{};
    // one bank's table per CTA: the SMs are dealt out to the banks
    const int ctas = num_sms() / banks.banks;
    const dim3 grid((unsigned)(ctas > 0 ? ctas : 1), (unsigned)banks.banks);
    p.lut_stride = banks.lut_stride;

    // shared-memory plan (must mirror the kernel's)
    const size_t kMaxSmem = 227 * 1024 - 1024;     // leave room for the 1 KiB the system may reserve
    size_t fixed;
    if (f.code == RPTC_CODE_HASH) fixed = kHashLutWindow + kHashLutBytes;      // addresses are absolute in the window
    else fixed = kBarBytes + (tma ? kRingBytes : 0) + (f.code == RPTC_CODE_LUT ? (size_t(2) << f.L) : (size_t(128) << f.S)) + 128;
    if (fixed + 1024 > kMaxSmem) return RPTC_ERR_UNSUPPORTED;
    size_t x_budget = kMaxSmem - fixed;
    if (x_budget > 96 * 1024) x_budget = 96 * 1024;
    const size_t unit_x_bytes = size_t(batch) * wpu * 2;
    int64_t seg = (int64_t)(x_budget / unit_x_bytes);
    if (x_order == RPTC_XORDER_K2_LEGACY) seg = seg / 32 * 32;
    if (seg < 1) return RPTC_ERR_TOO_LARGE;
    if (seg > p.n_units) seg = p.n_units;
    p.seg_units = (int32_t)seg;
    size_t smem = fixed + size_t(seg) * unit_x_bytes;
    if (in) {
        if (seg != p.n_units) return RPTC_ERR_TOO_LARGE;                        // computed activations live in one segment
        const size_t ex = (n > 4096 || batch > 1 ? 2 : 1) * kUnitFloats * sizeof(float);      // exchange buffers of the 4096-point transforms
        static_assert(2 * kUnitFloats * sizeof(float) <= kRingBytes, "they must fit into the ring");
        p.ex_on_ring = smem + ex > kMaxSmem;
        if (!p.ex_on_ring) smem += ex;
        if (smem > kMaxSmem) return RPTC_ERR_TOO_LARGE;
    }

    switch (f.code) {
        case RPTC_CODE_LUT:
            if (K == 2) return dispatch<RPTC_CODE_LUT, 2>(p, batch, tma, smem, grid, stream);
            if (K == 4) return dispatch<RPTC_CODE_LUT, 4>(p, batch, tma, smem, grid, stream);
            break;
        case RPTC_CODE_HASH:
            if (K == 2) return dispatch<RPTC_CODE_HASH, 2>(p, batch, tma, smem, grid, stream);
            break;
        case RPTC_CODE_LITE:
            if (K == 2) return dispatch<RPTC_CODE_LITE, 2>(p, batch, tma, smem, grid, stream);
            if (K == 4) return dispatch<RPTC_CODE_LITE, 4>(p, batch, tma, smem, grid, stream);
            break;
    }
    return RPTC_ERR_UNSUPPORTED;
}

int check_format(const rptc_format *f);   // api.cu

int gemv_banked(const void *codes, const void *lut, const void *x, int64_t ld_x, float *acc, int64_t ld_acc, int64_t m, int64_t n, int64_t tokens,
                const Banks &banks, const rptc_format &f, cudaStream_t stream, bool ordered, float *partial) {
    if (tokens > 2 && gemv_few_takes(m, n, tokens, banks, f, x, ld_x))
        return gemv_few(codes, lut, nullptr, x, ld_x, acc, ld_acc, m, n, tokens, banks, f, stream, ordered, partial);
    for (int64_t t = 0; t < tokens; t += 2) {
        const int e = gemv_one(codes, lut, nullptr, static_cast<const __half *>(x) + t * ld_x, ld_x, acc + t * ld_acc, ld_acc, m, n,
                               tokens - t >= 2 ? 2 : 1, RPTC_XORDER_NATURAL, f, stream, nullptr, banks);
        if (e) return e;
    }
    return RPTC_OK;
}

}  // namespace rptc

using namespace rptc;

constexpr int kMaxGemvBatch = 64;      // rows of activations per call

// Every check of rptc_gemv's arguments that needs no device work, in the order the entry point reports them.
int rptc::validate_gemv_args(const void *codes, const void *lut, const void *x, int64_t ld_x, const float *acc, int64_t ld_acc,
                              int64_t m, int64_t n, int batch, int x_order, const rptc_format *fmt) {
    if (!codes || !lut || !x || !acc || !fmt) return RPTC_ERR_ARG;
    if (int e = rptc::check_format(fmt)) return e;
    if (fmt->K != 2 && fmt->K != 4) return RPTC_ERR_UNSUPPORTED;
    if (batch < 1 || batch > kMaxGemvBatch) return RPTC_ERR_ARG;
    if (x_order != RPTC_XORDER_NATURAL && x_order != RPTC_XORDER_K2_LEGACY) return RPTC_ERR_ARG;
    if (m <= 0 || n <= 0 || (m % 32) || (n % (128 / fmt->K))) return RPTC_ERR_SHAPE;
    if (x_order == RPTC_XORDER_K2_LEGACY && (n % 2048 || fmt->K != 2)) return RPTC_ERR_SHAPE;
    if (fmt->layout == RPTC_LAYOUT_CHUNKED && (n / (128 / fmt->K)) % 32) return RPTC_ERR_SHAPE;
    if (m > (int64_t(1) << 30) || n > (int64_t(1) << 30) || (m / 32) * (n / (128 / fmt->K)) >= (int64_t(1) << 31))
        return RPTC_ERR_TOO_LARGE;
    if ((reinterpret_cast<uintptr_t>(codes) & 15) || (reinterpret_cast<uintptr_t>(lut) & 15) ||
        (reinterpret_cast<uintptr_t>(x) & 3) || (ld_x & 1))
        return RPTC_ERR_ALIGN;
    if (ld_x < n || ld_acc < m) return RPTC_ERR_SHAPE;
    return RPTC_OK;
}

extern "C" int rptc_gemv(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x,
                         float *acc, int64_t ld_acc, int64_t m, int64_t n, int batch, int x_order, const rptc_format *fmt,
                         rptc_stream_t stream) {
    if (int e = validate_gemv_args(codes, lut, x, ld_x, acc, ld_acc, m, n, batch, x_order, fmt)) return e;
    if (int e = rptc_check_device()) return e;
    // Up to two rows the lane-per-row kernel is the faster one (28672 x 8192: 28.0 against 30.6 us).
    if (batch > 2 && x_order == RPTC_XORDER_NATURAL && gemv_few_takes(m, n, batch, Banks(), *fmt, x, ld_x))
        return gemv_few(codes, lut, carry_in, x, ld_x, acc, ld_acc, m, n, batch, Banks(), *fmt, static_cast<cudaStream_t>(stream));
    // what the kernel for a few rows does not take (rows of x that are not 16-byte aligned, the legacy order): pairs of rows, and one at a
    // time where the general kernels are the only ones (the reference's layouts and deviations)
    const bool pairs = fmt->layout == RPTC_LAYOUT_TILED && fmt->quirk == RPTC_QUIRK_NONE;
    int done = 0;
    while (done < batch) {
        const int b = pairs && batch - done >= 2 ? 2 : 1;
        int e = gemv_one(codes, lut, carry_in, static_cast<const __half *>(x) + (int64_t)done * ld_x, ld_x,
                         acc + (int64_t)done * ld_acc, ld_acc, m, n, b, x_order, *fmt, static_cast<cudaStream_t>(stream));
        if (e) return e;
        done += b;
    }
    return RPTC_OK;
}

extern "C" int rptc_gemv_finish(float *acc, int64_t ld_acc, void *y, int64_t ld_y, int64_t m, int batch, float scale,
                                int accumulate, int clear, rptc_stream_t stream) {
    if (!acc || !y) return RPTC_ERR_ARG;
    if (m <= 0 || batch < 1 || ld_acc < m || ld_y < m) return RPTC_ERR_SHAPE;
    if (int e = rptc_check_device()) return e;
    const int64_t total = m * batch;
    return launch(gemv_finish_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, static_cast<cudaStream_t>(stream),
                  acc, ld_acc, static_cast<__half *>(y), ld_y, m, batch, scale, accumulate, clear);
}

// ---- entry point that allocates nothing --------------------------------------------------------------
// Some hosts of this library may not call cudaMalloc where they call us: a serving process whose memory
// pool owns every byte of the device, a plugin that runs under an allocator it must not bypass, or code
// that has been told its memory footprint is frozen.  For them the fp32 accumulator of the fused matvec
// lives in this fixed array, which every GPU that loads the library holds until the process exits.
namespace rptc {
constexpr int64_t kStaticAccFloats = 262144;                      // 1 MiB: batch * m may not exceed this
static __device__ __align__(256) float g_static_acc[kStaticAccFloats];
static float *g_static_acc_ptr[kMaxDevices];                               // device address of the array, per device
}  // namespace rptc

extern "C" int rptc_gemv_f16_static(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x,
                                    void *y, int64_t ld_y, int64_t m, int64_t n, int batch, int x_order, const rptc_format *fmt,
                                    rptc_stream_t stream) {
    if (!y) return RPTC_ERR_ARG;
    if (batch < 1 || batch > 8 || m <= 0) return RPTC_ERR_ARG;
    if ((int64_t)batch * m > kStaticAccFloats) return RPTC_ERR_TOO_LARGE;      // the fixed accumulator cannot hold it
    if (ld_y < m) return RPTC_ERR_SHAPE;
    // Everything that can refuse the call is checked before the shared array is touched: a rejected call must not put a
    // clearing of the array on the caller's stream (it could land in the middle of a valid call on another stream).
    // The non-null placeholder stands for the accumulator, whose address is not known yet.
    if (int e = validate_gemv_args(codes, lut, x, ld_x, reinterpret_cast<const float *>(codes), m, m, n, batch, x_order, fmt)) return e;
    if (int e = rptc_check_device()) return e;
    const int dev = current_device();
    if (dev < 0) return RPTC_ERR_ARG;
    if (!g_static_acc_ptr[dev]) {
        // Set-up, once per device, with that device current: in host code the array's name is only a handle,
        // the address a kernel can use has to be asked for.
        float *ptr = nullptr;
        RPTC_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&ptr), g_static_acc));
        g_static_acc_ptr[dev] = ptr;
    }
    float *acc = g_static_acc_ptr[dev];
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // every call shares the array and finds the previous call's leftovers in it: start from zero
    RPTC_CUDA(cudaMemsetAsync(acc, 0, sizeof(float) * (size_t)batch * (size_t)m, s));
    if (int e = rptc_gemv(codes, lut, carry_in, x, ld_x, acc, m, m, n, batch, x_order, fmt, stream)) return e;
    return rptc_gemv_finish(acc, m, y, ld_y, m, batch, 1.0f, 0, 0, stream);
}

extern "C" int rptc_gemv_glued(const void *codes, const void *lut, const uint32_t *carry_in, const rptc_gemv_input *in, float *acc,
                               int64_t ld_acc, int64_t m, int64_t n, int batch, const rptc_format *fmt, rptc_stream_t stream) {
    if (!codes || !lut || !in || !acc || !fmt) return RPTC_ERR_ARG;
    if (int e = check_format(fmt)) return e;
    if (fmt->K != 2 && fmt->K != 4) return RPTC_ERR_UNSUPPORTED;
    if (fmt->layout != RPTC_LAYOUT_TILED || fmt->quirk != RPTC_QUIRK_NONE || batch < 1 || batch > 2) return RPTC_ERR_UNSUPPORTED;
    if (m <= 0 || n <= 0 || (m % 32) || (n % (128 / fmt->K)) || ld_acc < m) return RPTC_ERR_SHAPE;
    if (m > (int64_t(1) << 30) || (m / 32) * (n / (128 / fmt->K)) >= (int64_t(1) << 31)) return RPTC_ERR_TOO_LARGE;
    auto misaligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
    if (misaligned(codes) || misaligned(lut) || misaligned(in->acc) || misaligned(in->signs_out) || misaligned(in->signs_in) ||
        misaligned(in->clear) || (in->ld_acc % 4) || (in->clear_count % 4))
        return RPTC_ERR_ALIGN;
    if (in->clear_count < 0 || (in->clear_count && !in->clear)) return RPTC_ERR_ARG;
    if (n != 4096 && n != 8192) return RPTC_ERR_UNSUPPORTED;                    // one or two 4096-point blocks, sixteen values a thread
    if (!in->h_in || !in->h_out || in->h_in == in->h_out || !in->w_norm) return RPTC_ERR_ARG;
    if (in->ld_h < n || (in->acc && in->ld_acc < n)) return RPTC_ERR_SHAPE;
    if (misaligned(in->h_in) || misaligned(in->h_out) || misaligned(in->w_norm) || (in->ld_h % 8)) return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    return gemv_one(codes, lut, carry_in, nullptr, 0, acc, ld_acc, m, n, batch, RPTC_XORDER_NATURAL, *fmt,
                    static_cast<cudaStream_t>(stream), in);
}

extern "C" int rptc_gemv_swiglu(const void *codes, const void *lut, const uint32_t *carry_in, const float *prev_acc, int64_t ld_prev,
                                const void *signs_out, float scale_out, const void *signs_in, int block, float *acc, int64_t ld_acc,
                                int64_t m, int64_t n, int batch, const rptc_format *fmt, float *clear, int64_t clear_count,
                                rptc_stream_t stream) {
    if (!codes || !lut || !prev_acc || !acc || !fmt) return RPTC_ERR_ARG;
    if (int e = check_format(fmt)) return e;
    if (fmt->K != 2 && fmt->K != 4) return RPTC_ERR_UNSUPPORTED;
    if (fmt->layout != RPTC_LAYOUT_TILED || fmt->quirk != RPTC_QUIRK_NONE || batch < 1 || batch > 2) return RPTC_ERR_UNSUPPORTED;
    if (block < 8 || block > 256 || (block & (block - 1))) return RPTC_ERR_UNSUPPORTED;
    if (m <= 0 || n <= 0 || (m % 32) || (n % 256) || ld_acc < m || ld_prev < 2 * n) return RPTC_ERR_SHAPE;
    if (m > (int64_t(1) << 30) || (m / 32) * (n / (128 / fmt->K)) >= (int64_t(1) << 31)) return RPTC_ERR_TOO_LARGE;
    auto misaligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
    if (misaligned(codes) || misaligned(lut) || misaligned(prev_acc) || misaligned(signs_out) || misaligned(signs_in) || misaligned(clear) ||
        (ld_prev % 4) || (clear_count % 4))
        return RPTC_ERR_ALIGN;
    if (clear_count < 0 || (clear_count && !clear)) return RPTC_ERR_ARG;
    if (int e = rptc_check_device()) return e;
    const int K = fmt->K, wpu = 128 / K;
    GemvParams p{};
    p.codes = static_cast<const uint4 *>(codes);
    p.n_units = (int32_t)(n / wpu);
    p.st = unit_strides(fmt->layout, m, p.n_units);
    p.lut = static_cast<const __half *>(lut);
    p.carry_in = carry_in;
    p.acc = acc;
    p.ld_acc = ld_acc;
    p.m = m;
    p.n = n;
    p.L = fmt->L;
    p.S = fmt->S;
    p.quirk = fmt->quirk;
    p.x_order = RPTC_XORDER_NATURAL;
    p.status = device_status_word();
    if (!p.status) return RPTC_ERR_CUDA;
    float norm = 1.f;
    for (int b = block; b > 1; b >>= 2) norm *= (b >= 4) ? 0.5f : 0.70710678118654752f;
    p.sw.acc = const_cast<float *>(prev_acc);
    p.sw.in16 = nullptr;
    p.sw.ld_acc = ld_prev;
    p.sw.out = nullptr;
    p.sw.ld_out = 0;
    p.sw.signs_out = static_cast<const __half *>(signs_out);
    p.sw.signs_in = static_cast<const __half *>(signs_in);
    p.sw.n = n;
    p.sw.block = block;
    p.sw.chunk = 256;
    p.sw.clear = 0;
    p.sw.scale_out = scale_out * norm;
    p.sw.scale_in = norm;
    p.clear = clear;
    p.clear_count = clear_count;
    // the most 256-column blocks one CTA's granules can touch
    const int64_t upb = 256 / wpu, n_rbp = (m / 32 + 1) / 2, cell = n_rbp * upb;
    const int64_t T = n_rbp * p.n_units;
    const int64_t cta_granules = T / num_sms() + 1;
    int64_t max_blocks = (cta_granules + cell - 2) / cell + 1;
    if (max_blocks > n / 256) max_blocks = n / 256;
    p.seg_units = (int32_t)(max_blocks * upb);
    const size_t kMaxSmem = 227 * 1024 - 1024;
    size_t fixed;
    if (fmt->code == RPTC_CODE_HASH) fixed = kHashLutWindow + kHashLutBytes;
    else fixed = kBarBytes + kRingBytes + (fmt->code == RPTC_CODE_LUT ? (size_t(2) << fmt->L) : (size_t(128) << fmt->S)) + 128;
    const size_t smem = fixed + (size_t)batch * max_blocks * 512;
    if (smem > kMaxSmem) return RPTC_ERR_TOO_LARGE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (fmt->code) {
        case RPTC_CODE_LUT:
            if (K == 2) return batch == 1 ? launch_gemv_rows<RPTC_CODE_LUT, 2, 1, 2>(p, smem, s) : launch_gemv_rows<RPTC_CODE_LUT, 2, 2, 2>(p, smem, s);
            return batch == 1 ? launch_gemv_rows<RPTC_CODE_LUT, 4, 1, 2>(p, smem, s) : launch_gemv_rows<RPTC_CODE_LUT, 4, 2, 2>(p, smem, s);
        case RPTC_CODE_HASH:
            if (K == 2) return batch == 1 ? launch_gemv_rows<RPTC_CODE_HASH, 2, 1, 2>(p, smem, s) : launch_gemv_rows<RPTC_CODE_HASH, 2, 2, 2>(p, smem, s);
            break;
        case RPTC_CODE_LITE:
            if (K == 2) return batch == 1 ? launch_gemv_rows<RPTC_CODE_LITE, 2, 1, 2>(p, smem, s) : launch_gemv_rows<RPTC_CODE_LITE, 2, 2, 2>(p, smem, s);
            return batch == 1 ? launch_gemv_rows<RPTC_CODE_LITE, 4, 1, 2>(p, smem, s) : launch_gemv_rows<RPTC_CODE_LITE, 4, 2, 2>(p, smem, s);
    }
    return RPTC_ERR_UNSUPPORTED;
}
