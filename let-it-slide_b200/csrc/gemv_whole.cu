// A matvec whose caller waits for it, in the layouts whose units of a row lie together (the reference's matvec functions).
#include "gemv_rows.cuh"

namespace rptc {

constexpr int kUnitsAhead = 4;
constexpr uint32_t kUnitsRing = kGemvWarps * kUnitsAhead * 512, kUnitsHist = kGemvWarps * kUnitsAhead * 4;
// A CTA has whole rows, so that there is no accumulator to zero, to add to and to convert in a kernel behind.  A warp takes every
// sixteenth of its rows chunk by chunk (the activations of a chunk are read into registers once for up to eight rows), or, of fewer rows
// than warps, a part of the chunks.  All activations are staged at once; a lane's running sums are kept in shared memory.  The last CTA to
// finish leaves the device time in host memory (DeviceTimer), where the calling thread waits for it: 4096 x 4096 HASH, a drop-in call
// 31.3 us with a kernel behind and events around, 23.4 so.
constexpr int kWholeRows = 8;
constexpr uint32_t kWholeSums = kGemvWarps * kWholeRows * 32 * 4, kWholeParts = 256;
static_assert(kBarBytes + kUnitsRing + kUnitsHist + kWholeSums + kWholeParts + 1024 <= kHashLutWindow, "in front of the HASH table window");
struct GemvWhole : GemvParams {
    __half *y;
    int32_t accumulate, parts;
    DeviceTimer timer;
};
// k2_legacy_pair in 32 bits, as n is at most 2^30 (one division instead of two long ones; gemv_rows_kernel as a whole is slower with it: a
// decode step of 32 layers 1437 us against 1427).
__device__ __forceinline__ int64_t k2_legacy_pair_32(int64_t s, int64_t n) {
    const uint32_t it = (uint32_t)(s >> 10), lane = (uint32_t)(s >> 5) & 31u, o = (uint32_t)(s >> 2) & 7u, j = (uint32_t)s & 3u;
    const uint32_t k = (0x36251407u >> (4 * o)) & 7u;
    const uint32_t p = ((it * 8 + k) * 4 + j) * 32 + lane, q8 = (uint32_t)(n >> 3), q = p / q8;
    return 4 * (int64_t)(p - q * q8) + q;
}
template <int CODE, int K>
__global__ void __launch_bounds__(kGemvThreads, 1) gemv_whole_kernel(const GemvWhole p) {
    constexpr int PAIRS = 64 / K, PPU = PAIRS / 4;            // activation pairs, 16-byte pieces of them, per unit
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t s0 = smem_addr(smem_raw);
    const uint32_t ring = s0 + kBarBytes + (uint32_t)warp * (kUnitsAhead * 512) + 16u * lane;
    const uint32_t hist = s0 + kBarBytes + kUnitsRing + (uint32_t)warp * (kUnitsAhead * 4);
    const uint32_t sums0 = kBarBytes + kUnitsRing + kUnitsHist, after = sums0 + kWholeSums + kWholeParts;
    float *sums = reinterpret_cast<float *>(smem_raw + sums0) + warp * (kWholeRows * 32) + lane;
    float *part_sums = reinterpret_cast<float *>(smem_raw + sums0 + kWholeSums);
    const uint32_t lut_tab = CODE == RPTC_CODE_HASH ? kHashLutWindow : s0 + after;
    const uint32_t xs = lut_tab + lut_bytes<CODE>(p.L, p.S);
    if (CODE == RPTC_CODE_HASH && s0 + after > kHashLutWindow) {
        if (threadIdx.x == 0) atomicExch(p.status, kStatusSmemPlan);
        return;
    }
    pdl_wait_prior_grids();
    if (threadIdx.x == 0) p.timer.begin();
    if (CODE == RPTC_CODE_LUT && threadIdx.x == 0) {
        mbar_init(s0, 1);
        mbar_fence_init();
        mbar_expect_tx(s0, 2u << p.L);
        bulk_g2s(lut_tab, p.lut, 2u << p.L, s0);
    }
    const uint32_t m = (uint32_t)p.m, chunks = (uint32_t)(p.n_units + 31) >> 5;
    const uint32_t r0 = (uint32_t)((uint64_t)m * blockIdx.x / gridDim.x), r1 = (uint32_t)((uint64_t)m * (blockIdx.x + 1) / gridDim.x);
    const uint32_t parts = (uint32_t)p.parts, part = warp % parts, lanes_of_rows = kGemvWarps / parts, first = r0 + warp / parts;
    const uint32_t ch0 = chunks * part / parts, ch1 = chunks * (part + 1) / parts;
    const uint32_t mine = first < r1 ? (r1 - first + lanes_of_rows - 1) / lanes_of_rows : 0u;      // rows first, first + lanes_of_rows, ...
    const uint32_t steps = mine * (ch1 - ch0);

    // fetch cursor: groups of up to kWholeRows rows, chunk by chunk, row by row
    uint32_t f_left = steps, f_group = 0, f_chunk = ch0, f_i = 0, f_slot = 0;
    auto fetch = [&]() {
        if (f_left) {
            --f_left;
            const uint32_t row = first + (f_group + f_i) * lanes_of_rows;
            const uint4 *src = p.codes + (int64_t)f_chunk * p.st.hi + (int64_t)row * p.st.row;
            if ((int32_t)(f_chunk * 32) + lane < p.n_units) cp_async16(ring + f_slot * 512u, src + lane);
            if (lane == 0) {
                if (f_chunk == 0) {
                    const uint32_t v = p.carry_in ? __ldg(p.carry_in + row) : 0u;
                    asm volatile("st.shared.u32 [%0], %1;" ::"r"(hist + 4u * f_slot), "r"(v) : "memory");
                } else {      // the last word of the row's unit in front of the chunk
                    const uint32_t *last = reinterpret_cast<const uint32_t *>(p.codes + (int64_t)(f_chunk - 1) * p.st.hi + 31 + (int64_t)row * p.st.row) + 3;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(hist + 4u * f_slot), "l"(last) : "memory");
                }
            }
            if (++f_i == min((uint32_t)kWholeRows, mine - f_group)) {
                f_i = 0;
                if (++f_chunk == ch1) {
                    f_chunk = ch0;
                    f_group += kWholeRows;
                }
            }
        }
        cp_async_commit();                                    // an empty group when nothing is left keeps the count constant
        f_slot = (f_slot + 1) % kUnitsAhead;
    };
#pragma unroll 1
    for (int i = 0; i < kUnitsAhead; ++i) fetch();
    // all activations; piece j of unit q of a chunk sits at piece j ^ swz(q), so that 32 lanes read theirs without conflicts
    auto swz = [](int q) { return (uint32_t)(PPU == 8 ? q & 7 : (q >> 1) & 3); };
    const int pairs = (int)(chunks * 32 * PAIRS);
    for (int i0 = threadIdx.x; i0 < pairs; i0 += 4 * kGemvThreads) {
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int64_t s = i0 + k * kGemvThreads;
            v[k] = 0;
            if (2 * s < p.n) v[k] = ld_ordered_u32(reinterpret_cast<const uint32_t *>(p.x) + (p.x_order == RPTC_XORDER_K2_LEGACY ? k2_legacy_pair_32(s, p.n) : s));
        }
        if (CODE != RPTC_CODE_LUT && i0 == (int)threadIdx.x) lut_fill<CODE>(lut_tab, p.lut, p.L, p.S);      // under the loads above
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = i0 + k * kGemvThreads, q = i / PAIRS, w = i % PAIRS;
            if (i < pairs)
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(xs + (((uint32_t)(q * PPU) + ((uint32_t)(w >> 2) ^ swz(q & 31))) << 4) + 4u * (w & 3)), "r"(v[k]) : "memory");
        }
    }
    if (CODE != RPTC_CODE_LUT && (int)threadIdx.x >= pairs) lut_fill<CODE>(lut_tab, p.lut, p.L, p.S);
    const Lut<CODE> lut = lut_view<CODE>(lut_tab, p.L, p.S);
    __syncthreads();
    if (CODE == RPTC_CODE_LUT && !mbar_wait(s0, 0, p.status)) {
        cp_async_wait<0>();
        return;
    }
    uint32_t slot = 0;
    for (uint32_t group = 0; group < mine; group += kWholeRows) {
        const uint32_t rows = min((uint32_t)kWholeRows, mine - group);
#pragma unroll 1
        for (uint32_t chunk = ch0; chunk < ch1; ++chunk) {
            const int32_t u = (int32_t)(chunk * 32) + lane;
            const bool active = u < p.n_units;
            uint32_t xr[PAIRS];
#pragma unroll
            for (int j = 0; j < PPU; ++j) {
                const uint4 v = lds128(xs + (((uint32_t)(u * PPU) + ((uint32_t)j ^ swz(lane))) << 4));
                xr[4 * j] = v.x, xr[4 * j + 1] = v.y, xr[4 * j + 2] = v.z, xr[4 * j + 3] = v.w;
            }
#pragma unroll 1
            for (uint32_t i = 0; i < rows; ++i) {
                cp_async_wait<kUnitsAhead - 1>();
                const uint4 v = lds128(ring + slot * 512u);
                uint32_t halo = __shfl_up_sync(0xFFFFFFFFu, v.w, 1);
                if (lane == 0) {
                    halo = lds32(hist + 4u * slot);
                    if (p.quirk == RPTC_QUIRK_K2_LANE0_CARRY) halo = v.w;      // the reference kernels' lane-0 deviations
                    else if (p.quirk == RPTC_QUIRK_K1_LANE0_SEED && u > 0) halo >>= 16;
                }
                fetch();                                      // the words are in registers
                slot = (slot + 1) % kUnitsAhead;
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                __half2 hacc[4];
                decode_group<CODE, K>(w, halo, lut, [&](int pi, __half2 wp) {
                    const __half2 x2 = u32_as_half2(xr[pi]);
                    hacc[pi & 3] = pi < 4 ? __hmul2(wp, x2) : __hfma2(wp, x2, hacc[pi & 3]);
                });
                const float2 f2 = __half22float2(__hadd2(__hadd2(hacc[0], hacc[1]), __hadd2(hacc[2], hacc[3])));
                const float sum = active ? f2.x + f2.y : 0.f;
                sums[32 * i] = chunk == ch0 ? sum : sums[32 * i] + sum;
            }
        }
        for (uint32_t i = 0; i < rows; ++i) {
            float sum = ch0 < ch1 ? sums[32 * i] : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
            const uint32_t row = first + (group + i) * lanes_of_rows;
            if (lane == 0) {
                if (parts > 1) part_sums[(row - r0) * parts + part] = sum;
                // the reference accumulates in fp16: out = out + delta (inference_t.cu:170-171)
                else p.y[row] = p.accumulate ? __hadd(p.y[row], __float2half_rn(sum)) : __float2half_rn(sum);
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    if (parts > 1 && threadIdx.x < r1 - r0) {
        float sum = 0.f;
        for (uint32_t q = 0; q < parts; ++q) sum += part_sums[threadIdx.x * parts + q];
        __half *y = p.y + r0 + threadIdx.x;
        *y = p.accumulate ? __hadd(*y, __float2half_rn(sum)) : __float2half_rn(sum);
    }
    __syncthreads();
    if (threadIdx.x == 0) p.timer.end(gridDim.x);
}

static size_t whole_smem(int64_t n, const rptc_format &f) {
    const int64_t chunks = (n / (128 / f.K) + 31) / 32;
    return fixed_smem(f, kUnitsRing + kUnitsHist + kWholeSums + kWholeParts) + (size_t)chunks * 32 * (128 / f.K) * 2;
}
// In the legacy order every CTA gathers all activations, 4 bytes here and there, with a division each: from some number of columns on that is more
// than the product with a kernel behind it costs (calls, us, that / this): 4096 rows HASH, 4096 columns 30.3 / 22.7, 8192 34.7 / 34.2, 10240 35.7 / 35.8,
// 12288 36.2 / 37.2, 16384 38.2 / 40.4, 24576 42.8 / 51.6; 1024 rows, 10240 29.9 / 26.1, 16384 30.2 / 35.6.  In the natural order what fits into shared
// memory pays: 8192 x 24576 LITE 61.5 / 57.1, 2048 x 32768 table code 54.0 / 53.8.
bool gemv_whole_takes(int64_t n, int x_order, const rptc_format &f) {
    return (f.layout == RPTC_LAYOUT_ROWMAJOR || f.layout == RPTC_LAYOUT_CHUNKED) && (f.K == 2 || f.K == 4) && whole_smem(n, f) <= kMaxSmem &&
           (x_order == RPTC_XORDER_NATURAL || n <= 10240);
}
int gemv_whole(const void *codes, const void *lut, const void *x, void *y, int64_t m, int64_t n, int x_order, int accumulate, const rptc_format &f,
               const DeviceTimer &timer, cudaStream_t stream) {
    if (!gemv_whole_takes(n, x_order, f)) return RPTC_ERR_UNSUPPORTED;
    GemvWhole p = {};
    p.codes = static_cast<const uint4 *>(codes);
    p.lut = static_cast<const __half *>(lut);
    p.x = static_cast<const __half *>(x);
    p.m = m;
    p.n = n;
    p.n_units = (int32_t)(n / (128 / f.K));
    p.st = unit_strides(f.layout, m, p.n_units);
    p.L = f.L;
    p.S = f.S;
    p.quirk = f.quirk;
    p.x_order = x_order;
    p.status = device_status_word();
    if (!p.status) return RPTC_ERR_CUDA;
    p.y = static_cast<__half *>(y);
    p.accumulate = accumulate;
    p.timer = timer;
    const int64_t chunks = (p.n_units + 31) / 32;
    const size_t smem = whole_smem(n, f);
    const int ctas = (int)(m < num_sms() ? m : num_sms());
    // warps that share a row's chunks: as many as leave no warp without one (kWholeParts holds 16 x 4 sums)
    const int64_t rows = (m + ctas - 1) / ctas;
    p.parts = 1;
    while (2 * p.parts * rows <= kGemvWarps && 2 * p.parts <= chunks) p.parts *= 2;
    return with_code(f, [&](auto code, auto k) -> int {
        static SmemOptIn opted;
        auto kern = gemv_whole_kernel<code.value, k.value>;
        if (int e = allow_max_smem(kern, opted)) return e;
        return launch(kern, dim3((unsigned)ctas), dim3(kGemvThreads), smem, stream, p);
    });
}

}  // namespace rptc
