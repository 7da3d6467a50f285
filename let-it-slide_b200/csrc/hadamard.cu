// Block-diagonal randomized fast Hadamard transform along rows (the incoherence transform applied
// to activations before, and to outputs after, a quantised linear layer).
//
// One CTA transforms one block (256..4096 elements, or 256 elements holding several smaller blocks)
// of one row.  A thread holds eight consecutive elements in fp32 registers: butterfly strides 1,2,4
// run in registers, strides 8..128 as warp shuffles (__shfl_xor), and strides >= 256 through a
// shared-memory exchange.  Sign flips, the 1/sqrt(block) scale and the fp16 conversion are fused in.
#include "common.cuh"
#include "fwht.cuh"
#include "matmul.cuh"

#include <type_traits>

namespace rptc {

struct HadParams {
    const void *in;
    int64_t ld_in;
    __half *out;
    int64_t ld_out;
    const __half *signs;
    const __half *residual;     // optional fp16 [rows][ld_res], added to the result
    int64_t ld_res;
    int32_t block, chunk;       // chunk: columns per CTA (a block, or 2048 = eight warps of 256 when blocks are <= 256)
    int32_t in_is_f32, transpose, clear_in;
    float scale;
    int64_t n;
    float *clear;               // optional fp32 range that this launch zeroes (its own, not the input)
    int64_t clear_count;        // a multiple of 4
    int32_t late;               // the next kernel may start behind this one's wait only
};
struct HadSumsParams : HadParams {
    GemvSums sums;              // the input is a product's sums, to be added up
};

template <bool SUMS>
__global__ void __launch_bounds__(512) hadamard_kernel(const std::conditional_t<SUMS, HadSumsParams, HadParams> p) {
    __shared__ __align__(16) float ex[4096];
    if (!p.late) pdl_allow_next_grid();
    int n_sums = 0;
    if constexpr (SUMS) n_sums = p.sums.count((uint32_t)(blockIdx.x * p.chunk + 8 * threadIdx.x), blockIdx.y);      // eight columns lie in one tile
    pdl_wait_prior_grids();
    if (p.late) pdl_allow_next_grid();
    const int t = threadIdx.x;
    const int64_t row = blockIdx.y;
    if (p.clear) {
        float4 *z = reinterpret_cast<float4 *>(p.clear);
        const int64_t step = (int64_t)gridDim.x * gridDim.y * blockDim.x;
        for (int64_t i = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + t; 4 * i < p.clear_count; i += step)
            z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int64_t col = (int64_t)blockIdx.x * p.chunk + 8 * t;
    if (col >= p.n) return;     // only with blocks <= 256 (whole warps leave; such blocks need no CTA barrier)
    float v[8];
    if constexpr (SUMS) {
        constexpr int kAhead = 4;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = 0.f;
        const float *src = static_cast<const float *>(p.in) + row * p.ld_in + col;
        for (int s = 0; s < n_sums; s += kAhead, src += kAhead * p.sums.plane) {
            float w[kAhead][8] = {};
#pragma unroll
            for (int k = 0; k < kAhead; ++k)
                if (s + k < n_sums) load8_f32_cg(src + k * p.sums.plane, w[k]);
#pragma unroll
            for (int k = 0; k < kAhead; ++k)
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] += w[k][i];
        }
    } else if (p.in_is_f32) {
        load8_f32(const_cast<float *>(static_cast<const float *>(p.in)) + row * p.ld_in + col, v, p.clear_in != 0);
    } else load8_f16(static_cast<const __half *>(p.in) + row * p.ld_in + col, v);
    float sg[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) sg[i] = 1.f;
    if (p.signs) load8_f16(p.signs + col, sg);
    if (!p.transpose) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] *= sg[i];
    }
    fwht8(v, p.block, ex);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] *= p.transpose ? p.scale * sg[i] : p.scale;
    if (p.residual) {
        float r[8];
        load8_f16(p.residual + row * p.ld_res + col, r);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += r[i];
    }
    store8_f16(p.out + row * p.ld_out + col, v);
}

__global__ void __launch_bounds__(512) swiglu_hadamard_kernel(const SwigluParams p) {
    __shared__ __align__(16) float ex[4096];
    pdl_allow_next_grid();
    const int64_t row = blockIdx.y;
    const int64_t col = (int64_t)blockIdx.x * p.chunk + 8 * threadIdx.x;
    prefetch_swiglu_constants(p, col);
    pdl_wait_prior_grids();
    if (col >= p.n) return;     // only with blocks <= 256 (whole warps leave; such blocks need no CTA barrier)
    swiglu_chunk(p, row, col, ex, p.clear != 0, p.out + row * p.ld_out + col);
}

// ---- fused glue kernels of the decode step ------------------------------------------------------------
// They exist to shorten the chain of small dependent launches between two fused dequant-GEMVs.


__global__ void __launch_bounds__(256) finish_norm_hadamard_kernel(const FinishNormParams p) {
    __shared__ __align__(16) float ex[2048];
    __shared__ float red[36];
    pdl_allow_next_grid();
    pdl_wait_prior_grids();
    finish_norm_row(p, blockIdx.x, ex, red);
}

// Rows of 4096 or 8192: 256 threads per 4096 elements (64 registers: see kFewRegisterThreads).
template <int UNITS>
__global__ void __launch_bounds__(UNITS * kUnitThreads, UNITS == 1 ? 4 : 1) finish_norm_unit_kernel(const FinishNormParams p) {
    __shared__ __align__(16) float ex[UNITS][kUnitFloats];
    __shared__ float red[16];
    pdl_allow_next_grid();
    prefetch_norm_constants(p.signs_out, p.w_norm, p.signs_in, p.n, threadIdx.x, blockDim.x);
    pdl_wait_prior_grids();
    const int unit = threadIdx.x / kUnitThreads;
    finish_norm_unit(p, blockIdx.x, unit, ex[unit], red, 1 + unit, 3, true, true);
}

// Output side of the fused qkv layer, rotary embedding and KV-cache append in one pass:
// y = s_out * H(acc) * scale over blocks of `block` (>= 128) columns of [q heads | k heads | v heads];
// q is rotated and written to `q_out`, rotated k and v go to the caches at pos[row].  Head size 128,
// rotate-half pairing (i, i + 64): the partner of a thread's eight columns sits eight threads away.
struct QkvFinishParams {
    float *acc;
    int64_t ld_acc;
    const __half *signs_out;
    float scale;
    __half *q_out;               // fp16 [rows][ld_q], hq * 128 columns
    int64_t ld_q;
    __half *kcache, *vcache;     // [rows][max_pos][hkv][128]
    const int32_t *pos;
    int32_t hq, hkv, max_pos, block, chunk;
    RopeFreq freq;
    unsigned int *status;
};

__global__ void __launch_bounds__(512) qkv_finish_kernel(const QkvFinishParams p) {
    __shared__ __align__(16) float ex[4096];
    pdl_allow_next_grid();
    pdl_wait_prior_grids();
    const int t = threadIdx.x;
    const int64_t row = blockIdx.y;
    const int col = blockIdx.x * p.chunk + 8 * t;
    float v[8], sg[8];
    const uint4 raw_so = raw8_or_ones(p.signs_out ? p.signs_out + col : nullptr);
    const int ps = p.pos[row];
    // a position outside [0, max_pos) has no row in the cache: q is still finished, k and v are dropped, the host is told
    const bool in_cache = ps >= 0 && ps < p.max_pos;
    if (!in_cache && t == 0 && blockIdx.x == 0) atomicExch(p.status, kStatusPosition);
    load8_f32(p.acc + row * p.ld_acc + col, v, true);
    fwht8(v, p.block, ex);
    unpack8(raw_so, sg);
    const float sc = p.scale * hadamard_norm_dev(p.block);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __half2float(__float2half_rn(v[i] * sc * sg[i]));     // the layer's fp16 output
    const int head = col >> 7, idx = col & 127;
    if (head < p.hq + p.hkv) {
        const bool upper = idx >= 64;
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float partner = __shfl_xor_sync(0xFFFFFFFFu, v[i], 8);
            const int j = (idx & 63) + i;                       // frequency index
            float sn, cs;
            sincosf(ps * rope_inv_freq(p.freq, j), &sn, &cs);
            o[i] = upper ? v[i] * cs + partner * sn : v[i] * cs - partner * sn;
        }
        if (head < p.hq) store8_f16(p.q_out + row * p.ld_q + col, o);
        else if (in_cache) store8_f16(p.kcache + ((row * p.max_pos + ps) * p.hkv + (head - p.hq)) * 128 + idx, o);
    } else if (in_cache) {
        store8_f16(p.vcache + ((row * p.max_pos + ps) * p.hkv + (head - p.hq - p.hkv)) * 128 + idx, v);
    }
}

static float hadamard_norm(int block) {
    float norm = 1.f;
    for (int b = block; b > 1; b >>= 2) norm *= (b >= 4) ? 0.5f : 0.70710678118654752f;
    return norm;
}

}  // namespace rptc

using namespace rptc;

namespace rptc {
// many rows (prompt_ops.cu)
int hadamard_rows(const void *in, int in_is_f32, int64_t ld_in, __half *out, int64_t ld_out, const __half *signs, const __half *residual,
                  int64_t ld_res, int64_t rows, int64_t n, int block, int transpose, float scale, int clear_in, float *clear, int64_t clear_count,
                  cudaStream_t stream, bool late);
// Which inputs go to the kernels that walk down the rows.  Blocks above 256 columns: from 32 rows on (2048 x 4096: 13.4 us
// against 19.3; up to 128 rows both take 3.3).  Smaller blocks, with rows on 32-byte boundaries: from 2.5 million values on (512 x 11008:
// 7.6 us against 8.9, 512 x 4096: 4.5 against 4.2).
int swiglu_rows(const SwigluParams &p, int64_t rows, cudaStream_t stream);
static bool many_rows(int64_t rows, int64_t n, int block, const HadParams &p) {
    if (block > 256) return rows >= 32;
    auto on_32_bytes = [](const void *q, int64_t ld_bytes) { return ((reinterpret_cast<uintptr_t>(q) | (uintptr_t)ld_bytes) & 31) == 0; };
    return block >= 16 && rows * n >= (int64_t(5) << 19) && on_32_bytes(p.in, p.ld_in * (p.in_is_f32 ? 4 : 2)) && on_32_bytes(p.out, p.ld_out * 2) &&
           (!p.residual || on_32_bytes(p.residual, p.ld_res * 2));
}

// Blocks of 8 to 4096 columns, a power of two, in rows of whole warps of them.
int check_blocks(int64_t n, int block) {
    if (block < 8 || block > 4096 || (block & (block - 1))) return RPTC_ERR_ARG;
    return n <= 0 || n % (block < 256 ? 256 : block) ? RPTC_ERR_SHAPE : RPTC_OK;
}
int check_signs(const void *signs) { return reinterpret_cast<uintptr_t>(signs) & 15 ? RPTC_ERR_ALIGN : RPTC_OK; }      // read sixteen bytes at a time

int hadamard_and_clear(const void *in, int in_is_f32, int64_t ld_in, void *out, int64_t ld_out, const void *signs, const void *residual,
                       int64_t ld_res, int64_t rows, int64_t n, int block, int transpose, float scale, int clear_in, float *clear,
                       int64_t clear_count, cudaStream_t stream, bool late) {
    if (!in || !out) return RPTC_ERR_ARG;
    if (int e = check_blocks(n, block)) return e;
    if (rows <= 0 || ld_in < n || ld_out < n || (residual && ld_res < n)) return RPTC_ERR_SHAPE;
    if (rows > 65535) return RPTC_ERR_TOO_LARGE;
    const int chunk = block < 256 ? 256 : block;
    if ((reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(out) & 15) ||
        check_signs(signs) || (residual && (reinterpret_cast<uintptr_t>(residual) & 15)) ||
        (ld_in % 8) || (ld_out % 8) || (residual && (ld_res % 8)))
        return RPTC_ERR_ALIGN;
    if (clear_in && !in_is_f32) return RPTC_ERR_ARG;
    if (int e = rptc_check_device()) return e;
    HadParams p;
    p.in = in;
    p.ld_in = ld_in;
    p.out = static_cast<__half *>(out);
    p.ld_out = ld_out;
    p.signs = static_cast<const __half *>(signs);
    p.residual = static_cast<const __half *>(residual);
    p.ld_res = ld_res;
    p.block = block;
    p.chunk = chunk;
    p.in_is_f32 = in_is_f32;
    p.transpose = transpose;
    if (many_rows(rows, n, block, p))
        return hadamard_rows(in, in_is_f32, ld_in, static_cast<__half *>(out), ld_out, static_cast<const __half *>(signs),
                             static_cast<const __half *>(residual), ld_res, rows, n, block, transpose, scale, clear_in, clear, clear_count, stream, late);
    p.late = late;
    p.clear_in = clear_in;
    p.scale = scale * hadamard_norm(block);
    p.n = n;
    p.clear = clear_count > 0 ? clear : nullptr;
    p.clear_count = clear_count;
    if (block <= 256 && n > 256) {
        // small blocks: a warp per 256 columns, eight warps per CTA, so that many-row inputs do not become
        // hundreds of thousands of one-warp CTAs
        p.chunk = 2048;
        return launch(hadamard_kernel<false>, dim3((unsigned)((n + 2047) / 2048), (unsigned)rows), dim3(256), 0, stream, p);
    }
    return launch(hadamard_kernel<false>, dim3((unsigned)(n / chunk), (unsigned)rows), dim3(chunk / 8), 0, stream, p);
}

// Where adding up here is faster than in a kernel in front (layers, us: in front / here).  Not beyond 20 sums a value, whose loads this kernel's
// few threads take in turn: HASH, 9 and 31 rows, 1536 x 2048 (17 sums) 16.3 / 14.2 and 15.6 / 15.8, 1024 x 8192 (23) 15.5 / 16.4 and 16.5 / 17.7,
// 1024 x 2048 (32) 16.1 / 18.8 and 15.8 / 19.3.  Blocks above 256 up to 31 rows, behind which the transform that walks down the rows takes over, and
// below 4096, whose CTA has a whole row to add up: 2048 x 2048 15.4 / 13.3 and 16.1 / 13.3, 22016 x 4096 26.3 / 23.4 and 29.1 / 27.9, 4096 x 4096
// 15.9 / 16.5 and 17.3 / 17.9.  Smaller blocks: 11008 x 4096, 9 rows 18.0 / 17.4, 72 33.3 / 32.7; 3840 x 3584, 9 rows 16.2 / 13.2, 72 25.3 / 24.9; 96 rows
// of few values 28.2 / 28.8 there, of many 24320 x 2560 61.4 / 57.8, 12544 x 7168 46.2 / 44.6, 7936 x 1280 25.3 / 24.6.
bool hadamard_takes_sums(int64_t rows, int64_t n, int block, int64_t sums) {
    if (block > 256) return sums <= 20 && rows < 32 && block < 4096;
    return sums <= 20 && (rows <= 72 || (rows <= 96 && rows * n >= 700000)) && rows * n < (int64_t(5) << 19);
}
int hadamard_of_sums(const float *partial, int64_t ld, const GemvSums &sums, void *out, int64_t ld_out, const void *signs, int64_t rows, int64_t n,
                     int block, float scale, cudaStream_t stream) {
    if (int e = check_blocks(n, block)) return e;
    if (int e = check_signs(signs)) return e;
    const int chunk = block < 256 ? 256 : block;
    HadSumsParams p = {};
    p.in = partial;
    p.ld_in = ld;
    p.out = static_cast<__half *>(out);
    p.ld_out = ld_out;
    p.signs = static_cast<const __half *>(signs);
    p.block = block;
    p.chunk = block <= 256 && n > 256 ? 2048 : chunk;
    p.transpose = 1;
    p.scale = scale * hadamard_norm(block);
    p.n = n;
    p.sums = sums;
    return launch(hadamard_kernel<true>, dim3((unsigned)((n + p.chunk - 1) / p.chunk), (unsigned)rows), dim3(p.chunk / 8), 0, stream, p);
}
}  // namespace rptc

extern "C" int rptc_hadamard(const void *in, int in_is_f32, int64_t ld_in, void *out, int64_t ld_out, const void *signs,
                             const void *residual, int64_t ld_res, int64_t rows, int64_t n, int block, int transpose,
                             float scale, int clear_in, rptc_stream_t stream) {
    return hadamard_and_clear(in, in_is_f32, ld_in, out, ld_out, signs, residual, ld_res, rows, n, block, transpose, scale, clear_in, nullptr, 0,
                              static_cast<cudaStream_t>(stream), false);
}

static int swiglu_launch(float *acc, const void *in16, int64_t ld_in, void *out, int64_t ld_out, const void *signs_out,
                         const void *signs_in, int64_t rows, int64_t n, int block, float scale_out, float scale_in, int clear,
                         rptc_stream_t stream) {
    if ((!acc && !in16) || !out) return RPTC_ERR_ARG;
    if (block < 8 || block > 4096 || (block & (block - 1))) return RPTC_ERR_ARG;
    if (rows <= 0 || n <= 0 || (n % block) || ld_in < 2 * n || ld_out < n) return RPTC_ERR_SHAPE;
    if (rows > 65535) return RPTC_ERR_TOO_LARGE;
    const int chunk = block < 256 ? 256 : block;
    if (n % chunk) return RPTC_ERR_SHAPE;
    const void *in = acc ? static_cast<const void *>(acc) : in16;
    if ((reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(out) & 15) ||
        (signs_out && (reinterpret_cast<uintptr_t>(signs_out) & 15)) || (signs_in && (reinterpret_cast<uintptr_t>(signs_in) & 15)) ||
        (ld_in % (acc ? 4 : 8)) || (ld_out % 8) || (n % 8))
        return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    SwigluParams p;
    p.acc = acc;
    p.in16 = acc ? nullptr : static_cast<const __half *>(in16);
    p.ld_acc = ld_in;
    p.out = static_cast<__half *>(out);
    p.ld_out = ld_out;
    p.signs_out = static_cast<const __half *>(signs_out);
    p.signs_in = static_cast<const __half *>(signs_in);
    p.n = n;
    p.block = block;
    p.chunk = chunk;
    p.clear = acc ? clear : 0;
    p.scale_out = scale_out * hadamard_norm(block);
    p.scale_in = scale_in * hadamard_norm(block);
    // Prompts: from a full set of warps on (16 per SM, 512 columns of a row each), with rows on 32-byte boundaries.
    if (in16 && block == 256 && rows * n >= (int64_t)num_sms() * 16 * 512 && ld_in % 16 == 0 && ld_out % 16 == 0 &&
        ((reinterpret_cast<uintptr_t>(in16) | reinterpret_cast<uintptr_t>(out)) & 31) == 0)
        return swiglu_rows(p, rows, static_cast<cudaStream_t>(stream));
    if (block <= 256 && n > 256) {      // a warp per 256 columns, eight warps per CTA
        p.chunk = 2048;
        static SmemOptIn preferred;
        if (int e = prefer_shared_memory(swiglu_hadamard_kernel, preferred)) return e;
        return launch(swiglu_hadamard_kernel, dim3((unsigned)((n + 2047) / 2048), (unsigned)rows), dim3(256), 0,
                      static_cast<cudaStream_t>(stream), p);
    }
    return launch(swiglu_hadamard_kernel, dim3((unsigned)(n / chunk), (unsigned)rows), dim3(chunk / 8), 0,
                  static_cast<cudaStream_t>(stream), p);
}

extern "C" int rptc_swiglu_hadamard(float *acc, int64_t ld_acc, void *out, int64_t ld_out, const void *signs_out,
                                    const void *signs_in, int64_t rows, int64_t n, int block, float scale_out, float scale_in,
                                    int clear, rptc_stream_t stream) {
    if (!acc) return RPTC_ERR_ARG;
    return swiglu_launch(acc, nullptr, ld_acc, out, ld_out, signs_out, signs_in, rows, n, block, scale_out, scale_in, clear, stream);
}

extern "C" int rptc_swiglu_hadamard_f16(const void *gate_up, int64_t ld_in, void *out, int64_t ld_out, const void *signs_out,
                                        const void *signs_in, int64_t rows, int64_t n, int block, float scale_out, float scale_in,
                                        rptc_stream_t stream) {
    if (!gate_up) return RPTC_ERR_ARG;
    return swiglu_launch(nullptr, gate_up, ld_in, out, ld_out, signs_out, signs_in, rows, n, block, scale_out, scale_in, 0, stream);
}

extern "C" int rptc_finish_norm_hadamard(float *acc, int64_t ld_acc, const void *signs_out, float scale_out, void *h, int64_t ld_h,
                                         const void *w_norm, float eps, const void *signs_in, int transform_in, void *out,
                                         int64_t ld_out, int64_t rows, int64_t n, rptc_stream_t stream) {
    if (!h || !w_norm || !out) return RPTC_ERR_ARG;
    if (n < 256 || n > 8192 || (n & (n - 1))) return RPTC_ERR_UNSUPPORTED;      // one Hadamard block per row, or two of 4096
    if (rows <= 0 || ld_h < n || ld_out < n || (acc && ld_acc < n)) return RPTC_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(h) & 15) || (reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(w_norm) & 15) ||
        (acc && (reinterpret_cast<uintptr_t>(acc) & 15)) || (ld_h % 8) || (ld_out % 8) || (ld_acc % 4))
        return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    FinishNormParams p;
    p.acc = acc;
    p.ld_acc = ld_acc;
    p.signs_out = static_cast<const __half *>(signs_out);
    p.scale_out = scale_out;
    p.h = static_cast<__half *>(h);
    p.h_out = nullptr;
    p.ld_h = ld_h;
    p.w_norm = static_cast<const __half *>(w_norm);
    p.eps = eps;
    p.signs_in = static_cast<const __half *>(signs_in);
    p.transform_in = transform_in;
    p.out = static_cast<__half *>(out);
    p.ld_out = ld_out;
    p.n = (int32_t)n;
    p.block = (int32_t)(n > 4096 ? 4096 : n);
    static SmemOptIn one, two;
    if (n == 4096) {
        if (int e = prefer_shared_memory(finish_norm_unit_kernel<1>, one)) return e;
        return launch(finish_norm_unit_kernel<1>, dim3((unsigned)rows), dim3(kUnitThreads), 0, static_cast<cudaStream_t>(stream), p);
    }
    if (n == 8192) {
        if (int e = prefer_shared_memory(finish_norm_unit_kernel<2>, two)) return e;
        return launch(finish_norm_unit_kernel<2>, dim3((unsigned)rows), dim3(2 * kUnitThreads), 0, static_cast<cudaStream_t>(stream), p);
    }
    return launch(finish_norm_hadamard_kernel, dim3((unsigned)rows), dim3((unsigned)(n / 8)), 0, static_cast<cudaStream_t>(stream), p);
}

extern "C" int rptc_qkv_finish(float *acc, int64_t ld_acc, const void *signs_out, float scale, void *q_out, int64_t ld_q,
                               void *kcache, void *vcache, const int32_t *pos, int64_t rows, int hq, int hkv, int max_pos, int block,
                               float theta, rptc_stream_t stream) {
    if (!acc || !q_out || !kcache || !vcache || !pos) return RPTC_ERR_ARG;
    if (block < 128 || block > 4096 || (block & (block - 1))) return RPTC_ERR_ARG;
    const int64_t n = (int64_t)(hq + 2 * hkv) * 128;
    const int chunk = block < 256 ? 256 : block;
    if (rows <= 0 || rows > 65535 || hq <= 0 || hkv <= 0 || (n % chunk) || ld_acc < n || ld_q < (int64_t)hq * 128 || max_pos <= 0)
        return RPTC_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(acc) & 15) || (reinterpret_cast<uintptr_t>(q_out) & 15) || (reinterpret_cast<uintptr_t>(kcache) & 15) ||
        (reinterpret_cast<uintptr_t>(vcache) & 15) || (ld_acc % 4) || (ld_q % 8))
        return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    QkvFinishParams p;
    p.acc = acc;
    p.ld_acc = ld_acc;
    p.signs_out = static_cast<const __half *>(signs_out);
    p.scale = scale;
    p.q_out = static_cast<__half *>(q_out);
    p.ld_q = ld_q;
    p.kcache = static_cast<__half *>(kcache);
    p.vcache = static_cast<__half *>(vcache);
    p.pos = pos;
    p.hq = hq;
    p.hkv = hkv;
    p.max_pos = max_pos;
    p.block = block;
    p.chunk = chunk;
    p.freq = rope_freq(theta, 128);
    p.status = device_status_word();
    if (!p.status) return RPTC_ERR_CUDA;
    return launch(qkv_finish_kernel, dim3((unsigned)(n / chunk), (unsigned)rows), dim3(chunk / 8), 0, static_cast<cudaStream_t>(stream), p);
}
