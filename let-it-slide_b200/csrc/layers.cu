// Whole quantised layers as one call: the host side of a forward pass is then one foreign call and two allocations
// instead of a dozen tensor operations, and the kernels of the pass follow one another by programmatic dependent launch.
//   rptc_linear   y = s_out * H( scale * W_hat( H( s_in * x ) ) )              (RPTCLinear)
//   rptc_packed   y = scales_out * W_hat(scales_in * x) + biases_out * sum(x) + <biases_in, x> + bias, W_hat in banks of
//                 rows with an alphabet each                                    (FactorizedRPTCLinear)
// The layer of one token through a 4096 x 4096 matrix took 63 us, all of it host time (the GPU needs 9); the packed layer
// of one token with 32 banks 2150 us in about 160 launches.
#include <cuda_bf16.h>

#include "common.cuh"
#include "matmul.cuh"

#include <math.h>
#include <type_traits>

namespace rptc {

int check_format(const rptc_format *f);   // api.cu
// rptc_hadamard with a range to zero on the side (fp32, a multiple of 4 values, 16-byte aligned); `late`: the kernel behind may start
// behind this one's wait only.                                                                    hadamard.cu
int hadamard_and_clear(const void *in, int in_is_f32, int64_t ld_in, void *out, int64_t ld_out, const void *signs, const void *residual,
                       int64_t ld_res, int64_t rows, int64_t n, int block, int transpose, float scale, int clear_in, float *clear,
                       int64_t clear_count, cudaStream_t stream, bool late = false);
int check_blocks(int64_t n, int block);
int check_signs(const void *signs);
// out = signs * H(the product's sums) * scale over blocks, fp16 [rows][ld_out]; whether that is as fast as adding them up, `sums` a value at
// most, in a kernel in front
bool hadamard_takes_sums(int64_t rows, int64_t n, int block, int64_t sums);
int hadamard_of_sums(const float *partial, int64_t ld, const GemvSums &sums, void *out, int64_t ld_out, const void *signs, int64_t rows, int64_t n,
                     int block, float scale, cudaStream_t stream);

// Programmatic dependent launch within a call, whatever the calling thread's setting.  The products read codes and tables before they
// wait for the kernel in front.  They must not do so while an earlier kernel of the stream still writes a layer's buffers, so nothing
// behind a call's first kernel may start before all work in front of the call is done.  The first kernel of a call lets the next one
// start only behind its own wait, and where the tiled product follows it is launched without the attribute.  Measured, calls one
// after the other, an ordinary launch of the first kernel against this: packed layer of one token 32.8 and 31.3 us; transform in front
// of 4096 x 4096, 1 row 12.4 and 11.9, 32 rows 21.9 and 19.0; 4096 x 11008, 256 rows 43.0 and 41.0; tiled product, 4096 x 4096 with
// 2048 rows 83 and 87.6 (its CTAs wait for the early ones to leave).
struct PdlScope {
    const bool before = pdl_enabled();
    explicit PdlScope(bool on) { set(on); }
    ~PdlScope() { set(before); }
    void set(bool on) { rptc_set_pdl(on ? 1 : 0); }
};

// From here on a layer's product takes its sums in a fixed order: equal calls give equal bits (4096 x 4096 HASH, 16 rows: 17 us a layer
// against 12.6 with atomics; 4096 x 11008, 512 rows 57 against 51).  Fewer rows are a decode step's, whose sums meet in any order.
constexpr int64_t kOrderedRows = 9;
static int64_t round_up(int64_t bytes) { return (bytes + 255) / 256 * 256; }
// fp32 values that the product of a few rows needs beside its accumulator.
static int64_t partials(int64_t m, int64_t n, int64_t rows, const Banks &banks, const rptc_format &f) {
    return rows >= kOrderedRows && gemv_few_takes(m, n, rows, banks, f, nullptr, n) ? gemv_few_partials(m, n, rows, banks, f) : 0;
}

// ---- the packed layer's two ends ----
__device__ __forceinline__ float to_float(__half v) { return __half2float(v); }
__device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_float(float v) { return v; }
template <typename T>
__device__ __forceinline__ T from_float(float v);
template <>
__device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ float from_float<float>(float v) { return v; }

constexpr int kPackedThreads = 512;

// One CTA per token: xs = fp16(x * scales_in), sums[token] = (sum of x, <biases_in, x>), and the token's accumulator zeroed.
template <typename T>
__global__ void __launch_bounds__(kPackedThreads) packed_input_kernel(const T *__restrict__ x, const float *__restrict__ scales_in,
                                                                      const float *__restrict__ biases_in, __half *__restrict__ xs,
                                                                      float2 *__restrict__ sums, float *__restrict__ acc, int64_t acc_cols, int n) {
    __shared__ float2 red[kPackedThreads / 32];
    pdl_wait_prior_grids();
    pdl_allow_next_grid();                           // in this order: see PdlScope
    const int64_t token = blockIdx.x;
    const T *xr = x + token * n;
    __half *xo = xs + token * n;
    float s = 0.f, b = 0.f;
    for (int i = 4 * threadIdx.x; i < n; i += 4 * kPackedThreads) {      // n is a multiple of 64
        T v[4];
        if (sizeof(T) == 4) *reinterpret_cast<uint4 *>(v) = *reinterpret_cast<const uint4 *>(xr + i);
        else *reinterpret_cast<uint2 *>(v) = *reinterpret_cast<const uint2 *>(xr + i);
        const float4 sc = __ldg(reinterpret_cast<const float4 *>(scales_in + i)), bi = __ldg(reinterpret_cast<const float4 *>(biases_in + i));
        const float f[4] = {to_float(v[0]), to_float(v[1]), to_float(v[2]), to_float(v[3])};
        s += (f[0] + f[1]) + (f[2] + f[3]);
        b += (f[0] * bi.x + f[1] * bi.y) + (f[2] * bi.z + f[3] * bi.w);
        uint2 o;
        o.x = half2_as_u32(__floats2half2_rn(f[0] * sc.x, f[1] * sc.y));
        o.y = half2_as_u32(__floats2half2_rn(f[2] * sc.z, f[3] * sc.w));
        *reinterpret_cast<uint2 *>(xo + i) = o;
    }
    if (acc)
        for (int64_t i = 4 * threadIdx.x; i < acc_cols; i += 4 * kPackedThreads)
            *reinterpret_cast<float4 *>(acc + token * acc_cols + i) = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o), b += __shfl_xor_sync(0xFFFFFFFFu, b, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_float2(s, b);
    __syncthreads();
    if (threadIdx.x == 0) {
        s = b = 0.f;
#pragma unroll
        for (int i = 0; i < kPackedThreads / 32; ++i) s += red[i].x, b += red[i].y;
        sums[token] = make_float2(s, b);
    }
}

// y[token][row] from the product's fp32 accumulator (`acc`) or fp16 result (`prod`), whose columns are banks of
// `bank_cols` of which the first `bank_rows` hold rows of the layer.  SUMS: the accumulator is to be added up first.
template <typename T, bool SUMS>
__global__ void __launch_bounds__(256) packed_output_kernel(const float *__restrict__ acc, const __half *__restrict__ prod, int64_t ld,
                                                            const float2 *__restrict__ sums, const float *__restrict__ scales_out,
                                                            const float *__restrict__ biases_out, const float *__restrict__ bias,
                                                            T *__restrict__ y, int m, int bank_rows, int bank_cols, const GemvSums parts) {
    pdl_allow_next_grid();
    const int row = blockIdx.x * 256 + threadIdx.x;
    const int64_t token = blockIdx.y;
    float so = 0.f, bo = 0.f, bb = 0.f;
    if (row < m) so = __ldg(scales_out + row), bo = __ldg(biases_out + row), bb = bias ? __ldg(bias + row) : 0.f;
    const int n_parts = SUMS ? parts.count((uint32_t)(row % bank_rows), (uint32_t)token) : 1;
    pdl_wait_prior_grids();
    if (row >= m) return;
    const int bank = row / bank_rows, col = bank * bank_cols + row - bank * bank_rows;
    float v;
    float2 s;
    if (SUMS) {
        constexpr int kAhead = 4;                    // loads under way at a time
        const float *src = acc + token * ld + col;
        s = __ldcg(sums + token);
        v = 0.f;
        for (int i = 0; i < n_parts; i += kAhead) {
            float w[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; ++k) w[k] = i + k < n_parts ? __ldcg(src + (i + k) * parts.plane) : 0.f;
#pragma unroll
            for (int k = 0; k < kAhead; ++k) v += w[k];
        }
    } else {
        s = sums[token];
        v = acc ? acc[token * ld + col] : __half2float(prod[token * ld + col]);
    }
    y[token * m + row] = from_float<T>(v * so + s.x * bo + s.y + bb);
}

static rptc_format packed_format(const rptc_packed &l) { return {RPTC_CODE_LUT, 2, l.L, 0, RPTC_LAYOUT_TILED, RPTC_QUIRK_NONE}; }
static Banks packed_banks(const rptc_packed &l) {
    Banks banks;
    banks.banks = l.banks;
    banks.lut_stride = int64_t(1) << l.L;
    return banks;
}

// One or two tokens: no kernel in front of the product.
static bool packed_alone(const rptc_packed &l, int64_t tokens) {
    return gemv_alone_takes((int64_t)l.bank_blocks * 32, l.n, tokens, kNoTransform, packed_banks(l), packed_format(l));
}

template <typename T>
static int packed_forward(const rptc_packed &l, const void *x, void *y, int64_t tokens, char *ws, bool few, int64_t cols, cudaStream_t s) {
    PdlScope pdl(true);
    const rptc_format f = packed_format(l);
    const Banks banks = packed_banks(l);
    const int64_t stored = (int64_t)l.bank_blocks * 32, ld = (int64_t)l.banks * cols;
    float2 *sums = reinterpret_cast<float2 *>(ws);
    __half *xs = reinterpret_cast<__half *>(ws + round_up(tokens * 8));
    const bool alone = packed_alone(l, tokens);      // nothing in xs
    char *prod = reinterpret_cast<char *>(xs) + (alone ? 0 : round_up(tokens * l.n * 2));
    auto output = [&](const float *acc, const GemvSums &parts) {
        return launch(parts.per ? packed_output_kernel<T, true> : packed_output_kernel<T, false>, dim3((unsigned)((l.m + 255) / 256), (unsigned)tokens), dim3(256),
                      0, s, acc, acc ? nullptr : reinterpret_cast<const __half *>(prod), ld, sums, l.scales_out, l.biases_out, l.bias, static_cast<T *>(y),
                      (int)l.m, (int)(l.m / l.banks), (int)cols, parts);
    };
    if (alone) {
        GemvInput in = {};
        in.x = x;
        in.dtype = std::is_same<T, __half>::value ? 0 : std::is_same<T, float>::value ? 2 : 1;
        in.scales_in = l.scales_in;
        in.biases_in = l.biases_in;
        in.sums = sums;
        GemvSums parts;
        if (int e = gemv_alone(l.codes, l.alphabets, nullptr, in, reinterpret_cast<float *>(prod), stored, l.n, tokens, banks, f, s, &parts)) return e;
        return output(reinterpret_cast<const float *>(prod), parts);
    }
    float *partial = few && partials(stored, l.n, tokens, banks, f) ? reinterpret_cast<float *>(prod + round_up(tokens * ld * 4)) : nullptr;
    if (int e = launch(packed_input_kernel<T>, dim3((unsigned)tokens), dim3(kPackedThreads), 0, s, static_cast<const T *>(x), l.scales_in, l.biases_in,
                       xs, sums, few && !partial ? reinterpret_cast<float *>(prod) : nullptr, ld, (int)l.n))
        return e;
    // The output side adds the sums up by itself, a value per thread, where there are few of them (in front / there, us): 1792 x 1536 in 32 banks, 9
    // tokens 15.8 / 13.2, 96 20.6 / 19.4; 5504 x 1088 in 16, 48 tokens (264 thousand values) 15.9 / 15.0; 7296 x 7104 in 16, 48 (350) 41.7 / 40.4;
    // 8832 x 4288 in 8, 48 (424) 32.6 / 32.5; 10240 x 576 in 16, 48 (492) 16.3 / 16.7; 96 tokens: 3072 x 512 in 16 (295) 18.7 / 18.3, 3712 x 832 in 16
    // (356) 19.8 / 20.2, 4480 x 640 in 8 (430) 20.2 / 20.9.
    if (partial && tokens <= kFewOwnTokens && tokens * l.m <= (tokens <= 48 ? 420 : 310) << 10) {
        GemvSums parts;
        if (int e = gemv_few(l.codes, l.alphabets, nullptr, xs, l.n, nullptr, ld, stored, l.n, tokens, banks, f, s, true, partial, &parts)) return e;
        return output(partial, parts);
    }
    const int e = few ? gemv_banked(l.codes, l.alphabets, xs, l.n, reinterpret_cast<float *>(prod), ld, stored, l.n, tokens, banks, f, s, tokens >= kOrderedRows, partial)
                      : gemm_banked(l.codes, l.alphabets, nullptr, xs, l.n, prod, ld, stored, l.n, tokens, banks, f, s);
    if (e) return e;
    return output(few ? reinterpret_cast<const float *>(prod) : nullptr, GemvSums{});
}

// Which product a packed layer takes, and how many columns it gives per bank.
static bool packed_plan(const rptc_packed &l, int64_t tokens, int64_t &cols) {
    const rptc_format f = packed_format(l);
    const Banks banks = packed_banks(l);
    const bool few = tokens <= kFewOwnTokens || gemv_few_takes((int64_t)l.bank_blocks * 32, l.n, tokens, banks, f, nullptr, l.n);
    cols = few ? (int64_t)l.bank_blocks * 32 : gemm_bank_columns((int64_t)l.bank_blocks * 32, l.n, tokens, banks, f);
    return few;
}

static int check_packed(const rptc_packed *l, int64_t tokens) {
    if (!l) return RPTC_ERR_ARG;
    if (l->L < 3 || l->L > 16) return RPTC_ERR_ARG;
    if (l->m <= 0 || l->n <= 0 || tokens <= 0 || l->banks <= 0 || l->m % l->banks || l->n % 64 || l->bank_blocks <= 0 ||
        (int64_t)l->bank_blocks * 32 < l->m / l->banks)
        return RPTC_ERR_SHAPE;
    if (l->m > (1 << 30) || l->n > (1 << 30) || tokens > 65535) return RPTC_ERR_TOO_LARGE;
    return RPTC_OK;
}

}  // namespace rptc

using namespace rptc;

extern "C" int64_t rptc_packed_workspace_bytes(const rptc_packed *l, int64_t tokens) {
    if (check_packed(l, tokens)) return -1;
    int64_t cols;
    const bool few = packed_plan(*l, tokens, cols);
    if (packed_alone(*l, tokens))
        return round_up(tokens * 8) + 4 * gemv_alone_partials((int64_t)l->bank_blocks * 32, l->n, tokens, packed_banks(*l), packed_format(*l));
    const int64_t partial = few ? partials((int64_t)l->bank_blocks * 32, l->n, tokens, packed_banks(*l), packed_format(*l)) : 0;
    return round_up(tokens * 8) + round_up(tokens * l->n * 2) + round_up(tokens * l->banks * cols * (few ? 4 : 2)) + partial * 4;
}

extern "C" int rptc_packed_forward(const rptc_packed *l, const void *x, int dtype, void *y, int64_t tokens, void *workspace,
                                   int64_t workspace_bytes, rptc_stream_t stream) {
    if (int e = check_packed(l, tokens)) return e;
    if (!x || !y || !workspace || !l->codes || !l->alphabets || !l->biases_out || !l->biases_in || !l->scales_out || !l->scales_in) return RPTC_ERR_ARG;
    if (workspace_bytes < rptc_packed_workspace_bytes(l, tokens)) return RPTC_ERR_TOO_LARGE;
    auto misaligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
    if (misaligned(l->codes) || misaligned(l->alphabets) || misaligned(x) || misaligned(l->scales_in) || misaligned(l->biases_in) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255))
        return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    int64_t cols;
    const bool few = packed_plan(*l, tokens, cols);
    if (!few && !cols) return RPTC_ERR_UNSUPPORTED;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char *ws = static_cast<char *>(workspace);
    switch (dtype) {
        case 0: return packed_forward<__half>(*l, x, y, tokens, ws, few, cols, s);
        case 1: return packed_forward<__nv_bfloat16>(*l, x, y, tokens, ws, few, cols, s);
        case 2: return packed_forward<float>(*l, x, y, tokens, ws, few, cols, s);
    }
    return RPTC_ERR_ARG;
}

// ---- the incoherent layer ----
constexpr int64_t kFewRows = 65535;      // the transforms and the readers of an accumulator have a grid row per activation row
// Whether the product goes through the fp32 accumulator: one or two rows, whatever the kernel for a few rows takes, and
// up to 64 rows of a reduction that is not whole steps of 64 columns.  The others take the tiled product, whose last tile may be partial.
static bool linear_few(const rptc_linear &l, int64_t rows) {
    if (rows > kFewRows) return false;
    return rows <= 2 || gemv_few_takes(l.m, l.n, rows, Banks(), l.fmt, nullptr, l.n) || (rows <= 64 && l.n % 64);
}

// A single row: no kernel in front of the product.
static bool linear_alone(const rptc_linear &l, int64_t rows) {
    return l.signs_in && rows == 1 && gemv_alone_takes(l.m, l.n, rows, l.block_in, Banks(), l.fmt);
}

extern "C" int64_t rptc_linear_workspace_bytes(const rptc_linear *l, int64_t rows) {
    if (!l || rows <= 0) return -1;
    if (linear_alone(*l, rows)) return 4 * gemv_alone_partials(l->m, l->n, rows, Banks(), l->fmt);
    const int64_t xt = l->signs_in ? round_up(rows * l->n * 2) : 0;
    return xt + (linear_few(*l, rows) ? round_up(rows * l->m * 4) + 4 * partials(l->m, l->n, rows, Banks(), l->fmt) : 0);
}

extern "C" int rptc_linear_forward(const rptc_linear *l, const void *x, void *y, int64_t rows, void *workspace, int64_t workspace_bytes,
                                   rptc_stream_t stream) {
    if (!l || !x || !y || !l->codes || !l->lut) return RPTC_ERR_ARG;
    if (int e = check_format(&l->fmt)) return e;
    if (l->fmt.layout != RPTC_LAYOUT_TILED || l->fmt.quirk != RPTC_QUIRK_NONE || (l->fmt.K != 2 && l->fmt.K != 4)) return RPTC_ERR_UNSUPPORTED;
    if (!l->signs_in != !l->signs_out) return RPTC_ERR_ARG;
    if (l->m <= 0 || l->n <= 0 || rows <= 0 || (l->m % 32) || (l->n % (128 / l->fmt.K)) || (l->m % 4)) return RPTC_ERR_SHAPE;
    if (rows > (l->signs_in ? kFewRows : int64_t(1) << 24)) return RPTC_ERR_TOO_LARGE;
    const bool few = linear_few(*l, rows);
    if (!few && (l->n % 64)) return RPTC_ERR_SHAPE;
    if (l->m > (int64_t(1) << 30) || l->n > (int64_t(1) << 30) || (l->m / 32) * (l->n / (128 / l->fmt.K)) >= (int64_t(1) << 31))
        return RPTC_ERR_TOO_LARGE;
    const int64_t need = rptc_linear_workspace_bytes(l, rows);
    if (need && (!workspace || workspace_bytes < need)) return RPTC_ERR_TOO_LARGE;
    auto misaligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
    if (misaligned(l->codes) || misaligned(l->lut) || misaligned(x) || misaligned(y) || misaligned(workspace) || (l->n % 8) || (l->m % 8))
        return RPTC_ERR_ALIGN;
    if (l->signs_in) {
        if (int e = check_blocks(l->n, l->block_in)) return e;
        if (int e = check_blocks(l->m, l->block_out)) return e;
    }
    if (int e = check_signs(l->signs_in)) return e;
    if (int e = check_signs(l->signs_out)) return e;
    if (int e = rptc_check_device()) return e;
    PdlScope pdl(l->signs_in && few);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char *ws = static_cast<char *>(workspace);
    const int64_t m = l->m, n = l->n;
    if (linear_alone(*l, rows)) {
        pdl.set(true);
        GemvInput in = {};
        in.x = x;
        in.signs = static_cast<const __half *>(l->signs_in);
        in.block = l->block_in;
        in.norm = 1.f / sqrtf((float)l->block_in);
        GemvSums sums;
        float *partial = static_cast<float *>(workspace);
        if (int e = gemv_alone(l->codes, l->lut, l->carry_in, in, partial, m, n, rows, Banks(), l->fmt, s, &sums)) return e;
        return hadamard_of_sums(partial, m, sums, y, m, l->signs_out, rows, m, l->block_out, l->scale, s);
    }
    const void *xt = x;
    float *acc = few ? reinterpret_cast<float *>(ws + (l->signs_in ? round_up(rows * n * 2) : 0)) : nullptr;
    float *partial = few && partials(m, n, rows, Banks(), l->fmt) ? acc + round_up(rows * m * 4) / 4 : nullptr;
    const int64_t clear = few && !partial ? rows * m : 0;
    if (l->signs_in) {
        if (int e = hadamard_and_clear(x, 0, n, ws, n, l->signs_in, nullptr, 0, rows, n, l->block_in, 0, 1.f, 0, acc, clear, s, true)) return e;
        pdl.set(true);
        xt = ws;
    } else if (clear) {
        RPTC_CUDA(cudaMemsetAsync(acc, 0, (size_t)(rows * m) * 4, s));
    }
    if (few) {
        if (rows < kOrderedRows || !gemv_few_takes(m, n, rows, Banks(), l->fmt, xt, n)) {
            if (int e = rptc_gemv(l->codes, l->lut, l->carry_in, xt, n, acc, m, m, n, (int)rows, RPTC_XORDER_NATURAL, &l->fmt, stream)) return e;
        } else {
            GemvSums parts;
            const bool added_up = partial && l->signs_out && hadamard_takes_sums(rows, m, l->block_out, partials(m, n, rows, Banks(), l->fmt) / (rows * m));
            if (int e = gemv_few(l->codes, l->lut, l->carry_in, xt, n, acc, m, m, n, rows, Banks(), l->fmt, s, true, partial, added_up ? &parts : nullptr)) return e;
            pdl.set(true);
            if (added_up) return hadamard_of_sums(partial, m, parts, y, m, l->signs_out, rows, m, l->block_out, l->scale, s);
        }
        pdl.set(true);
        if (l->signs_out)
            return hadamard_and_clear(acc, 1, m, y, m, l->signs_out, nullptr, 0, rows, m, l->block_out, 1, l->scale, 0, nullptr, 0, s);
        // without transforms, beyond 64 rows, the scale is left to the caller whichever product was taken
        return rptc_gemv_finish(acc, m, y, m, m, (int)rows, rows > 64 ? 1.f : l->scale, 0, 0, stream);
    }
    if (int e = gemm_banked(l->codes, l->lut, l->carry_in, xt, n, y, m, m, n, rows, Banks(), l->fmt, s)) return e;
    if (l->signs_out) return hadamard_and_clear(y, 0, m, y, m, l->signs_out, nullptr, 0, rows, m, l->block_out, 1, l->scale, 0, nullptr, 0, s);
    return RPTC_OK;
}
