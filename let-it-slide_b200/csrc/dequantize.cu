// Symbols to weights without a packed stream in between (rptc.py:74-85), and symbols to the packed stream.
//
// dequantize: out[row][i] = alphabet[state_i] rounded to fp16, state_i = the last L bits of the row's 2-bit symbols up to i.
// A lane takes eight consecutive symbols (two 128-bit loads) and packs them into 16 bits; with the 16 bits of the lane to
// its left they are the windows of its eight states.  A warp walks along contiguous pieces of 256 symbols, so that the
// bits in front of a piece come from the piece before.  The alphabet sits in shared memory as fp16 (128 KiB at L = 16).
// Bound: HBM, 8 bytes per weight.  4096 x 4096, L = 16: 381 us with the symbols packed by tensor operations in 64-bit
// integers and decoded by the decompress kernel, 33 us a call as it is, 26 of them in the kernel (floor 20.6 us).
#include "common.cuh"

namespace rptc {

constexpr int kDeqThreads = 1024;

template <typename T>
__device__ __forceinline__ __half alphabet_entry(T v);
template <>
__device__ __forceinline__ __half alphabet_entry<float>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __half alphabet_entry<__half>(__half v) { return v; }
__device__ __forceinline__ void put(float *p, __half v) { *p = __half2float(v); }
__device__ __forceinline__ void put(__half *p, __half v) { *p = v; }
__device__ __forceinline__ void put8(float *p, const __half (&w)[8]) {
    float4 *q = reinterpret_cast<float4 *>(p);
    q[0] = make_float4(__half2float(w[0]), __half2float(w[1]), __half2float(w[2]), __half2float(w[3]));
    q[1] = make_float4(__half2float(w[4]), __half2float(w[5]), __half2float(w[6]), __half2float(w[7]));
}
__device__ __forceinline__ void put8(__half *p, const __half (&w)[8]) {
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = half2_as_u32(__halves2half2(w[2 * i], w[2 * i + 1]));
    *reinterpret_cast<uint4 *>(p) = make_uint4(o[0], o[1], o[2], o[3]);
}

// TABLE: the alphabet through shared memory; otherwise straight from L2 (few weights: not worth 128 KiB per SM).
// VEC: rows start on 16-byte boundaries of symbols and results.
template <typename T, bool TABLE, bool VEC>
__global__ void __launch_bounds__(kDeqThreads, 1) dequantize_kernel(const T *__restrict__ alphabet, const int32_t *__restrict__ symbols,
                                                                    T *__restrict__ out, int64_t rows, int length, int L) {
    extern __shared__ __align__(16) __half table[];
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const uint32_t mask = (1u << L) - 1u;
    pdl_wait_prior_grids();                             // launched with the calling thread's rptc_set_pdl setting
    if (TABLE) {
        constexpr int kBatch = 8;                       // loads in flight per thread
        for (int i0 = threadIdx.x; i0 < (1 << L); i0 += kBatch * kDeqThreads) {
            T v[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
                if (i0 + k * kDeqThreads < (1 << L)) v[k] = __ldg(alphabet + i0 + k * kDeqThreads);
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
                if (i0 + k * kDeqThreads < (1 << L)) table[i0 + k * kDeqThreads] = alphabet_entry<T>(v[k]);
        }
    }
    const int pieces = (length + 255) / 256;            // per row
    const int64_t total = rows * pieces;
    const int64_t p0 = total * warp / warps, p1 = total * (warp + 1) / warps;
    int64_t row = p0 / pieces;
    int piece = (int)(p0 - row * pieces);
    // the eight symbols of this lane in a piece, packed with the first one on top; past the row's end zeros
    auto load = [&](int64_t r, int pc, int4 &a, int4 &b) {
        const int i = pc * 256 + lane * 8;
        const int32_t *src = symbols + r * length + i;
        a = b = make_int4(0, 0, 0, 0);
        if (VEC && i + 8 <= length) {
            a = __ldcs(reinterpret_cast<const int4 *>(src));
            b = __ldcs(reinterpret_cast<const int4 *>(src) + 1);
        } else {
            if (i + 0 < length) a.x = src[0];
            if (i + 1 < length) a.y = src[1];
            if (i + 2 < length) a.z = src[2];
            if (i + 3 < length) a.w = src[3];
            if (i + 4 < length) b.x = src[4];
            if (i + 5 < length) b.y = src[5];
            if (i + 6 < length) b.z = src[6];
            if (i + 7 < length) b.w = src[7];
        }
    };
    int4 a, b;
    if (p0 < p1) load(row, piece, a, b);
    // the 16 bits in front of the first piece
    uint32_t before = 0;
    if (p0 < p1 && piece > 0) {
        const uint32_t q = lane < 8 ? (uint32_t)symbols[row * length + piece * 256 - 8 + lane] & 3u : 0u;
        before = __reduce_or_sync(0xFFFFFFFFu, lane < 8 ? q << (2 * (7 - lane)) : 0u);
    }
    if (TABLE) __syncthreads();
    for (int64_t p = p0; p < p1; ++p) {
        const uint32_t bits = ((uint32_t)a.x & 3u) << 14 | ((uint32_t)a.y & 3u) << 12 | ((uint32_t)a.z & 3u) << 10 | ((uint32_t)a.w & 3u) << 8 |
                              ((uint32_t)b.x & 3u) << 6 | ((uint32_t)b.y & 3u) << 4 | ((uint32_t)b.z & 3u) << 2 | ((uint32_t)b.w & 3u);
        const int64_t r = row;
        const int i = piece * 256 + lane * 8;
        if (++piece == pieces) piece = 0, ++row;
        if (p + 1 < p1) load(row, piece, a, b);         // the next piece is in flight under this one's lookups
        uint32_t left = __shfl_up_sync(0xFFFFFFFFu, bits, 1);
        if (lane == 0) left = before;
        before = piece == 0 ? 0u : __shfl_sync(0xFFFFFFFFu, bits, 31);      // a new row starts from state 0
        const uint32_t window = left << 16 | bits;
        __half w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t state = (window >> (2 * (7 - j))) & mask;
            w[j] = TABLE ? table[state] : alphabet_entry<T>(__ldg(alphabet + state));
        }
        T *dst = out + r * length + i;
        if (VEC && i + 8 <= length) {
            put8(dst, w);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (i + j < length) put(dst + j, w[j]);
        }
    }
}

// One thread per 32-bit word: 32 / bits consecutive symbols, first one on top, zeros past the row's end.
__global__ void __launch_bounds__(256) pack_symbols_kernel(const int32_t *__restrict__ symbols, uint32_t *__restrict__ words, int64_t total,
                                                           int64_t length, int64_t row_words, int bits) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const int64_t row = i / row_words, first = (i - row * row_words) * (32 / bits);
    const int32_t *src = symbols + row * length + first;
    uint32_t v = 0;
    if ((length & 3) == 0 && first + 32 / bits <= length) {
        for (int j = 0; j < 32 / bits; j += 4) {
            const int4 q = __ldcs(reinterpret_cast<const int4 *>(src + j));
            v = v << bits | (uint32_t)q.x;
            v = v << bits | (uint32_t)q.y;
            v = v << bits | (uint32_t)q.z;
            v = v << bits | (uint32_t)q.w;
        }
    } else {
        for (int j = 0; j < 32 / bits; ++j) v = v << bits | (first + j < length ? (uint32_t)src[j] : 0u);
    }
    words[i] = v;
}

template <typename T, bool VEC>
static int launch_dequantize(const T *alphabet, const int32_t *symbols, T *out, int64_t rows, int64_t length, int L, cudaStream_t s) {
    const int64_t pieces = rows * ((length + 255) / 256);
    // Shared memory costs each SM the whole alphabet; below 64 pieces per SM the lookups in L2 are the cheaper way.
    if (pieces >= 64 * (int64_t)num_sms()) {
        static SmemOptIn opted;
        auto kern = dequantize_kernel<T, true, VEC>;
        if (int e = allow_max_smem(kern, opted, 128 * 1024)) return e;
        return launch(kern, dim3(num_sms()), dim3(kDeqThreads), (size_t)2 << L, s, alphabet, symbols, out, rows, (int)length, L);
    }
    const int64_t ctas = (pieces + 3) / 4;                // four warps each
    const int64_t most = 16 * (int64_t)num_sms();
    return launch(dequantize_kernel<T, false, VEC>, dim3((unsigned)(ctas < most ? ctas : most)), dim3(128), 0, s, alphabet, symbols, out, rows,
                  (int)length, L);
}

}  // namespace rptc

using namespace rptc;

extern "C" int rptc_dequantize(const void *alphabet, const int32_t *symbols, void *out, int is_f32, int64_t rows, int64_t length, int L,
                               rptc_stream_t stream) {
    if (!alphabet || !symbols || !out) return RPTC_ERR_ARG;
    if (L < 3 || L > 16) return RPTC_ERR_ARG;
    if (rows <= 0 || length <= 0) return RPTC_ERR_SHAPE;
    if (length > (int64_t(1) << 30) || rows > (int64_t(1) << 40) / length) return RPTC_ERR_TOO_LARGE;
    if (int e = rptc_check_device()) return e;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool vec = length % (is_f32 ? 4 : 8) == 0 && ((reinterpret_cast<uintptr_t>(symbols) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    if (is_f32) {
        auto *a = static_cast<const float *>(alphabet);
        auto *o = static_cast<float *>(out);
        return vec ? launch_dequantize<float, true>(a, symbols, o, rows, length, L, s) : launch_dequantize<float, false>(a, symbols, o, rows, length, L, s);
    }
    auto *a = static_cast<const __half *>(alphabet);
    auto *o = static_cast<__half *>(out);
    return vec ? launch_dequantize<__half, true>(a, symbols, o, rows, length, L, s) : launch_dequantize<__half, false>(a, symbols, o, rows, length, L, s);
}

extern "C" int rptc_pack_symbols(const int32_t *symbols, void *words, int64_t rows, int64_t length, int64_t row_words, int bits, rptc_stream_t stream) {
    if (!symbols || !words) return RPTC_ERR_ARG;
    if (bits != 1 && bits != 2 && bits != 4 && bits != 8) return RPTC_ERR_ARG;
    if (rows <= 0 || length <= 0 || row_words <= 0 || row_words * (32 / bits) < length) return RPTC_ERR_SHAPE;
    if (rows > (int64_t(1) << 38) / row_words) return RPTC_ERR_TOO_LARGE;
    if (reinterpret_cast<uintptr_t>(symbols) & 15) return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    const int64_t total = rows * row_words;
    pack_symbols_kernel<<<(unsigned)((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(symbols, static_cast<uint32_t *>(words), total,
                                                                                                       length, row_words, bits);
    RPTC_CUDA(cudaGetLastError());
    return RPTC_OK;
}
