// The transforms and the glue of a prompt's forward pass: many rows at once, fp16 in and out, fp32 inside.
//   hadamard_rows     rptc_hadamard for many rows
//   norm_rows         h += s_out * H(y) * scale;  xn = rmsnorm(h) * w;  out = H(s_in * xn)        (rptc_prompt_norm)
//   qkv_rows          output transform of the fused qkv layer, rotary embedding, cache writes     (rptc_prompt_qkv)
// Bound: HBM / L2 (each input read once, each output written once).  A warp or CTA keeps its columns and walks down the rows,
// so that signs and weights of its columns stay in registers.
#include "common.cuh"
#include "fwht.cuh"
#include "prompt_fwht.cuh"

namespace rptc {

static float norm_of(int block) {
    float norm = 1.f;
    for (int b = block; b > 1; b >>= 2) norm *= (b >= 4) ? 0.5f : 0.70710678118654752f;
    return norm;
}
static int log2_of(int block) {
    int b = 0;
    while ((1 << b) < block) ++b;
    return b;
}

struct HadRowsParams {
    const void *in;
    int64_t ld_in;
    __half *out;
    int64_t ld_out;
    const __half *signs, *residual;
    int64_t ld_res, rows, n;
    int32_t block_bits, transpose, clear_in;
    float scale;
    float *clear;
    int64_t clear_count;
    int32_t late;                    // the next kernel may start behind this one's wait only
};

__device__ __forceinline__ uint32_t ldcg_u32(const void *p) { return __ldcg(static_cast<const uint32_t *>(p)); }

// Blocks above 256: one segment of a row per CTA of 128 threads, results in the layout of the pairs.
template <bool IN_F32>
__global__ void __launch_bounds__(128, 4) hadamard_rows_kernel(const HadRowsParams p) {
    constexpr int kSeg = 4096;
    constexpr uint32_t kOnes = 0x3C003C00u;
    __shared__ __align__(16) float buf[kCtaSegFloats];
    const SegThread th;
    const int segs = (int)((p.n + kSeg - 1) / kSeg);
    const int64_t worker = blockIdx.x, workers = (int64_t)gridDim.x / segs * segs;
    if (!p.late) pdl_allow_next_grid();
    pdl_wait_prior_grids();
    if (p.late) pdl_allow_next_grid();
    if (p.clear) {
        float4 *z = reinterpret_cast<float4 *>(p.clear);
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; 4 * i < p.clear_count; i += (int64_t)gridDim.x * blockDim.x)
            z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (worker >= workers) return;
    const int64_t col0 = (worker % segs) * kSeg;
    // the columns of pair of values i (v[2 i], v[2 i + 1]) as loaded and as stored
    auto col_in = [&](int i) { return col0 + th.piece(i >> 2) + 2 * (i & 3); };
    auto col_out = [&](int i) { return col0 + th.pair(i); };
    uint32_t sg[16];                                         // signs of the columns where they apply, two to a register
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int64_t c = p.transpose ? col_out(i) : col_in(i);
        sg[i] = (p.signs && c < p.n) ? __ldg(reinterpret_cast<const uint32_t *>(p.signs + c)) : kOnes;
    }
    for (int64_t row = worker / segs; row < p.rows; row += workers / segs) {
        float v[32];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t c = col0 + th.piece(j);
            if (IN_F32) {
                float *src = const_cast<float *>(static_cast<const float *>(p.in)) + row * p.ld_in + c;
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
                if (c < p.n) {
                    a = __ldcg(reinterpret_cast<const float4 *>(src)), b = __ldcg(reinterpret_cast<const float4 *>(src) + 1);
                    if (p.clear_in) reinterpret_cast<float4 *>(src)[0] = reinterpret_cast<float4 *>(src)[1] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                v[8 * j] = a.x, v[8 * j + 1] = a.y, v[8 * j + 2] = a.z, v[8 * j + 3] = a.w;
                v[8 * j + 4] = b.x, v[8 * j + 5] = b.y, v[8 * j + 6] = b.z, v[8 * j + 7] = b.w;
            } else {
                const uint4 raw = c < p.n ? __ldcg(reinterpret_cast<const uint4 *>(static_cast<const __half *>(p.in) + row * p.ld_in + c)) : make_uint4(0u, 0u, 0u, 0u);
                unpack8_at(raw, v + 8 * j);
            }
        }
        uint32_t res[16];
        if (p.residual) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (col_out(i) < p.n) res[i] = ldcg_u32(p.residual + row * p.ld_res + col_out(i));
        }
        if (!p.transpose) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float2 s = __half22float2(u32_as_half2(sg[i]));
                v[2 * i] *= s.x, v[2 * i + 1] *= s.y;
            }
        }
        piece_stages(v);
        th.put_pieces(buf, v);
        th.sync();
        th.get_columns(buf, v);
        column_stages(v, p.block_bits);
        th.put_columns(buf, v);
        th.sync();
        th.get_pairs(buf, v);
        far_stages(v, p.block_bits);
        uint32_t o[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float2 s = make_float2(p.scale, p.scale);
            if (p.transpose) {
                const float2 f = __half22float2(u32_as_half2(sg[i]));
                s.x *= f.x, s.y *= f.y;
            }
            float2 w = make_float2(__fmul_rn(v[2 * i], s.x), __fmul_rn(v[2 * i + 1], s.y));
            if (p.residual) {
                const float2 r = __half22float2(u32_as_half2(res[i]));
                w.x = __fadd_rn(w.x, r.x), w.y = __fadd_rn(w.y, r.y);
            }
            o[i] = half2_as_u32(__floats2half2_rn(w.x, w.y));
        }
        __half *dst = p.out + row * p.ld_out;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (col_out(i) < p.n) *reinterpret_cast<uint32_t *>(dst + col_out(i)) = o[i];
        th.sync();                                           // the buffer is free for the next row
    }
}

// ---- blocks of at most 256: sixteen values per thread ------------------------------------------------------------------
// A warp takes 512 columns (a half-warp 256, thread t of 16) and walks down the rows, the next row's values under way:
//   near   elements 16 t .. 16 t + 15: the stages of bits 0-3, loads and stores of 32 bytes
//   far    elements t + 16 k: the stages of bits 4-7
// with an exchange through shared memory in between, a fifth of the cost of a shuffle per value and stage.  The four 16-byte pieces
// of sixteen values sit at piece ^ (t >> 1): no bank conflicts in either layout.  Bound: HBM.  2048 x 11008 with 32 values per thread and no
// row ahead 26.8 us, with eight values and shuffles 31.5, as it is 20.1 (fp32 input 26.5); four CTAs per SM spill registers: 25.3.
constexpr int kHalfFloats = 256 + 16, kPairFloats = 2 * kHalfFloats;
struct Near16 {
    float *row;
    int x;
    __device__ __forceinline__ Near16(float *half, int t) : row(half + 16 * t), x((t >> 1) & 3) {}
    __device__ __forceinline__ void put(const float (&v)[16]) const {
#pragma unroll
        for (int c = 0; c < 4; ++c) *reinterpret_cast<float4 *>(row + 4 * (c ^ x)) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    }
    __device__ __forceinline__ void get(float (&v)[16]) const {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float4 f = *reinterpret_cast<const float4 *>(row + 4 * (c ^ x));
            v[4 * c] = f.x, v[4 * c + 1] = f.y, v[4 * c + 2] = f.z, v[4 * c + 3] = f.w;
        }
    }
};
struct Far16 {
    float *at[4];
    __device__ __forceinline__ Far16(float *half, int t) {
#pragma unroll
        for (int q = 0; q < 4; ++q) at[q] = half + 4 * ((t >> 2) ^ q) + (t & 3);
    }
    __device__ __forceinline__ void put(const float (&v)[16]) const {
#pragma unroll
        for (int k = 0; k < 16; ++k) at[(k >> 1) & 3][16 * k] = v[k];
    }
    __device__ __forceinline__ void get(float (&v)[16]) const {
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = at[(k >> 1) & 3][16 * k];
    }
};
__device__ __forceinline__ void ld_32_bytes(const void *p, uint32_t (&r)[8]) {
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "l"(p));
}
__device__ __forceinline__ void st_32_bytes(void *p, const uint32_t (&r)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
                 "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void unpack_pairs(const uint32_t (&r)[8], float (&v)[16]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 f = __half22float2(u32_as_half2(r[i]));
        v[2 * i] = f.x, v[2 * i + 1] = f.y;
    }
}

// Bits 4-7 of blocks of 32 to 256: v[k] is element bits 4-7 = k.
__device__ __forceinline__ void far_stages16(float (&v)[16], int block_bits) {
    if (block_bits == 8) return stages16(v);
#pragma unroll
    for (int h = 1; h < 8; h <<= 1)
        if (block_bits > 4 + (h == 1 ? 0 : h == 2 ? 1 : 2)) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if ((i & h) == 0) {
                    const float a = v[i], b = v[i + h];
                    v[i] = a + b;
                    v[i + h] = a - b;
                }
        }
}
template <bool IN_F32>
__global__ void __launch_bounds__(256, IN_F32 ? 2 : 3) hadamard_half_rows_kernel(const HadRowsParams p) {
    __shared__ __align__(16) float smem[8 * kPairFloats];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & 15, half = lane >> 4;
    float *buf = smem + warp * kPairFloats + half * kHalfFloats;
    const Near16 near(buf, t);
    const Far16 far(buf, t);
    const int segs = (int)((p.n + 511) / 512);
    const int64_t worker = (int64_t)blockIdx.x * 8 + warp, workers = (int64_t)gridDim.x * 8 / segs * segs;
    if (!p.late) pdl_allow_next_grid();
    const int64_t col = (worker % segs) * 512 + 256 * half + 16 * t;
    const bool active = col < p.n;                           // a last segment of 256 columns leaves half of the warp without
    uint32_t sg[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) sg[i] = p.signs && active ? __ldg(reinterpret_cast<const uint32_t *>(p.signs + col) + i) : 0x3C003C00u;
    pdl_wait_prior_grids();
    if (p.late) pdl_allow_next_grid();
    if (p.clear) {
        float4 *z = reinterpret_cast<float4 *>(p.clear);
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; 4 * i < p.clear_count; i += (int64_t)gridDim.x * blockDim.x)
            z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (worker >= workers) return;
    const int64_t step = workers / segs;
    uint32_t raw[IN_F32 ? 2 : 1][8] = {};
    auto fetch = [&](int64_t row) {
        if (!active) return;
        if (IN_F32) {
            float *src = const_cast<float *>(static_cast<const float *>(p.in)) + row * p.ld_in + col;
            ld_32_bytes(src, raw[0]);
            ld_32_bytes(src + 8, raw[IN_F32 ? 1 : 0]);
            if (p.clear_in) {
                const uint32_t zero[8] = {};
                st_32_bytes(src, zero);
                st_32_bytes(src + 8, zero);
            }
        } else {
            ld_32_bytes(static_cast<const __half *>(p.in) + row * p.ld_in + col, raw[0]);
        }
    };
    int64_t row = worker / segs;
    if (row < p.rows) fetch(row);
    for (; row < p.rows; row += step) {
        float v[16], s[16];
        if (IN_F32) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(raw[IN_F32 ? i >> 3 : 0][i & 7]);
        } else {
            unpack_pairs(raw[0], v);
        }
        uint32_t res[8];
        if (p.residual && active) ld_32_bytes(p.residual + row * p.ld_res + col, res);
        if (row + step < p.rows) fetch(row + step);
        unpack_pairs(sg, s);
        if (!p.transpose) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] *= s[i];
        }
        stages16(v);
        if (p.block_bits > 4) {
            near.put(v);                                     // where this thread has read
            __syncwarp();
            far.get(v);
            far_stages16(v, p.block_bits);
            far.put(v);
            __syncwarp();
            near.get(v);
        }
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float2 f = make_float2(p.scale, p.scale);
            if (p.transpose) f.x *= s[2 * i], f.y *= s[2 * i + 1];
            float2 w = make_float2(__fmul_rn(v[2 * i], f.x), __fmul_rn(v[2 * i + 1], f.y));
            if (p.residual) {
                const float2 r = __half22float2(u32_as_half2(res[i]));
                w.x = __fadd_rn(w.x, r.x), w.y = __fadd_rn(w.y, r.y);
            }
            o[i] = half2_as_u32(__floats2half2_rn(w.x, w.y));
        }
        if (active) st_32_bytes(p.out + row * p.ld_out + col, o);
    }
}

// Grid of a kernel whose CTAs walk down the rows: as many as are resident at once, no more than there is work for.
static unsigned rows_grid(int64_t rows, int64_t segs, int units, int resident) {
    const int64_t want = (rows * segs + units - 1) / units, most = (int64_t)num_sms() * resident;
    const int64_t least = (segs + units - 1) / units;        // every segment needs a worker
    const int64_t g = want < most ? want : most;
    return (unsigned)(g > least ? g : least);
}

int hadamard_rows(const void *in, int in_is_f32, int64_t ld_in, __half *out, int64_t ld_out, const __half *signs, const __half *residual,
                  int64_t ld_res, int64_t rows, int64_t n, int block, int transpose, float scale, int clear_in, float *clear, int64_t clear_count,
                  cudaStream_t stream, bool late) {
    HadRowsParams p;
    p.in = in;
    p.ld_in = ld_in;
    p.out = out;
    p.ld_out = ld_out;
    p.signs = signs;
    p.residual = residual;
    p.ld_res = ld_res;
    p.rows = rows;
    p.n = n;
    p.block_bits = log2_of(block);
    p.transpose = transpose;
    p.clear_in = clear_in;
    p.scale = scale * norm_of(block);
    p.clear = clear_count > 0 ? clear : nullptr;
    p.clear_count = clear_count;
    p.late = late;
    if (block <= 256) {
        const dim3 grid(rows_grid(rows, (n + 511) / 512, 8, in_is_f32 ? 2 : 3));
        return in_is_f32 ? launch(hadamard_half_rows_kernel<true>, grid, dim3(256), 0, stream, p)
                         : launch(hadamard_half_rows_kernel<false>, grid, dim3(256), 0, stream, p);
    }
    const dim3 grid(rows_grid(rows, (n + 4095) / 4096, 1, 4));
    return in_is_f32 ? launch(hadamard_rows_kernel<true>, grid, dim3(128), 0, stream, p)
                     : launch(hadamard_rows_kernel<false>, grid, dim3(128), 0, stream, p);
}

// ---- SwiGLU between its transforms, blocks of 256 ---------------------------------------------------------------------
// out = H(s_in * fp16(silu(g) * u)) * scale_in with (g | u) = fp16(s_out * H(in) * scale_out): the arithmetic and the order of
// stages of swiglu_hadamard_kernel, so the results are the same bits.  A warp takes 512 columns (a half-warp per block) and walks down
// the rows, the next row's values under way.  The kernel with eight values per thread is bound by its five shuffle stages per value.  2048 x
// 11008: 84.8 -> 55.5 us (bound by instruction issue, the division most of all).
__global__ void __launch_bounds__(256, 2) swiglu_rows_kernel(const SwigluParams p, int64_t rows) {
    __shared__ __align__(16) float smem[8 * kPairFloats];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & 15, half = lane >> 4;
    float *buf = smem + warp * kPairFloats + half * kHalfFloats;
    const Near16 near(buf, t);
    const Far16 far(buf, t);
    const int segs = (int)((p.n + 511) / 512);
    const int64_t worker = (int64_t)blockIdx.x * 8 + warp, workers = (int64_t)gridDim.x * 8 / segs * segs;
    pdl_allow_next_grid();
    // A last segment of one block: both halves of the warp take it, one stores.  (Zeros instead cost 1.6 times the kernel's time:
    // a division of zero takes the slow path.)
    const int64_t first = (worker % segs) * 512 + 256 * half;
    const bool active = first < p.n;
    const int64_t block0 = active ? first : p.n - 256;
    uint32_t sg[8], su[8], si[8];                            // signs in the far layout, two to a register
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        auto pair = [&](const __half *s) {
            return s ? half2_as_u32(__halves2half2(s[block0 + t + 32 * i], s[block0 + t + 32 * i + 16])) : 0x3C003C00u;
        };
        sg[i] = pair(p.signs_out), su[i] = pair(p.signs_out ? p.signs_out + p.n : nullptr), si[i] = pair(p.signs_in);
    }
    pdl_wait_prior_grids();
    if (worker >= workers) return;
    const int64_t step = workers / segs;
    uint32_t rg[8], ru[8];
    auto fetch = [&](int64_t row) {
        const __half *src = p.in16 + row * p.ld_acc + block0 + 16 * t;
        ld_32_bytes(src, rg);
        ld_32_bytes(src + p.n, ru);
    };
    int64_t row = worker / segs;
    if (row < rows) fetch(row);
    for (; row < rows; row += step) {
        float g[16], u[16], s[16];
        unpack_pairs(rg, g);
        unpack_pairs(ru, u);
        if (row + step < rows) fetch(row + step);
        stages16(g);
        near.put(g);
        stages16(u);
        __syncwarp();
        far.get(g);
        __syncwarp();
        near.put(u);
        stages16(g);
        __syncwarp();
        far.get(u);
        stages16(u);
        unpack_pairs(sg, s);
#pragma unroll
        for (int k = 0; k < 16; ++k) g[k] *= p.scale_out * s[k];
        unpack_pairs(su, s);
#pragma unroll
        for (int k = 0; k < 16; ++k) u[k] *= p.scale_out * s[k];
        unpack_pairs(si, s);
#pragma unroll
        for (int k = 0; k < 16; ++k) {                       // fp16 where the unfused path stores fp16
            const float gg = __half2float(__float2half_rn(g[k])), uu = __half2float(__float2half_rn(u[k]));
            g[k] = __half2float(__float2half_rn(gg / (1.f + __expf(-gg)) * uu)) * s[k];
        }
        far.put(g);                                          // where this thread has read
        __syncwarp();
        near.get(g);
        stages16(g);
        near.put(g);
        __syncwarp();
        far.get(g);
        stages16(g);
        far.put(g);
        __syncwarp();
        near.get(g);
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = half2_as_u32(__floats2half2_rn(g[2 * i] * p.scale_in, g[2 * i + 1] * p.scale_in));
        if (active) st_32_bytes(p.out + row * p.ld_out + block0 + 16 * t, o);
    }
}
int swiglu_rows(const SwigluParams &p, int64_t rows, cudaStream_t stream) {
    return launch(swiglu_rows_kernel, dim3(rows_grid(rows, (p.n + 511) / 512, 8, 2)), dim3(256), 0, stream, p, rows);
}

// ---- residual + RMSNorm + input transform -----------------------------------------------------------------------------
struct NormRowsParams {
    const __half *y;                 // [rows][ld_y]: the product in front, before its output transform, or NULL
    int64_t ld_y;
    const __half *signs_out;         // of the layer in front, or NULL
    float scale_out;
    __half *h;                       // [rows][ld_h] residual stream, updated in place when y is given
    int64_t ld_h;
    const __half *w_norm;
    float eps;
    const __half *signs_in;          // of the layer behind, or NULL
    __half *out;                     // [rows][ld_out]
    int64_t ld_out, rows;
};

// A row of NH x 4096 elements (each 4096 one Hadamard block of both transforms) per CTA of NH x 128 threads.  The results are
// the bits that rptc_hadamard, rptc_rmsnorm and rptc_hadamard give one after the other: same order of all sums.  (That of the
// squares is one of 256 threads over pairs 512 elements apart: a thread here holds what two of those hold.)
template <int NH>
__global__ void __launch_bounds__(128 * NH, 4 / NH) norm_rows_kernel(const NormRowsParams p) {
    constexpr int n = 4096 * NH;
    __shared__ __align__(16) float smem[NH * kCtaSegFloats];
    __shared__ float red[8], carry[2][128];
    const SegThread th;
    const int part = threadIdx.x >> 7;
    float *buf = smem + part * kCtaSegFloats;
    const int col0 = 4096 * part;
    // this thread's columns between the transforms: signs of the layer in front, and weight x sign of what comes next (a sign
    // commutes with the rounding of the normalised value)
    uint32_t so[16], ws[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int c = col0 + th.pair(k);
        so[k] = p.signs_out ? __ldg(reinterpret_cast<const uint32_t *>(p.signs_out + c)) : 0x3C003C00u;
        const float2 w = __half22float2(u32_as_half2(__ldg(reinterpret_cast<const uint32_t *>(p.w_norm + c))));
        const float2 si = p.signs_in ? __half22float2(u32_as_half2(__ldg(reinterpret_cast<const uint32_t *>(p.signs_in + c)))) : make_float2(1.f, 1.f);
        ws[k] = half2_as_u32(__floats2half2_rn(w.x * si.x, w.y * si.y));
    }
    pdl_allow_next_grid();
    pdl_wait_prior_grids();
    const float hn = 0.015625f;                              // 1 / sqrt(4096)
    for (int64_t row = blockIdx.x; row < p.rows; row += gridDim.x) {
        uint32_t hr[16];
        __half *hrow = p.h + row * p.ld_h + col0;
#pragma unroll
        for (int k = 0; k < 16; ++k) hr[k] = ldcg_u32(hrow + th.pair(k));
        float v[32];
        if (p.y) {
            const __half *yrow = p.y + row * p.ld_y + col0;
#pragma unroll
            for (int j = 0; j < 4; ++j) unpack8_at(__ldcg(reinterpret_cast<const uint4 *>(yrow + th.piece(j))), v + 8 * j);
            piece_stages(v);
            th.put_pieces(buf, v);
            __syncthreads();
            th.get_columns(buf, v);
            column_stages(v, 12);
            th.put_columns(buf, v);
            __syncthreads();
            th.get_pairs(buf, v);
            far_stages(v, 12);
            const float sc = p.scale_out * hn;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const float2 s = __half22float2(u32_as_half2(so[k])), r = __half22float2(u32_as_half2(hr[k]));
                const float a = __fadd_rn(__fmul_rn(v[2 * k], sc * s.x), r.x), b = __fadd_rn(__fmul_rn(v[2 * k + 1], sc * s.y), r.y);
                hr[k] = half2_as_u32(__floats2half2_rn(a, b));
                *reinterpret_cast<uint32_t *>(hrow + th.pair(k)) = hr[k];
            }
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) {                        // go on from the rounded residual stream, as a reader of h would
            const float2 f = __half22float2(u32_as_half2(hr[k]));
            v[2 * k] = f.x, v[2 * k + 1] = f.y;
        }
        float ss[2] = {0.f, 0.f};
        if (NH == 2) {                                        // the second piece goes on with the sums of the first
            if (part == 1) asm volatile("bar.sync 1, 256;" ::: "memory");
            if (part == 1) ss[0] = carry[0][th.t], ss[1] = carry[1][th.t];
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) ss[k & 1] += v[2 * k] * v[2 * k] + v[2 * k + 1] * v[2 * k + 1];
        if (NH == 2 && part == 0) {
            carry[0][th.t] = ss[0], carry[1][th.t] = ss[1];
            asm volatile("bar.arrive 1, 256;" ::: "memory");
        }
        if (part == NH - 1) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ss[i] += __shfl_xor_sync(0xFFFFFFFFu, ss[i], o);
                if (th.lane == 0) red[4 * i + th.warp] = ss[i];
            }
        }
        __syncthreads();
        float tot = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) tot += red[i];
        const float inv = rsqrtf(tot / n + p.eps);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float2 w = __half22float2(u32_as_half2(ws[k]));
            const float2 f = __half22float2(__floats2half2_rn(v[2 * k] * inv * w.x, v[2 * k + 1] * inv * w.y));
            v[2 * k] = f.x, v[2 * k + 1] = f.y;
        }
        th.put_pairs(buf, v);
        __syncthreads();
        th.get_pieces(buf, v);
        piece_stages(v);
        th.put_pieces(buf, v);
        __syncthreads();
        th.get_columns(buf, v);
        column_stages(v, 12);
        th.put_columns(buf, v);
        __syncthreads();
        th.get_pairs(buf, v);
        far_stages(v, 12);
        __half *orow = p.out + row * p.ld_out + col0;
#pragma unroll
        for (int k = 0; k < 16; ++k)
            *reinterpret_cast<uint32_t *>(orow + th.pair(k)) = half2_as_u32(__floats2half2_rn(v[2 * k] * hn, v[2 * k + 1] * hn));
        __syncthreads();                                      // the buffer is free for the next row
    }
}

// The same for rows of 2^BITS = 256 to 2048 elements, one Hadamard block each: a segment of 4096 elements is 4096 / 2^BITS rows.  Bound as
// above by the trips through shared memory and their barriers.  2048 rows of 2048 14.8 us, a row per CTA with eight values a thread and
// shuffles 31.1, as three kernels 38; a prompt of 1024 tokens through 24 layers of hidden 2048 5.62 -> 4.96 ms, of 64 tokens 3.83 -> 3.03.
template <int BITS>
__global__ void __launch_bounds__(128, 4) norm_short_rows_kernel(const NormRowsParams p, float hn) {
    constexpr int n = 1 << BITS, R = 4096 >> BITS, KR = n / 256;      // rows of a segment, pairs of a thread in each
    __shared__ __align__(16) float smem[kCtaSegFloats];
    __shared__ float red[R][8];
    const SegThread th;
    uint32_t so[KR], ws[KR];
#pragma unroll
    for (int k = 0; k < KR; ++k) {
        const int c = th.pair(k);
        so[k] = p.signs_out ? __ldg(reinterpret_cast<const uint32_t *>(p.signs_out + c)) : 0x3C003C00u;
        const float2 w = __half22float2(u32_as_half2(__ldg(reinterpret_cast<const uint32_t *>(p.w_norm + c))));
        const float2 si = p.signs_in ? __half22float2(u32_as_half2(__ldg(reinterpret_cast<const uint32_t *>(p.signs_in + c)))) : make_float2(1.f, 1.f);
        ws[k] = half2_as_u32(__floats2half2_rn(w.x * si.x, w.y * si.y));
    }
    pdl_allow_next_grid();
    pdl_wait_prior_grids();
    for (int64_t row0 = (int64_t)blockIdx.x * R; row0 < p.rows; row0 += (int64_t)gridDim.x * R) {
        // rows past the end read the last one and store nothing
        auto row_of = [&](int e) { return min(row0 + (e >> BITS), p.rows - 1); };
        auto inside = [&](int k) { return row0 + k / KR < p.rows; };
        uint32_t hr[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) hr[k] = ldcg_u32(p.h + row_of(256 * k) * p.ld_h + th.pair(k % KR));
        float v[32];
        if (p.y) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                unpack8_at(__ldcg(reinterpret_cast<const uint4 *>(p.y + row_of(th.piece(j)) * p.ld_y + (th.piece(j) & (n - 1)))), v + 8 * j);
            piece_stages(v);
            th.put_pieces(smem, v);
            __syncthreads();
            th.get_columns(smem, v);
            column_stages(v, BITS);
            th.put_columns(smem, v);
            __syncthreads();
            th.get_pairs(smem, v);
            far_stages(v, BITS);
            const float sc = p.scale_out * hn;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const float2 s = __half22float2(u32_as_half2(so[k % KR])), r = __half22float2(u32_as_half2(hr[k]));
                const float a = __fadd_rn(__fmul_rn(v[2 * k], sc * s.x), r.x), b = __fadd_rn(__fmul_rn(v[2 * k + 1], sc * s.y), r.y);
                hr[k] = half2_as_u32(__floats2half2_rn(a, b));
                if (inside(k)) *reinterpret_cast<uint32_t *>(p.h + row_of(256 * k) * p.ld_h + th.pair(k % KR)) = hr[k];
            }
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float2 f = __half22float2(u32_as_half2(hr[k]));
            v[2 * k] = f.x, v[2 * k + 1] = f.y;
        }
#pragma unroll
        for (int q = 0; q < R; ++q) {
            float ss[2] = {0.f, 0.f};
#pragma unroll
            for (int k = q * KR; k < (q + 1) * KR; ++k) ss[(k - q * KR) & 1] += v[2 * k] * v[2 * k] + v[2 * k + 1] * v[2 * k + 1];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ss[i] += __shfl_xor_sync(0xFFFFFFFFu, ss[i], o);
                if (th.lane == 0) red[q][4 * i + th.warp] = ss[i];
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < R; ++q) {
            float tot = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) tot += red[q][i];
            const float inv = rsqrtf(tot / n + p.eps);
#pragma unroll
            for (int k = q * KR; k < (q + 1) * KR; ++k) {
                const float2 w = __half22float2(u32_as_half2(ws[k % KR]));
                const float2 f = __half22float2(__floats2half2_rn(v[2 * k] * inv * w.x, v[2 * k + 1] * inv * w.y));
                v[2 * k] = f.x, v[2 * k + 1] = f.y;
            }
        }
        th.put_pairs(smem, v);
        __syncthreads();
        th.get_pieces(smem, v);
        piece_stages(v);
        th.put_pieces(smem, v);
        __syncthreads();
        th.get_columns(smem, v);
        column_stages(v, BITS);
        th.put_columns(smem, v);
        __syncthreads();
        th.get_pairs(smem, v);
        far_stages(v, BITS);
#pragma unroll
        for (int k = 0; k < 16; ++k)
            if (inside(k))
                *reinterpret_cast<uint32_t *>(p.out + row_of(256 * k) * p.ld_out + th.pair(k % KR)) =
                    half2_as_u32(__floats2half2_rn(v[2 * k] * hn, v[2 * k + 1] * hn));
        __syncthreads();                                      // the buffer is free for the next rows
    }
}

// ---- output side of the fused qkv layer for a prompt -------------------------------------------------------------------
struct QkvRowsParams {
    __half *qkv;                     // [rows * tokens][ld]: the product; q comes back in place
    int64_t ld;
    const __half *signs_out;
    float scale;                     // includes 1 / sqrt(128)
    const float2 *angles;            // [tokens][64] cosine, sine
    __half *kcache, *vcache;         // [rows][max_pos][hkv][128]
    int64_t rows, tokens;
    int32_t hq, hkv, max_pos;
};

// cos and sin of position x inverse frequency, once per prompt
__global__ void __launch_bounds__(64) rope_angles_kernel(float2 *__restrict__ out, RopeFreq freq) {
    pdl_allow_next_grid();
    pdl_wait_prior_grids();
    float sn, cs;
    sincosf((float)blockIdx.x * rope_inv_freq(freq, threadIdx.x), &sn, &cs);
    out[(int64_t)blockIdx.x * 64 + threadIdx.x] = make_float2(cs, sn);
}

// A half-warp takes two heads of a token: in the far layout a thread holds both members of every rotated pair (elements i and
// i + 64 differ in bit 6).  WIDE: everything on 32-byte boundaries.  Bound: HBM, with the next token's values under way.
template <bool WIDE>
__device__ __forceinline__ void ld_half_row(const __half *p, uint32_t (&r)[8]) {
    if (WIDE) return ld_32_bytes(p, r);
    const uint4 a = __ldcg(reinterpret_cast<const uint4 *>(p)), b = __ldcg(reinterpret_cast<const uint4 *>(p) + 1);
    r[0] = a.x, r[1] = a.y, r[2] = a.z, r[3] = a.w, r[4] = b.x, r[5] = b.y, r[6] = b.z, r[7] = b.w;
}
template <bool WIDE>
__global__ void __launch_bounds__(256, 3) qkv_rows_kernel(const QkvRowsParams p) {
    __shared__ __align__(16) float smem[8 * kPairFloats];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & 15, half = lane >> 4;
    float *buf = smem + warp * kPairFloats + half * kHalfFloats;
    const Near16 near(buf, t);
    const Far16 far(buf, t);
    const int heads = p.hq + 2 * p.hkv, n = heads * 128, segs = (n + 511) / 512;
    const int64_t worker = (int64_t)blockIdx.x * 8 + warp, workers = (int64_t)gridDim.x * 8 / segs * segs;
    pdl_allow_next_grid();
    if (worker >= workers) return;
    const int col0 = (int)(worker % segs) * 512 + 256 * half, head0 = col0 >> 7, col = col0 + 16 * t, head = col >> 7;
    const bool active = col < n;
    uint32_t signs = 0;                                       // bit k: the sign of this thread's far element k
    if (p.signs_out) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int c = col0 + t + 16 * k;
            if (c < n) signs |= (uint32_t)(__ldg(reinterpret_cast<const unsigned short *>(p.signs_out) + c) >> 15) << k;
        }
    }
    const int rotated = p.hq + p.hkv - head0;                 // how many of the two heads, if positive
    const int64_t step = workers / segs, last = p.rows * p.tokens;
    pdl_wait_prior_grids();
    uint32_t raw[8] = {};
    int64_t row = worker / segs;
    if (row < last && active) ld_half_row<WIDE>(p.qkv + row * p.ld + col, raw);
    for (; row < last; row += step) {
        const int64_t seq = row / p.tokens, pos = row - seq * p.tokens;
        float v[16];
        unpack_pairs(raw, v);
        float2 cs[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) cs[k] = __ldg(p.angles + pos * 64 + t + 16 * k);
        if (row + step < last && active) ld_half_row<WIDE>(p.qkv + (row + step) * p.ld + col, raw);
        stages16(v);
        near.put(v);                                          // where this thread has read
        __syncwarp();
        far.get(v);
        far_stages16(v, 7);
#pragma unroll
        for (int k = 0; k < 16; ++k) {                        // the layer's fp16 output
            const float sc = ((signs >> k) & 1u) ? -p.scale : p.scale;
            v[k] = __half2float(__float2half_rn(v[k] * sc));
        }
#pragma unroll
        for (int hd = 0; hd < 2; ++hd) {
            if (hd >= rotated) continue;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float a = v[8 * hd + k], b = v[8 * hd + 4 + k];
                v[8 * hd + k] = a * cs[k].x - b * cs[k].y;
                v[8 * hd + 4 + k] = b * cs[k].x + a * cs[k].y;
            }
        }
        far.put(v);
        __syncwarp();
        near.get(v);
        if (active) {
            const int i = col & 127;
            __half *dst = head < p.hq ? p.qkv + row * p.ld + col
                          : head < p.hq + p.hkv ? p.kcache + ((seq * p.max_pos + pos) * p.hkv + head - p.hq) * 128 + i
                                                : p.vcache + ((seq * p.max_pos + pos) * p.hkv + head - p.hq - p.hkv) * 128 + i;
            uint32_t o[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) o[q] = half2_as_u32(__floats2half2_rn(v[2 * q], v[2 * q + 1]));
            if (WIDE) {
                st_32_bytes(dst, o);
            } else {
                reinterpret_cast<uint4 *>(dst)[0] = make_uint4(o[0], o[1], o[2], o[3]);
                reinterpret_cast<uint4 *>(dst)[1] = make_uint4(o[4], o[5], o[6], o[7]);
            }
        }
    }
}

}  // namespace rptc

using namespace rptc;

extern "C" int rptc_prompt_norm(const void *y, int64_t ld_y, const void *signs_out, float scale_out, void *h, int64_t ld_h, const void *w_norm,
                                float eps, const void *signs_in, void *out, int64_t ld_out, int64_t rows, int64_t n, rptc_stream_t stream) {
    if (!h || !w_norm || !out) return RPTC_ERR_ARG;
    if (n < 256 || n > 8192 || (n & (n - 1))) return RPTC_ERR_UNSUPPORTED;
    if (rows <= 0 || ld_h < n || ld_out < n || (y && ld_y < n)) return RPTC_ERR_SHAPE;
    auto misaligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
    if (misaligned(y) || misaligned(h) || misaligned(w_norm) || misaligned(out) || misaligned(signs_out) || misaligned(signs_in) || (ld_h % 8) ||
        (ld_out % 8) || (y && (ld_y % 8)))
        return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    NormRowsParams p;
    p.y = static_cast<const __half *>(y);
    p.ld_y = ld_y;
    p.signs_out = static_cast<const __half *>(signs_out);
    p.scale_out = scale_out;
    p.h = static_cast<__half *>(h);
    p.ld_h = ld_h;
    p.w_norm = static_cast<const __half *>(w_norm);
    p.eps = eps;
    p.signs_in = static_cast<const __half *>(signs_in);
    p.out = static_cast<__half *>(out);
    p.ld_out = ld_out;
    p.rows = rows;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n < 4096) {
        const dim3 grid(rows_grid((rows * n + 4095) / 4096, 1, 1, 4));
        const float hn = norm_of((int)n);
        if (n == 2048) return launch(norm_short_rows_kernel<11>, grid, dim3(128), 0, s, p, hn);
        if (n == 1024) return launch(norm_short_rows_kernel<10>, grid, dim3(128), 0, s, p, hn);
        if (n == 512) return launch(norm_short_rows_kernel<9>, grid, dim3(128), 0, s, p, hn);
        return launch(norm_short_rows_kernel<8>, grid, dim3(128), 0, s, p, hn);
    }
    if (n == 4096) return launch(norm_rows_kernel<1>, dim3(rows_grid(rows, 1, 1, 4)), dim3(128), 0, s, p);
    return launch(norm_rows_kernel<2>, dim3(rows_grid(rows, 1, 1, 2)), dim3(256), 0, s, p);
}

extern "C" int rptc_prompt_qkv(void *qkv, int64_t ld, const void *signs_out, float scale, int64_t rows, int64_t tokens, void *kcache, void *vcache,
                               int hq, int hkv, int max_pos, const void *angles, rptc_stream_t stream) {
    if (!qkv || !kcache || !vcache || !angles) return RPTC_ERR_ARG;
    if (rows <= 0 || tokens <= 0 || hq <= 0 || hkv <= 0 || tokens > max_pos || ld < (int64_t)(hq + 2 * hkv) * 128) return RPTC_ERR_SHAPE;
    auto misaligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
    if (misaligned(qkv) || misaligned(kcache) || misaligned(vcache) || misaligned(angles) || (ld % 8)) return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;
    QkvRowsParams p;
    p.qkv = static_cast<__half *>(qkv);
    p.ld = ld;
    p.signs_out = static_cast<const __half *>(signs_out);
    p.scale = scale * norm_of(128);
    p.angles = static_cast<const float2 *>(angles);
    p.kcache = static_cast<__half *>(kcache);
    p.vcache = static_cast<__half *>(vcache);
    p.rows = rows;
    p.tokens = tokens;
    p.hq = hq;
    p.hkv = hkv;
    p.max_pos = max_pos;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid(rows_grid(rows * tokens, ((int64_t)(hq + 2 * hkv) * 128 + 511) / 512, 8, 3));
    const bool wide = ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache)) & 31) == 0 && ld % 16 == 0;
    return wide ? launch(qkv_rows_kernel<true>, grid, dim3(256), 0, s, p) : launch(qkv_rows_kernel<false>, grid, dim3(256), 0, s, p);
}

extern "C" int rptc_rope_angles(void *angles, int64_t tokens, float theta, rptc_stream_t stream) {
    if (!angles) return RPTC_ERR_ARG;
    if (tokens <= 0 || tokens > (1 << 30)) return RPTC_ERR_SHAPE;
    if (int e = rptc_check_device()) return e;
    return launch(rope_angles_kernel, dim3((unsigned)tokens), dim3(64), 0, static_cast<cudaStream_t>(stream), static_cast<float2 *>(angles),
                  rope_freq(theta, 128));
}
