// The transforms and the glue of a prompt's forward pass: many rows at once, fp16 in and out, fp32 inside.
//   hadamard_rows     rptc_hadamard for many rows
//   norm_rows         h += s_out * H(y) * scale;  xn = rmsnorm(h) * w;  out = H(s_in * xn)        (rptc_prompt_norm)
//   qkv_rows          output transform of the fused qkv layer, rotary embedding, cache writes     (rptc_prompt_qkv)
//   swiglu_rows       rptc_swiglu_hadamard_f16 for many rows
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
};

// One segment of a row per warp (blocks up to 256) or per CTA of 128 threads.
template <bool CTA, bool IN_F32>
__global__ void __launch_bounds__(CTA ? 128 : 256, CTA ? 4 : 2) hadamard_rows_kernel(const HadRowsParams p) {
    constexpr int kSeg = CTA ? 4096 : 1024, kUnits = CTA ? 1 : 8;       // segments per CTA
    __shared__ __align__(16) float smem[CTA ? kCtaSegFloats : 8 * kWarpSegFloats];
    const SegThread<CTA> th;
    const int unit = CTA ? 0 : threadIdx.x >> 5;
    float *buf = smem + unit * kWarpSegFloats;
    const int segs = (int)((p.n + kSeg - 1) / kSeg);
    const int64_t worker = (int64_t)blockIdx.x * kUnits + unit, workers = (int64_t)gridDim.x * kUnits / segs * segs;
    pdl_allow_next_grid();
    pdl_wait_prior_grids();
    if (p.clear) {
        float4 *z = reinterpret_cast<float4 *>(p.clear);
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; 4 * i < p.clear_count; i += (int64_t)gridDim.x * blockDim.x)
            z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (worker >= workers) return;
    const int64_t col0 = (worker % segs) * kSeg;
    const int lo = CTA ? 10 : 8;                             // the bits that number the pieces as loaded
    uint4 sg[4];                                             // of the pieces as they are when the signs apply
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int64_t c = col0 + th.piece(j, !p.transpose);
        sg[j] = (p.signs && c < p.n) ? __ldg(reinterpret_cast<const uint4 *>(p.signs + c)) : make_uint4(0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u);
    }
    for (int64_t row = worker / segs; row < p.rows; row += workers / segs) {
        float v[32];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t c = col0 + th.piece(j, true);
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
        uint4 res[4];
        if (p.residual) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int64_t c = col0 + th.piece(j, false);
                if (c < p.n) res[j] = __ldcg(reinterpret_cast<const uint4 *>(p.residual + row * p.ld_res + c));
            }
        }
        if (!p.transpose) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float s[8];
                unpack8_at(sg[j], s);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[8 * j + i] *= s[i];
            }
        }
        row_stages(v, p.block_bits, lo);
        th.put_pieces(buf, v, true);
        th.sync();
        th.get_columns(buf, v);
        column_stages(v, p.block_bits);
        th.put_columns(buf, v);
        th.sync();
        th.get_pieces(buf, v, false);
        if (CTA) {
            if (p.block_bits > 8) stage<8>(v);
            if (p.block_bits > 9) stage<16>(v);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t c = col0 + th.piece(j, false);
            if (c >= p.n) continue;
            float s[8], r[8];
            if (p.transpose) unpack8_at(sg[j], s);
            if (p.residual) unpack8_at(res[j], r);
            float o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                o[i] = v[8 * j + i] * (p.transpose ? p.scale * s[i] : p.scale);
                if (p.residual) o[i] += r[i];
            }
            *reinterpret_cast<uint4 *>(p.out + row * p.ld_out + c) = pack8_from(o);
        }
        th.sync();                                           // the buffer is free for the next row
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
                  cudaStream_t stream) {
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
    if (block <= 256) {
        const dim3 grid(rows_grid(rows, (n + 1023) / 1024, 8, 2));
        return in_is_f32 ? launch(hadamard_rows_kernel<false, true>, grid, dim3(256), 0, stream, p)
                         : launch(hadamard_rows_kernel<false, false>, grid, dim3(256), 0, stream, p);
    }
    const dim3 grid(rows_grid(rows, (n + 4095) / 4096, 1, 4));
    return in_is_f32 ? launch(hadamard_rows_kernel<true, true>, grid, dim3(128), 0, stream, p)
                     : launch(hadamard_rows_kernel<true, false>, grid, dim3(128), 0, stream, p);
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

// A row of NH x 4096 elements (each 4096 one Hadamard block of both transforms) per CTA of NH x 128 threads.
template <int NH>
__global__ void __launch_bounds__(128 * NH, 4 / NH) norm_rows_kernel(const NormRowsParams p) {
    constexpr int n = 4096 * NH;
    __shared__ __align__(16) float smem[NH * kCtaSegFloats];
    __shared__ float red[2][4 * NH];
    const SegThread<true> th;
    const int part = threadIdx.x >> 7, warp = threadIdx.x >> 5;
    float *buf = smem + part * kCtaSegFloats;
    const uint4 ones = make_uint4(0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u);
    // this thread's columns after the output transform: signs of the layer in front, and weight x sign of what comes next
    // (a sign commutes with the rounding of the normalised value)
    uint4 so[4], ws[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = 4096 * part + th.piece(j, false);
        so[j] = p.signs_out ? __ldg(reinterpret_cast<const uint4 *>(p.signs_out + c)) : ones;
        const uint4 w = __ldg(reinterpret_cast<const uint4 *>(p.w_norm + c)), si = p.signs_in ? __ldg(reinterpret_cast<const uint4 *>(p.signs_in + c)) : ones;
        float a[8], b[8];
        unpack8_at(w, a);
        unpack8_at(si, b);
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] *= b[i];
        ws[j] = pack8_from(a);
    }
    pdl_allow_next_grid();
    pdl_wait_prior_grids();
    const float hn = 0.015625f;                              // 1 / sqrt(4096)
    int turn = 0;
    for (int64_t row = blockIdx.x; row < p.rows; row += gridDim.x, turn ^= 1) {
        uint4 hr[4];
        __half *hrow = p.h + row * p.ld_h + 4096 * part;
#pragma unroll
        for (int j = 0; j < 4; ++j) hr[j] = __ldcg(reinterpret_cast<const uint4 *>(hrow + th.piece(j, false)));
        float v[32];
        if (p.y) {
            const __half *yrow = p.y + row * p.ld_y + 4096 * part;
#pragma unroll
            for (int j = 0; j < 4; ++j) unpack8_at(__ldcg(reinterpret_cast<const uint4 *>(yrow + th.piece(j, true))), v + 8 * j);
            row_stages(v, 12, 10);
            th.put_pieces(buf, v, true);
            __syncthreads();
            th.get_columns(buf, v);
            column_stages(v, 12);
            th.put_columns(buf, v);
            __syncthreads();
            th.get_pieces(buf, v, false);
            stage<8>(v);
            stage<16>(v);
            const float sc = p.scale_out * hn;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float s[8], r[8];
                unpack8_at(so[j], s);
                unpack8_at(hr[j], r);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[8 * j + i] = r[i] + v[8 * j + i] * sc * s[i];
                const uint4 o = pack8_from(v + 8 * j);
                *reinterpret_cast<uint4 *>(hrow + th.piece(j, false)) = o;
                unpack8_at(o, v + 8 * j);                     // go on from the rounded residual stream, as a reader of h would
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) unpack8_at(hr[j], v + 8 * j);
        }
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) ss += v[i] * v[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
        if (th.lane == 0) red[turn][warp] = ss;
        __syncthreads();                                      // also: everyone is done with the exchange buffer
        ss = 0.f;
#pragma unroll
        for (int i = 0; i < 4 * NH; ++i) ss += red[turn][i];
        const float inv = rsqrtf(ss / n + p.eps);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float w[8];
            unpack8_at(ws[j], w);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[8 * j + i] = __half2float(__float2half_rn(v[8 * j + i] * inv * w[i]));
        }
        row_stages(v, 12, 8);
        th.put_pieces(buf, v, false);
        __syncthreads();
        th.get_columns(buf, v);
        column_stages(v, 12);
        th.put_columns(buf, v);
        __syncthreads();
        th.get_pieces(buf, v, true);
        stage<8>(v);
        stage<16>(v);
        __half *orow = p.out + row * p.ld_out + 4096 * part;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[8 * j + i] *= hn;
            *reinterpret_cast<uint4 *>(orow + th.piece(j, true)) = pack8_from(v + 8 * j);
        }
        __syncthreads();                                      // the buffer is free for the next row
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

// A warp takes eight heads of a token: after the column stages a thread holds both members of every rotated pair
// (elements i and i + 64 differ in bit 6).
__global__ void __launch_bounds__(256, 2) qkv_rows_kernel(const QkvRowsParams p) {
    __shared__ __align__(16) float smem[8 * kWarpSegFloats];
    const SegThread<false> th;
    const int unit = threadIdx.x >> 5;
    float *buf = smem + unit * kWarpSegFloats;
    const int heads = p.hq + 2 * p.hkv, n = heads * 128, segs = (n + 1023) / 1024;
    const int64_t worker = (int64_t)blockIdx.x * 8 + unit, workers = (int64_t)gridDim.x * 8 / segs * segs;
    pdl_allow_next_grid();
    if (worker >= workers) return;
    const int col0 = (int)(worker % segs) * 1024;
    uint32_t signs = 0;                                       // bit k: the sign of this thread's column element k
    if (p.signs_out) {
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const int c = col0 + th.column() + 8 * k;
            if (c < n) signs |= (uint32_t)(__ldg(reinterpret_cast<const unsigned short *>(p.signs_out) + c) >> 15) << k;
        }
    }
    const int head0 = (col0 >> 7) + 2 * (th.lane >> 3);       // of k < 16; k >= 16 belong to the next head
    const bool rot0 = head0 < p.hq + p.hkv, rot1 = head0 + 1 < p.hq + p.hkv;
    pdl_wait_prior_grids();
    for (int64_t row = worker / segs; row < p.rows * p.tokens; row += workers / segs) {
        const int64_t seq = row / p.tokens, pos = row - seq * p.tokens;
        __half *src = p.qkv + row * p.ld + col0;
        float v[32];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = th.piece(j, true);
            unpack8_at(col0 + c < n ? __ldcg(reinterpret_cast<const uint4 *>(src + c)) : make_uint4(0u, 0u, 0u, 0u), v + 8 * j);
        }
        float2 cs[8];
        const float2 *ang = p.angles + pos * 64 + (th.lane & 7);
#pragma unroll
        for (int k = 0; k < 8; ++k) cs[k] = __ldg(ang + 8 * k);
        row_stages(v, 7, 8);
        th.put_pieces(buf, v, true);
        __syncwarp();
        th.get_columns(buf, v);
        column_stages(v, 7);
#pragma unroll
        for (int k = 0; k < 32; ++k) {                        // the layer's fp16 output
            const float sc = ((signs >> k) & 1u) ? -p.scale : p.scale;
            v[k] = __half2float(__float2half_rn(v[k] * sc));
        }
#pragma unroll
        for (int hd = 0; hd < 2; ++hd) {
            if (!(hd ? rot1 : rot0)) continue;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float a = v[16 * hd + k], b = v[16 * hd + 8 + k];
                v[16 * hd + k] = a * cs[k].x - b * cs[k].y;
                v[16 * hd + 8 + k] = b * cs[k].x + a * cs[k].y;
            }
        }
        th.put_columns(buf, v);
        __syncwarp();
        th.get_pieces(buf, v, true);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = th.piece(j, true), head = (col0 + c) >> 7, i = c & 127;
            if (col0 + c >= n) continue;
            __half *dst = head < p.hq ? src + c
                          : head < p.hq + p.hkv ? p.kcache + ((seq * p.max_pos + pos) * p.hkv + head - p.hq) * 128 + i
                                                : p.vcache + ((seq * p.max_pos + pos) * p.hkv + head - p.hq - p.hkv) * 128 + i;
            *reinterpret_cast<uint4 *>(dst) = pack8_from(v + 8 * j);
        }
        __syncwarp();
    }
}

// ---- gated MLP middle ---------------------------------------------------------------------------------------------------
struct SwigluRowsParams {
    const __half *in;                // [rows][ld_in >= 2n]: gate | up, before the output transform
    int64_t ld_in;
    __half *out;
    int64_t ld_out;
    const __half *signs_out, *signs_in;
    int64_t rows, n;
    int32_t block_bits;
    float scale_out, scale_in;       // include the 1 / sqrt(block) of their transform
};

// A warp takes 1024 columns of a row (blocks up to 256).  Gate and up end their transforms in the column layout, the product
// starts its own there, so that three transforms cost six passes through the exchange buffer instead of twelve.
__global__ void __launch_bounds__(256, 2) swiglu_rows_kernel(const SwigluRowsParams p) {
    __shared__ __align__(16) float smem[8 * kWarpSegFloats];
    const SegThread<false> th;
    const int unit = threadIdx.x >> 5;
    float *buf = smem + unit * kWarpSegFloats;
    const int segs = (int)((p.n + 1023) / 1024);
    const int64_t worker = (int64_t)blockIdx.x * 8 + unit, workers = (int64_t)gridDim.x * 8 / segs * segs;
    pdl_allow_next_grid();
    if (worker >= workers) return;
    const int64_t col0 = (worker % segs) * 1024;
    uint32_t sgn_g = 0, sgn_u = 0, sgn_i = 0;                 // bit k: sign of this thread's column element k
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
        const int64_t c = col0 + th.column() + 8 * k;
        if (c >= p.n) continue;
        const unsigned short *so = reinterpret_cast<const unsigned short *>(p.signs_out), *si = reinterpret_cast<const unsigned short *>(p.signs_in);
        if (so) sgn_g |= (uint32_t)(__ldg(so + c) >> 15) << k, sgn_u |= (uint32_t)(__ldg(so + p.n + c) >> 15) << k;
        if (si) sgn_i |= (uint32_t)(__ldg(si + c) >> 15) << k;
    }
    pdl_wait_prior_grids();
    for (int64_t row = worker / segs; row < p.rows; row += workers / segs) {
        const __half *src = p.in + row * p.ld_in + col0;
        uint4 ru[4];
        float g[32], u[32];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = th.piece(j, true);
            const bool in = col0 + c < p.n;
            const uint4 rg = in ? __ldcg(reinterpret_cast<const uint4 *>(src + c)) : make_uint4(0u, 0u, 0u, 0u);
            ru[j] = in ? __ldcg(reinterpret_cast<const uint4 *>(src + p.n + c)) : make_uint4(0u, 0u, 0u, 0u);
            unpack8_at(rg, g + 8 * j);
        }
        row_stages(g, p.block_bits, 8);
        th.put_pieces(buf, g, true);
        __syncwarp();
        th.get_columns(buf, g);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) unpack8_at(ru[j], u + 8 * j);
        row_stages(u, p.block_bits, 8);
        th.put_pieces(buf, u, true);
        __syncwarp();
        th.get_columns(buf, u);
        column_stages(g, p.block_bits);
        column_stages(u, p.block_bits);
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            // the layer's own output is fp16, and so is the gated product
            const float gg = __half2float(__float2half_rn(g[k] * (((sgn_g >> k) & 1u) ? -p.scale_out : p.scale_out)));
            const float uu = __half2float(__float2half_rn(u[k] * (((sgn_u >> k) & 1u) ? -p.scale_out : p.scale_out)));
            const float m = __half2float(__float2half_rn(__fdividef(gg, 1.f + __expf(-gg)) * uu));
            g[k] = ((sgn_i >> k) & 1u) ? -m : m;
        }
        column_stages(g, p.block_bits);
        __syncwarp();
        th.put_columns(buf, g);
        __syncwarp();
        th.get_pieces(buf, g, true);
        row_stages(g, p.block_bits, 8);
        __half *dst = p.out + row * p.ld_out + col0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = th.piece(j, true);
            if (col0 + c >= p.n) continue;
#pragma unroll
            for (int i = 0; i < 8; ++i) g[8 * j + i] *= p.scale_in;
            *reinterpret_cast<uint4 *>(dst + c) = pack8_from(g + 8 * j);
        }
        __syncwarp();
    }
}

int swiglu_rows(const void *gate_up, int64_t ld_in, void *out, int64_t ld_out, const void *signs_out, const void *signs_in, int64_t rows, int64_t n,
                int block, float scale_out, float scale_in, cudaStream_t stream) {
    SwigluRowsParams p;
    p.in = static_cast<const __half *>(gate_up);
    p.ld_in = ld_in;
    p.out = static_cast<__half *>(out);
    p.ld_out = ld_out;
    p.signs_out = static_cast<const __half *>(signs_out);
    p.signs_in = static_cast<const __half *>(signs_in);
    p.rows = rows;
    p.n = n;
    p.block_bits = log2_of(block);
    p.scale_out = scale_out * norm_of(block);
    p.scale_in = scale_in * norm_of(block);
    return launch(swiglu_rows_kernel, dim3(rows_grid(rows, (n + 1023) / 1024, 8, 2)), dim3(256), 0, stream, p);
}

}  // namespace rptc

using namespace rptc;

extern "C" int rptc_prompt_norm(const void *y, int64_t ld_y, const void *signs_out, float scale_out, void *h, int64_t ld_h, const void *w_norm,
                                float eps, const void *signs_in, void *out, int64_t ld_out, int64_t rows, int64_t n, rptc_stream_t stream) {
    if (!h || !w_norm || !out) return RPTC_ERR_ARG;
    if (n != 4096 && n != 8192) return RPTC_ERR_UNSUPPORTED;
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
    return launch(qkv_rows_kernel, dim3(rows_grid(rows * tokens, ((int64_t)(hq + 2 * hkv) * 128 + 1023) / 1024, 8, 2)), dim3(256), 0, s, p);
}

extern "C" int rptc_rope_angles(void *angles, int64_t tokens, float theta, rptc_stream_t stream) {
    if (!angles) return RPTC_ERR_ARG;
    if (tokens <= 0 || tokens > (1 << 30)) return RPTC_ERR_SHAPE;
    if (int e = rptc_check_device()) return e;
    return launch(rope_angles_kernel, dim3((unsigned)tokens), dim3(64), 0, static_cast<cudaStream_t>(stream), static_cast<float2 *>(angles),
                  rope_freq(theta, 128));
}
