// Standalone RPTC decompress: packed trellis codes -> dense fp16 [m][n] on sm_100a.
//
// A persistent grid of one CTA per SM keeps the lookup table in shared memory for the whole launch.  Work is cut into
// warp tasks of 32 "groups" (a group is one 128-bit unit, or three units when K = 3) and the flattened task list is split
// evenly over all warps.  Two lane mappings:
//   ROWLANES  (TILED / UNITMAJOR codes): lane = row of a 32-row block, the warp walks along the rows group
//             by group; the load of a group is one coalesced 512-byte request and the 16 bits of
//             history come from the previous iteration's last word.  At most 64 columns at a time go through a
//             per-warp shared-memory tile (4 KiB), swizzled as a TMA store reads it, which takes it to the output: the
//             load/store unit is left to the lookups, and 24 warps fit beside the 128 KiB table.
//   !ROWLANES (ROWMAJOR / CHUNKED codes): lane = one of 32 consecutive groups of one row; history
//             comes from the lane to the left by shuffle.  The tile is copied out with 128-bit stores in which every
//             group of lanes covers whole 128-byte lines of the output.
// Output is 8x (K=2) the input.  Bound: HBM; with the 65,536-entry table the shared-memory banks (32 lookups of random
// 2-byte entries take about 3.5 passes: 148 SMs look up 2.6e12 weights a second).
#include "common.cuh"
#include "tc_ptx.cuh"

namespace rptc {

constexpr int kDecThreads = 768;

struct DecParams {
    const uint4 *codes;
    UnitStrides st;
    const __half *lut;
    const uint32_t *carry_in;
    __half *out;
    int64_t ld_out;
    int64_t m;
    int32_t n_groups;
    int32_t L, S, quirk;
    unsigned int *status;
};

template <int K>
struct DecTile {
    static constexpr int kRowBytes = 2 * GroupShape<K>::kWeights;      // 128, 256, 64
    static constexpr int kChunks = kRowBytes / 16;                     // 8, 16, 4
    static constexpr int kBytes = 32 * kRowBytes;
    // the tile of the ROWLANES mapping: at most 64 columns of 32 rows
    static constexpr int kCols = GroupShape<K>::kWeights < 64 ? GroupShape<K>::kWeights : 64;
    static constexpr int kStoreBytes = 32 * 2 * kCols;
    // 16-byte chunk c of tile row r lives at chunk swz(r, c) of that row
    __device__ static __forceinline__ uint32_t swz(uint32_t r, uint32_t c) {
        return kChunks == 4 ? (c ^ ((r >> 1) & 3u)) : (c ^ (r & 7u));
    }
};

template <int CODE, int K, bool ROWLANES>
__global__ void __launch_bounds__(kDecThreads, 1) decompress_kernel(const DecParams p, const __grid_constant__ CUtensorMap out_map) {
    using G = GroupShape<K>;
    using T = DecTile<K>;
    constexpr int P = G::P;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t s0 = smem_addr(smem_raw);
    uint32_t lut_tab, tiles;
    if (CODE == RPTC_CODE_HASH) {
        lut_tab = kHashLutWindow;
        tiles = kHashLutWindow + kHashLutBytes;
    } else {
        lut_tab = s0;
        tiles = (s0 + lut_bytes<CODE>(p.L, p.S) + 1023u) & ~1023u;       // the swizzle pattern repeats every 1024 bytes
    }
    const uint32_t tile = tiles + (uint32_t)warp * (ROWLANES ? T::kStoreBytes : T::kBytes);
    __shared__ __align__(8) unsigned long long table_bar;
    if (CODE == RPTC_CODE_LUT) {                                          // a plain image of the codebook: one bulk copy
        if (threadIdx.x == 0) {
            const uint32_t bar = smem_addr(&table_bar);
            mbar_init(bar, 1);
            mbar_fence_init();
            mbar_expect_tx(bar, 2u << p.L);
            bulk_g2s(lut_tab, p.lut, 2u << p.L, bar);
        }
    } else {
        lut_fill<CODE>(lut_tab, p.lut, p.L, p.S);
    }
    const Lut<CODE> lut = lut_view<CODE>(lut_tab, p.L, p.S);
    pdl_allow_next_grid();
    pdl_wait_prior_grids();
    __syncthreads();
    if (CODE == RPTC_CODE_LUT && !mbar_wait(smem_addr(&table_bar), 0, p.status)) return;

    const int nwarps = blockDim.x >> 5;
    const int32_t ng = p.n_groups;
    const int32_t ngb = (ng + 31) >> 5;                                   // 32-group blocks per row (!ROWLANES)
    const int64_t Ttot = ROWLANES ? (p.m >> 5) * (int64_t)ng : p.m * (int64_t)ngb;
    // ROWLANES: an equal range of tasks per CTA, which its warps take in turn, so that at any time the CTA writes 32 rows
    // of a few thousand adjacent columns (a range per warp writes 128 bytes here and there: 120 us for 8192 x 28672 with
    // the HASH code).  !ROWLANES: an equal range per warp, whose tasks are whole pieces of a row anyway.
    const int64_t part = ROWLANES ? blockIdx.x : (int64_t)blockIdx.x * nwarps + warp, parts = ROWLANES ? gridDim.x : (int64_t)gridDim.x * nwarps;
    const int64_t f0 = Ttot * part / parts + (ROWLANES ? warp : 0), f1 = Ttot * (part + 1) / parts;
    const int32_t f_step = ROWLANES ? nwarps : 1;

    // (outer, inner) = (row block, group) or (row, 32-group block); advanced without divisions
    const int32_t inner_n = ROWLANES ? ng : ngb;
    int64_t outer = (f0 < f1) ? f0 / inner_n : 0;
    int32_t inner = (f0 < f1) ? (int32_t)(f0 - outer * inner_n) : 0;

    // the word in front of a group of a row
    auto history = [&](int32_t g, int64_t row) -> uint32_t {
        if (g == 0) return p.carry_in ? __ldg(p.carry_in + row) : 0u;
        return __ldg(reinterpret_cast<const uint32_t *>(p.codes + unit_index(p.st, (int64_t)g * P - 1, row)) + 3);
    };
    uint32_t wnext[G::kWords], before_next = 0;
    auto load_group = [&](int64_t o, int32_t in) {
        const int64_t row = ROWLANES ? (o << 5) + lane : o;
        const int32_t g = ROWLANES ? in : in * 32 + lane;
#pragma unroll
        for (int k = 0; k < P; ++k) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (g < ng) v = ldg128_stream(p.codes + unit_index(p.st, (int64_t)g * P + k, row));
            wnext[4 * k] = v.x, wnext[4 * k + 1] = v.y, wnext[4 * k + 2] = v.z, wnext[4 * k + 3] = v.w;
        }
        if (ROWLANES || lane == 0) before_next = history(g, row);      // !ROWLANES: the other lanes ask the lane to their left
    };
    if (f0 < f1) load_group(outer, inner);

    for (int64_t f = f0; f < f1; f += f_step) {
        const int64_t o = outer;
        const int32_t in = inner;
        const int64_t row = ROWLANES ? (o << 5) + lane : o;
        const int32_t g = ROWLANES ? in : in * 32 + lane;
        const bool active = g < ng;
        inner += f_step;
        while (inner >= inner_n) {
            inner -= inner_n;
            ++outer;
        }
        uint32_t w[G::kWords], halo = before_next;
#pragma unroll
        for (int k = 0; k < G::kWords; ++k) w[k] = wnext[k];
        if (f + f_step < f1) load_group(outer, inner);         // next task's codes are in flight while this one decodes

        const uint32_t lastw = w[G::kWords - 1];
        if (!ROWLANES) {
            const uint32_t left = __shfl_up_sync(0xFFFFFFFFu, lastw, 1);
            if (lane > 0) halo = left;
        }
        if (K == 2 && p.quirk != RPTC_QUIRK_NONE && (g & 31) == 0) {
            if (p.quirk == RPTC_QUIRK_K2_LANE0_CARRY) halo = lastw;
            else if (g > 0) halo >>= 16;
        }

        if (ROWLANES) {
            constexpr int kSub = G::kWeights / T::kCols, kSubPairs = T::kCols / 2;
            uint32_t R[2 * G::kWords];
            make_windows<K>(w, halo, R);
#pragma unroll
            for (int h = 0; h < kSub; ++h) {
                uint32_t buf[kSubPairs];
#pragma unroll
                for (int pi = 0; pi < kSubPairs; ++pi) buf[pi] = decode_pair_bits<CODE, K>(R, lut, h * kSubPairs + pi);
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the tile has been read out
                __syncwarp();
                const uint32_t my_row = tile + (uint32_t)lane * (2 * T::kCols);
#pragma unroll
                for (int c = 0; c < T::kCols / 8; ++c) {
                    const uint32_t at = T::kCols == 64 ? (uint32_t)c ^ (lane & 7u) : (uint32_t)c ^ ((lane >> 1) & 3u);
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(my_row + 16u * at), "r"(buf[4 * c]), "r"(buf[4 * c + 1]),
                                 "r"(buf[4 * c + 2]), "r"(buf[4 * c + 3])
                                 : "memory");
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    tma_store_2d(&out_map, g * G::kWeights + h * T::kCols, (int)(o << 5), tile);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
            continue;
        }
        // decode into this lane's row of the tile
        if (active) {
            const uint32_t my_row = tile + (uint32_t)lane * T::kRowBytes;
            uint32_t buf[4];
            decode_group<CODE, K>(w, halo, lut, [&](int pi, __half2 wp) {
                buf[pi & 3] = half2_as_u32(wp);
                if ((pi & 3) == 3) {
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(my_row + 16u * T::swz(lane, pi >> 2)), "r"(buf[0]),
                                 "r"(buf[1]), "r"(buf[2]), "r"(buf[3])
                                 : "memory");
                }
            });
        }
        __syncwarp();
        // copy the tile out: chunk q = i*32 + lane  ->  tile row q / kChunks, chunk q % kChunks
#pragma unroll
        for (int i = 0; i < T::kChunks; ++i) {
            const uint32_t q = (uint32_t)i * 32u + lane;
            const uint32_t r = q / T::kChunks, c = q % T::kChunks;
            __half *dst;
            bool ok;
            const int32_t gr = in * 32 + (int32_t)r;
            dst = p.out + row * p.ld_out + (int64_t)gr * G::kWeights + 8 * c;
            ok = gr < ng;
            if (ok) {
                const uint4 v = lds128(tile + r * T::kRowBytes + 16u * T::swz(r, c));
                asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
            }
        }
        __syncwarp();
    }
    if (ROWLANES && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// `smem` is the table's share; the per-warp tiles are added here, with fewer warps when they do not fit.
template <int CODE, int K, bool ROWLANES>
static int launch_dec(const DecParams &p, size_t smem, cudaStream_t stream) {
    using T = DecTile<K>;
    const size_t tile = ROWLANES ? T::kStoreBytes : T::kBytes;
    int warps = kDecThreads / 32;
    while (warps > 2 && smem + 1024 + warps * tile > 226 * 1024) --warps;
    smem += 1024 + warps * tile;
    CUtensorMap map = {};
    if (ROWLANES) {
        if (int e = encode_map(map, p.out, p.n_groups * (int64_t)GroupShape<K>::kWeights, p.m, p.ld_out, 32, T::kCols)) return e;
    }
    static SmemOptIn opted;
    auto kern = decompress_kernel<CODE, K, ROWLANES>;
    if (int e = allow_max_smem(kern, opted, 226 * 1024)) return e;
    return launch(kern, dim3(num_sms()), dim3(32 * warps), smem, stream, p, map);
}

template <int CODE, int K>
static int dispatch_dec(const DecParams &p, bool rowlanes, size_t smem, cudaStream_t stream) {
    return rowlanes ? launch_dec<CODE, K, true>(p, smem, stream) : launch_dec<CODE, K, false>(p, smem, stream);
}

int check_format(const rptc_format *f);   // api.cu

}  // namespace rptc

using namespace rptc;

extern "C" int rptc_decompress(const void *codes, const void *lut, const uint32_t *carry_in, void *out, int64_t ld_out,
                               int64_t m, int64_t n, const rptc_format *fmt, rptc_stream_t stream) {
    if (!codes || !lut || !out || !fmt) return RPTC_ERR_ARG;
    if (int e = check_format(fmt)) return e;
    const int K = fmt->K;
    const int P = (K == 3) ? 3 : 1;
    const int wpg = 128 * P / K;
    if (m <= 0 || n <= 0 || (m % 32) || (n % wpg) || ld_out < n) return RPTC_ERR_SHAPE;
    if (m > (int64_t(1) << 30) || n > (int64_t(1) << 30)) return RPTC_ERR_TOO_LARGE;
    const int64_t n_units = n / wpg * P;
    if (fmt->layout == RPTC_LAYOUT_CHUNKED && (n_units % 32)) return RPTC_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(codes) & 15) || (reinterpret_cast<uintptr_t>(lut) & 15) ||
        (reinterpret_cast<uintptr_t>(out) & 15) || (ld_out % 8))
        return RPTC_ERR_ALIGN;
    if (int e = rptc_check_device()) return e;

    DecParams p;
    p.codes = static_cast<const uint4 *>(codes);
    p.st = unit_strides(fmt->layout, m, n_units);
    p.lut = static_cast<const __half *>(lut);
    p.carry_in = carry_in;
    p.out = static_cast<__half *>(out);
    p.ld_out = ld_out;
    p.m = m;
    p.n_groups = (int32_t)(n / wpg);
    p.L = fmt->L;
    p.S = fmt->S;
    p.quirk = fmt->quirk;
    p.status = device_status_word();
    if (!p.status) return RPTC_ERR_CUDA;
    const bool rowlanes = fmt->layout == RPTC_LAYOUT_UNITMAJOR || fmt->layout == RPTC_LAYOUT_TILED;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    size_t smem;
    switch (fmt->code) {
        case RPTC_CODE_LUT:
            smem = (size_t(2) << fmt->L) + 128;
            if (K == 2) return dispatch_dec<RPTC_CODE_LUT, 2>(p, rowlanes, smem, s);
            if (K == 3) return dispatch_dec<RPTC_CODE_LUT, 3>(p, rowlanes, smem, s);
            return dispatch_dec<RPTC_CODE_LUT, 4>(p, rowlanes, smem, s);
        case RPTC_CODE_HASH:
            smem = kHashLutWindow + kHashLutBytes;
            return dispatch_dec<RPTC_CODE_HASH, 2>(p, rowlanes, smem, s);
        case RPTC_CODE_LITE:
            smem = (size_t(128) << fmt->S) + 128;
            if (K == 2) return dispatch_dec<RPTC_CODE_LITE, 2>(p, rowlanes, smem, s);
            return dispatch_dec<RPTC_CODE_LITE, 4>(p, rowlanes, smem, s);
    }
    return RPTC_ERR_UNSUPPORTED;
}
