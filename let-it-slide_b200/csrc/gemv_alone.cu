// One or two activation rows as the first kernel of a layer's call: the product makes the layer's input side itself, and leaves its sums for
// the output side to add up (gemv_rows.cuh, MODE 3 and 4).
#include "gemv_rows.cuh"

namespace rptc {

struct AlonePlan {
    GemvSums sums;
    int ctas, slots;
    size_t smem;
    bool ex_on_ring;
};
static bool alone_plan(AlonePlan &a, int64_t m, int64_t n, int64_t rows, int block, const Banks &banks, const rptc_format &f) {
    if (rows < 1 || rows > 2 || f.layout != RPTC_LAYOUT_TILED || f.quirk != RPTC_QUIRK_NONE || (f.K != 2 && f.K != 4) || n % 64) return false;
    // The transform in every CTA pays for one short row, whose call is bound by the host's launches: 11.0 us a call with a kernel in front, 9.1
    // (3072 x 2304) and 10.8 (4096 x 4096, from 12.8) without; on the device alone 7.2 and 8.6, 8.9 and 9.2, since nothing but the
    // wait may lie in front of the first loads.  Two rows of 4096: 11.1 against 12.0; 4096 x 5120: 11.0 and 12.7.
    if (block != kNoTransform && (rows > 1 || n > 4096 || block < 8 || block > 4096 || (block & (block - 1)) || n % (block < 256 ? 256 : block))) return false;
    const int64_t units = n / (128 / f.K), blocks = m / 32, total = blocks * units;
    if (total >= (int64_t(1) << 31)) return false;
    int64_t ctas = num_sms() / banks.banks > 0 ? num_sms() / banks.banks : 1;
    if (ctas > total / 2) ctas = total / 2;                     // every CTA has a granule
    if (ctas < 1) return false;
    a.ctas = (int)ctas;
    a.sums.per = (uint32_t)(total / ctas);
    a.sums.extra = (uint32_t)(total % ctas);
    a.sums.paired = (uint32_t)(blocks / 2 * units);
    a.sums.units = (uint32_t)units;
    a.sums.tile_rows = 64;
    a.sums.token_tiles = 1;
    a.sums.n_cols = 1;
    if ((a.sums.per + 1 + kGemvWarps - 1) / kGemvWarps + 1 > units) return false;      // two runs a warp at most
    a.slots = (int)((2 * units - 1 + a.sums.per - 1) / a.sums.per) + 1;
    a.smem = fixed_smem(f, kRingBytes + kGemvWarps * 64 * (size_t)rows * 4) + (size_t)rows * n * 2;
    const size_t ex = block > 256 ? 2 * kUnitFloats * sizeof(float) : 0;
    a.ex_on_ring = a.smem + ex > kMaxSmem;
    if (!a.ex_on_ring) a.smem += ex;
    return a.smem <= kMaxSmem;
}
bool gemv_alone_takes(int64_t m, int64_t n, int64_t rows, int block, const Banks &banks, const rptc_format &f) {
    AlonePlan a;
    return alone_plan(a, m, n, rows, block, banks, f);
}
int64_t gemv_alone_partials(int64_t m, int64_t n, int64_t rows, const Banks &banks, const rptc_format &f) {
    AlonePlan a;
    return alone_plan(a, m, n, rows, kNoTransform, banks, f) ? a.slots * rows * banks.banks * m : 0;
}
int gemv_alone(const void *codes, const void *lut, const uint32_t *carry_in, const GemvInput &in, float *partial, int64_t m, int64_t n, int64_t rows,
               const Banks &banks, const rptc_format &f, cudaStream_t stream, GemvSums *sums) {
    AlonePlan a;
    if (!alone_plan(a, m, n, rows, in.scales_in ? kNoTransform : in.block, banks, f)) return RPTC_ERR_UNSUPPORTED;
    GemvAlone p = {};
    p.codes = static_cast<const uint4 *>(codes);
    p.lut = static_cast<const __half *>(lut);
    p.carry_in = carry_in;
    p.acc = partial;
    p.ld_acc = banks.banks * m;
    p.m = m;
    p.n = n;
    p.n_units = p.seg_units = (int32_t)(n / (128 / f.K));
    p.L = f.L;
    p.S = f.S;
    p.status = device_status_word();
    if (!p.status) return RPTC_ERR_CUDA;
    p.in = in;
    a.sums.plane = rows * banks.banks * m;
    p.sums = *sums = a.sums;
    p.lut_stride = banks.lut_stride;
    p.ex_on_ring = a.ex_on_ring;
    const dim3 grid((unsigned)a.ctas, (unsigned)banks.banks);
    if (in.scales_in) {
        if (f.code != RPTC_CODE_LUT || f.K != 2) return RPTC_ERR_UNSUPPORTED;
        return rows == 1 ? launch_gemv_rows<RPTC_CODE_LUT, 2, 1, 3>(p, a.smem, stream, grid) : launch_gemv_rows<RPTC_CODE_LUT, 2, 2, 3>(p, a.smem, stream, grid);
    }
    return with_code(f, [&](auto code, auto k) {
        return launch_gemv_rows<code.value, k.value, 1, 4>(p, a.smem, stream, grid);
    });
}

}  // namespace rptc
