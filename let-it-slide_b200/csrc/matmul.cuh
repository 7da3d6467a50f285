// The fused matrix products as the library's own entry points call them (host side): the checks of arguments are done,
// and the rows of W may come in banks that each have a lookup table of their own.
#pragma once
#include "common.cuh"
#include "waited_timer.cuh"

namespace rptc {

// W is `banks` groups of `m` rows (m a multiple of 32, TILED codes one bank after the other); bank b decodes through
// lut + b * lut_stride.
struct Banks {
    int32_t banks = 1;
    int64_t lut_stride = 0;      // fp16 elements
    bool may_split = true;       // false: every sum is one chain along the reduction, whatever the number of tokens
};

// Columns of y per bank: a bank's rows rounded up to whole tiles.
int64_t gemm_bank_columns(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f);
// y[t][bank * gemm_bank_columns + row] = fp16(sum_c x[t][c] W[bank][row][c]); columns beyond a bank's m rows hold no
// result.  Shapes and alignments as rptc_gemm's, with any m % 32 == 0; banks == 1: ld_y >= m,
// nothing is stored behind column m.
int gemm_banked(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x, void *y, int64_t ld_y, int64_t m,
                int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f, cudaStream_t stream);
// The estimate that gemm_banked's choice of tiles rests on, microseconds; 0 where it takes no such product.
double gemm_us(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f);
// acc[b][bank * m + row] += sum_c W[bank][row][c] x[b][c] for any number of activation rows that gemv_few_takes says yes to (up to
// kFewOwnTokens whatever the shape).
constexpr int64_t kFewOwnTokens = 96;
bool gemv_few_takes(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f, const void *x, int64_t ld_x);
// Ordered sums: every sum is taken in the same order on every run, so that equal calls give equal bits.  `partial` is room for
// gemv_few_partials fp32 values (16-byte aligned; ld_acc a multiple of 4), and acc = instead of +=.  Where that is 0 the sums meet in acc as
// they do without (+=, from zeros): there are two of them at most, and a + b is b + a.
int64_t gemv_few_partials(int64_t m, int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f);
// With `parts` the caller adds them up: partial[slot][token][ld_acc] for slot < parts->count(row, token), nothing in acc.
struct GemvSums;
int gemv_few(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x, float *acc, int64_t ld_acc, int64_t m,
             int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f, cudaStream_t stream, bool ordered = false, float *partial = nullptr,
             GemvSums *parts = nullptr);
// The same for any number of activation rows (TILED codes, no quirk, no carry): gemv_few where it takes them, else the
// lane-per-row kernel for one or two rows at a time.
int gemv_banked(const void *codes, const void *lut, const void *x, int64_t ld_x, float *acc, int64_t ld_acc, int64_t m, int64_t n, int64_t tokens,
                const Banks &banks, const rptc_format &f, cudaStream_t stream, bool ordered = false, float *partial = nullptr);

// ---- one or two activation rows, as the first kernel of a layer's call (gemv_alone.cu) ----
// The input side that the product makes in its CTAs.
struct GemvInput {
    const void *x;                       // [batch][n]: fp16, or with scales_in fp16, bf16, fp32 (dtype 0, 1, 2)
    const float *scales_in, *biases_in;  // fp32 [n]: x * scales_in goes in, and sums[row] = (sum of x, <biases_in, x>) comes out
    float2 *sums;
    const __half *signs;                 // [n]: H(signs * x) * norm over blocks of `block` goes in
    int32_t dtype, block;
    float norm;
};
// Where a product's sums are: a value's as many as there are CTAs that meet in its tile, `plane` values apart, in order.  The tiles' granules
// (steps along the rows), laid end to end, are cut into ranges of equal weight.  gemv_alone: a tile is a pair of 32-row blocks, a granule
// of which counts two, that of an odd last block one.  gemv_few: tiles of rows x tokens, all granules count one.
struct GemvSums {
    int64_t plane;
    uint32_t per, extra;                 // weight of a CTA's range, and how many CTAs have one more
    uint32_t paired, units;              // how many granules count two; granules of a tile
    int32_t tile_rows, token_tiles, n_cols;      // tiles of the same rows, n_cols tokens each
#ifdef __CUDACC__
    __device__ __forceinline__ uint32_t begin(uint32_t cta) const { return cta * per + min(cta, extra); }
    __device__ __forceinline__ uint32_t weight(uint32_t granule) const { return granule + min(granule, paired); }
    __device__ __forceinline__ uint32_t granule_at(uint32_t w) const { return w >= 2 * paired ? w - paired : (w + 1) >> 1; }
    __device__ __forceinline__ uint32_t cta_of(uint32_t w) const {
        return w < extra * (per + 1) ? w / (per + 1) : extra + (w - extra * (per + 1)) / per;
    }
    // how many there are of a bank's row and a token
    __device__ __forceinline__ int count(uint32_t row, uint32_t token) const {
        const uint32_t g = (row / (uint32_t)tile_rows * (uint32_t)token_tiles + (token_tiles > 1 ? token / (uint32_t)n_cols : 0u)) * units;
        return (int)(cta_of(weight(g + units - 1)) - cta_of(weight(g))) + 1;
    }
#endif
};
// Whether gemv_alone takes the layer (`block`: of the Hadamard transform, kNoTransform with scales_in), and the fp32 values of room for its sums.
constexpr int kNoTransform = -1;
bool gemv_alone_takes(int64_t m, int64_t n, int64_t rows, int block, const Banks &banks, const rptc_format &f);
int64_t gemv_alone_partials(int64_t m, int64_t n, int64_t rows, const Banks &banks, const rptc_format &f);
// partial[slot][row of x][bank * m + row] for slot < sums.count(row)
int gemv_alone(const void *codes, const void *lut, const uint32_t *carry_in, const GemvInput &in, float *partial, int64_t m, int64_t n, int64_t rows,
               const Banks &banks, const rptc_format &f, cudaStream_t stream, GemvSums *sums);

// ---- a matvec whose caller waits for it (gemv_whole.cu) ----
int validate_gemv_args(const void *codes, const void *lut, const void *x, int64_t ld_x, const float *acc, int64_t ld_acc, int64_t m, int64_t n, int batch,
                       int x_order, const rptc_format *fmt);
// y = (or +=) W x, one row, for codes whose units of a row lie together (ROWMAJOR, CHUNKED) and rows that fit into shared memory and are gathered
// cheaply enough (gemv_whole_takes).  The arguments have been checked, and y lies over none of them.
bool gemv_whole_takes(int64_t n, int x_order, const rptc_format &f);
int gemv_whole(const void *codes, const void *lut, const void *x, void *y, int64_t m, int64_t n, int x_order, int accumulate, const rptc_format &f,
               const DeviceTimer &timer, cudaStream_t stream);

}  // namespace rptc
