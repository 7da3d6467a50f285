// The fused matrix products as the library's own entry points call them (host side): the checks of arguments are done,
// and the rows of W may come in banks that each have a lookup table of their own.
#pragma once
#include "common.cuh"

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
int gemv_few(const void *codes, const void *lut, const uint32_t *carry_in, const void *x, int64_t ld_x, float *acc, int64_t ld_acc, int64_t m,
             int64_t n, int64_t tokens, const Banks &banks, const rptc_format &f, cudaStream_t stream, bool ordered = false, float *partial = nullptr);
// The same for any number of activation rows (TILED codes, no quirk, no carry): gemv_few where it takes them, else the
// lane-per-row kernel for one or two rows at a time.
int gemv_banked(const void *codes, const void *lut, const void *x, int64_t ld_x, float *acc, int64_t ld_acc, int64_t m, int64_t n, int64_t tokens,
                const Banks &banks, const rptc_format &f, cudaStream_t stream, bool ordered = false, float *partial = nullptr);

}  // namespace rptc
