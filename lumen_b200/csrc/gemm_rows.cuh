// Products of at most kGemmRowsMax rows with their epilogues (gemm_rows.cu).
#pragma once

#include "common.cuh"

namespace lumen {

constexpr int kGemmRowsMax = 64;

struct GemmRowsArgs {
    enum Epi {
        kStore = 0,     // c = A . W^T
        kResidual = 1,  // x += A . W^T; (hi, lo) = pair of x * gain; ss_out[tile of 128 columns][64]: sums of squares of x
        kSwiglu = 2     // W: N / 2 rows of gate, then of up; (hi, lo) = pair of silu(gate) * up, [M, N / 2]
    } epi = kStore;
    int M = 0, N = 0, K = 0;
    const __nv_bfloat16 *x_hi = nullptr, *x_lo = nullptr;  // [M, K]
    const __nv_bfloat16 *w_hi = nullptr, *w_lo = nullptr;  // [N, K]; w_lo null: bf16 weights
    // Rows whose RMSNorm is still owed (the gains are in the pair): the product is multiplied by 1 / rms of the row, from n_ss sums of
    // squares (layout of ss_out).  n_ss == 0: none.
    const float *ss_in = nullptr;
    int n_ss = 0;
    float eps = 0.f;
    float *c = nullptr, *x = nullptr, *ss_out = nullptr;
    const float *gain = nullptr;
    __nv_bfloat16 *hi = nullptr, *lo = nullptr;
    int *advance = nullptr;  // kResidual: a number that grows by one (the length of the cache that the kernel before has read)
};
bool gemm_rows_usable(lumen_dtype wdt, size_t M, size_t K, size_t N, const void *w);
size_t gemm_rows_ss_floats(size_t N);
int launch_gemm_rows(lumen_ctx *ctx, const GemmRowsArgs &a, cudaStream_t s);
// Operands of a chain's first product: (hi, lo) = pair of x * gain, ss[row] = sum of squares (n_ss = 1).  dim: a multiple of 4.
int launch_rows_start(lumen_ctx *ctx, const float *x, const float *gain, size_t rows, size_t dim, __nv_bfloat16 *hi, __nv_bfloat16 *lo, float *ss,
                      cudaStream_t s);

}  // namespace lumen
