// Products of many rows by pairs of SMs (gemm_pair.cu).
#pragma once

#include "common.cuh"
#include "gemm_plan.cuh"

namespace lumen {

struct GemmPairArgs {
    const __nv_bfloat16 *a_hi = nullptr, *a_lo = nullptr;  // activations [M, K]
    const __nv_bfloat16 *w_hi = nullptr, *w_lo = nullptr;  // weights [N, K]; w_lo null: bf16 weights
    size_t M = 0, K = 0, N = 0;
    float *c = nullptr;               // [M, N], or [splits][M][N]
    const float *residual = nullptr;  // one slice only
    // Set: the weights are gate and up rows of N / 2 each (a multiple of 8), and the bf16 split of silu(gate) * up is stored
    // here, [M, N / 2], instead of c.
    __nv_bfloat16 *out_hi = nullptr, *out_lo = nullptr;
};
int launch_gemm_pair(lumen_ctx *ctx, const GemmPairArgs &g, const GemmPairPlan &plan, cudaStream_t s);

}  // namespace lumen
