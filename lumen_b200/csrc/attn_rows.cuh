// Decode attention of a batched step (attn_rows.cu).
#pragma once

#include "attn_plan.cuh"
#include "common.cuh"

namespace lumen {

struct AttnRowsArgs {
    const float *qkv = nullptr;  // [B, stride]: q heads, k heads, v heads of one position
    size_t stride = 0;
    float *k_cache = nullptr, *v_cache = nullptr;  // [B, Hkv, max_seq, D]
    const int *d_len = nullptr;                    // read, not advanced
    size_t max_seq = 0;
    const float *cos_t = nullptr, *sin_t = nullptr, *q_norm = nullptr, *k_norm = nullptr;
    float norm_eps = 0.f, scale = 0.f;
    __nv_bfloat16 *out_hi = nullptr, *out_lo = nullptr;  // [B, Hq * D]
    DeviceStatus *status = nullptr;
};
// `splits`: of attn_rows_splits, not 0.
int launch_attn_rows(lumen_ctx *ctx, const AttnRowsArgs &a, size_t B, size_t Hq, size_t Hkv, size_t D, int splits, cudaStream_t s);

}  // namespace lumen
