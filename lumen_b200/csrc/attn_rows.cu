// Decode attention of a batched step (one new position per sequence; self_attention.rs:141-297 of the reference): rotate the new k
// into cache row `len`, copy v, rotate q, then softmax(q.K^T * scale).V over rows 0..=len with 1/(l + 1e-9).
//
// A CTA of four warps serves one KV head of one sequence (all query heads of its group), or, as one of a cluster, a part of its
// context; the parts meet over distributed shared memory and the result leaves as the bf16 pair that the output projection reads.
// What bounds it: latency.  Cached rows do not depend on this step, so their copies (bulk copies of 4 KB of K and of V, a tile of each
// per warp; the rows behind them go to the L2) are under way before the kernel waits for the projections; then two or four
// lanes form the scores of one row for all heads of the group from 16-byte reads in an order rotated by row (no bank
// conflicts), and the lanes share out the context's elements for P.V.  Some 40 KB of shared memory and 128 threads: 512 CTAs (64 sequences of
// eight KV heads) are resident at once, and the products before and after find room beside them.  Steps of two Qwen3-8B layers with 64
// sequences at 60 / 250 / 1000 / 4096 positions: 518 / 569 / 719 / 1257 us (rows beyond 1000 positions at 6.0 TB/s), with the general kernel and its merge
// 571 / 619 / 785 / 1413.  Which lengths come here: attn_plan.cuh.
#include <cooperative_groups.h>

#include "attn_decode.cuh"
#include "attn_rows.cuh"
#include "tc_common.cuh"

namespace lumen {
namespace {

namespace cg = cooperative_groups;
constexpr int kArWarps = 4, kArThreads = 32 * kArWarps;

template <int D, int G>
struct ArGeom {
    static constexpr int kRows = 1024 / D;           // rows of a tile: 4 KB of K and 4 KB of V
    static constexpr int kLanes = 32 / kRows;        // lanes that share a row's score
    static constexpr int kVec = D / 4 / kLanes;      // 16-byte steps of a lane through a row
    static constexpr int kEl = D / 32;               // elements of the context per lane
    // tiles (afterwards the warps' contexts) | q | new k | new v | weights | per warp: maxima, sums | of the CTA: maxima, sums, context
    static constexpr int kTiles = kArWarps * 2 * kRows * D;
    static constexpr int kFloats = kTiles + G * D + 2 * D + kArWarps * kRows * G + 2 * kArWarps * G + 2 * G + G * D;
    static_assert(kArWarps * G * D <= kTiles, "");
};

__device__ __forceinline__ void bulk_rows(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(tc::saddr(dst)), "l"(src), "r"(bytes), "r"(tc::saddr(bar)) : "memory");
}
__device__ __forceinline__ void prefetch_rows(const void *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

// grid (splits, Hkv, B), clusters of (splits, 1, 1)
template <int D, int G>
__global__ void __launch_bounds__(kArThreads) attn_rows_kernel(const AttnRowsArgs p) {
    using A = ArGeom<D, G>;
    constexpr int TR = A::kRows;
    extern __shared__ __align__(128) float ar_smem[];
    float *tiles = ar_smem, *qs = tiles + A::kTiles, *knew = qs + G * D, *vnew = knew + D, *wsoft = vnew + D;
    float *wm = wsoft + kArWarps * TR * G, *wl = wm + kArWarps * G, *cm = wl + kArWarps * G, *cl = cm + G, *cctx = cl + G;
    __shared__ uint64_t kbar[kArWarps], vbar[kArWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int split = blockIdx.x, nsplit = gridDim.x, hk = blockIdx.y, b = blockIdx.z, hkv = gridDim.y;
    pdl_launch();
    if (tid == 0) {
        for (int w = 0; w < kArWarps; ++w) {
            tc::bar_init(&kbar[w], 1);
            tc::bar_init(&vbar[w], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int past = *p.d_len, total = past + 1, chunk = (total + nsplit - 1) / nsplit;
    const int j0 = split * chunk, jc = min(min(total, j0 + chunk), past);  // cached rows [j0, jc)
    const bool owns_new = past >= j0 && past < j0 + chunk;
    const size_t head = (size_t)b * hkv + hk;
    float *kbase = p.k_cache + head * p.max_seq * D, *vbase = p.v_cache + head * p.max_seq * D;
    float *kt = tiles + warp * 2 * TR * D, *vt = kt + TR * D;
    int k_issued = 0, v_issued = 0;
    auto fetch = [&](float *dst, const float *base, int j, uint64_t *bar, int &issued) {
        if (j >= jc) return;
        if (lane == 0) {
            const uint32_t bytes = (uint32_t)min(TR, jc - j) * D * 4;
            tc::bar_expect(bar, bytes);
            bulk_rows(dst, base + (size_t)j * D, bytes, bar);
        }
        ++issued;
    };
    const int step = kArWarps * TR;
    int j = j0 + warp * TR;
    fetch(kt, kbase, j, &kbar[warp], k_issued);
    fetch(vt, vbase, j, &vbar[warp], v_issued);
    if (tid == 0 && j0 + step < jc) {  // the rest of the rows: to the L2
        prefetch_rows(kbase + (size_t)(j0 + step) * D, (uint32_t)(jc - j0 - step) * D * 4);
        prefetch_rows(vbase + (size_t)(j0 + step) * D, (uint32_t)(jc - j0 - step) * D * 4);
    }
    // ---- this step's q, k and v: a lane holds the elements lane, lane + 32, ... of a head; what a warp needs is requested at once ----
    constexpr int E = D / 32, HV = (G + 1 + kArWarps - 1) / kArWarps;  // q heads and the new k, dealt out over the warps
    float co[E / 2], sn[E / 2], q_gain[E], k_gain[E];
#pragma unroll
    for (int t = 0; t < E / 2; ++t) {
        co[t] = __ldg(p.cos_t + (size_t)past * (D / 2) + lane + 32 * t);
        sn[t] = __ldg(p.sin_t + (size_t)past * (D / 2) + lane + 32 * t);
    }
#pragma unroll
    for (int t = 0; t < E; ++t) {
        q_gain[t] = p.q_norm ? __ldg(p.q_norm + lane + 32 * t) : 1.f;
        k_gain[t] = p.k_norm ? __ldg(p.k_norm + lane + 32 * t) : 1.f;
    }
    pdl_wait();
    const float *row = p.qkv + (size_t)b * p.stride;
    float hv[HV][E], vn[E];
#pragma unroll
    for (int u = 0; u < HV; ++u) {
        const int h = warp + u * kArWarps;
        if (h > G) continue;
        const float *src = row + (size_t)(h < G ? hk * G + h : hkv * G + hk) * D;
#pragma unroll
        for (int t = 0; t < E; ++t) hv[u][t] = __ldcg(src + lane + 32 * t);
    }
    if (warp == kArWarps - 1)
#pragma unroll
        for (int t = 0; t < E; ++t) vn[t] = __ldcg(row + (size_t)(hkv * G + hkv + hk) * D + lane + 32 * t);
#pragma unroll
    for (int u = 0; u < HV; ++u) {
        const int h = warp + u * kArWarps;
        if (h > G) continue;
        const bool is_k = h == G;
        if (is_k ? p.k_norm != nullptr : p.q_norm != nullptr) {  // RMSNorm of the head (rms_norm.rs:49-56)
            float ss = 0.f;
#pragma unroll
            for (int t = 0; t < E; ++t) ss = fmaf(hv[u][t], hv[u][t], ss);
            ss = attn_warp_sum(ss);
            const float inv = __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(ss, (float)D), p.norm_eps)));
#pragma unroll
            for (int t = 0; t < E; ++t) hv[u][t] = __fmul_rn(__fmul_rn(hv[u][t], inv), is_k ? k_gain[t] : q_gain[t]);
        }
#pragma unroll
        for (int t = 0; t < E / 2; ++t) {  // encoding.rs:195-203
            const float x1 = hv[u][t], x2 = hv[u][t + E / 2];
            hv[u][t] = __fsub_rn(__fmul_rn(x1, co[t]), __fmul_rn(x2, sn[t]));
            hv[u][t + E / 2] = __fadd_rn(__fmul_rn(x2, co[t]), __fmul_rn(x1, sn[t]));
        }
        if (is_k && !owns_new) continue;
#pragma unroll
        for (int t = 0; t < E; ++t) {
            (is_k ? knew : qs + h * D)[lane + 32 * t] = hv[u][t];
            if (is_k) kbase[(size_t)past * D + lane + 32 * t] = hv[u][t];
        }
    }
    if (owns_new && warp == kArWarps - 1)
#pragma unroll
        for (int t = 0; t < E; ++t) {
            vnew[lane + 32 * t] = vn[t];
            vbase[(size_t)past * D + lane + 32 * t] = vn[t];
        }
    __syncthreads();
    float m[G], l[G], ctx[G][A::kEl];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        m[g] = -INFINITY;
        l[g] = 0.f;
#pragma unroll
        for (int i = 0; i < A::kEl; ++i) ctx[g][i] = 0.f;
    }
    const int r_l = lane % TR, part = lane / TR, e0 = lane * A::kEl;
    const float4 *q4 = reinterpret_cast<const float4 *>(qs) + part * A::kVec;
    float *ws = wsoft + warp * TR * G;
    bool alive = true;
    // The cached tiles of this warp, then, for the warp that has least to do, this token's row as a tile of one row.
    const int cached = jc > j ? (jc - j + step - 1) / step : 0;
    const bool takes_new = owns_new && warp == (max(jc - j0, 0) + TR - 1) / TR % kArWarps;
#pragma unroll 1
    for (int it = 0; it < cached + takes_new; ++it, j += step) {
        const bool fresh = it == cached;
        const int rows = fresh ? 1 : min(TR, jc - j);
        if (!fresh) alive = __all_sync(0xffffffffu, tc::bar_wait(&kbar[warp], (uint32_t)(it & 1), p.status, 570));
        if (!alive) break;
        float s[G];
#pragma unroll
        for (int g = 0; g < G; ++g) s[g] = 0.f;
        const float4 *k4 = reinterpret_cast<const float4 *>(fresh ? knew : kt) + min(r_l, rows - 1) * (D / 4) + part * A::kVec;
#pragma unroll 2
        for (int i = 0; i < A::kVec; ++i) {
            const int at = (i + r_l) % A::kVec;
            const float4 k = k4[at];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float4 q = q4[g * (D / 4) + at];
                s[g] = fmaf(q.w, k.w, fmaf(q.z, k.z, fmaf(q.y, k.y, fmaf(q.x, k.x, s[g]))));
            }
        }
        __syncwarp();
        fetch(kt, kbase, j + step, &kbar[warp], k_issued);
        float top[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
            for (int o = 16; o >= TR; o >>= 1) s[g] += __shfl_xor_sync(0xffffffffu, s[g], o);
            s[g] = r_l < rows ? __fmul_rn(s[g], p.scale) : -INFINITY;
            top[g] = s[g];
        }
#pragma unroll
        for (int o = TR / 2; o > 0; o >>= 1)
#pragma unroll
            for (int g = 0; g < G; ++g) top[g] = fmaxf(top[g], __shfl_xor_sync(0xffffffffu, top[g], o));
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float mn = fmaxf(m[g], top[g]), r = expf(m[g] - mn), w = expf(s[g] - mn);  // (a tile has a row: mn is finite)
            m[g] = mn;
            l[g] = fmaf(l[g], r, part == 0 ? w : 0.f);
            if (part == 0) ws[r_l * G + g] = w;
#pragma unroll
            for (int i = 0; i < A::kEl; ++i) ctx[g][i] *= r;
        }
        __syncwarp();
        if (!fresh) alive = __all_sync(0xffffffffu, tc::bar_wait(&vbar[warp], (uint32_t)(it & 1), p.status, 571));
        if (!alive) break;
        const float *v_tile = fresh ? vnew : vt;
#pragma unroll 2
        for (int r = 0; r < rows; ++r) {
            float v[A::kEl], w[G];
            if constexpr (A::kEl == 4) *reinterpret_cast<float4 *>(v) = *reinterpret_cast<const float4 *>(v_tile + r * D + e0);
            else *reinterpret_cast<float2 *>(v) = *reinterpret_cast<const float2 *>(v_tile + r * D + e0);
            if constexpr (G % 4 == 0) {
#pragma unroll
                for (int g = 0; g < G; g += 4) *reinterpret_cast<float4 *>(w + g) = *reinterpret_cast<const float4 *>(ws + r * G + g);
            } else {
#pragma unroll
                for (int g = 0; g < G; ++g) w[g] = ws[r * G + g];
            }
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int i = 0; i < A::kEl; ++i) ctx[g][i] = fmaf(w[g], v[i], ctx[g][i]);
        }
        __syncwarp();
        fetch(vt, vbase, j + step, &vbar[warp], v_issued);
    }
    if (!alive && lane == 0) {  // (bounded) let the copies in flight land
        const long long t0 = clock64();
        if (k_issued) while (!tc::bar_try(&kbar[warp], (uint32_t)(k_issued - 1) & 1) && clock64() - t0 < tc::kTcWaitCycles) {}
        if (v_issued) while (!tc::bar_try(&vbar[warp], (uint32_t)(v_issued - 1) & 1) && clock64() - t0 < tc::kTcWaitCycles) {}
    }
    __syncwarp();
    // ---- the warps' parts, then the cluster's ----
    __syncthreads();  // the tiles are no longer read
    float *wctx = tiles + warp * G * D;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int g = 0; g < G; ++g) l[g] += __shfl_xor_sync(0xffffffffu, l[g], o);
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (lane == 0) {
            wm[warp * G + g] = m[g];
            wl[warp * G + g] = l[g];
        }
#pragma unroll
        for (int i = 0; i < A::kEl; ++i) wctx[g * D + e0 + i] = ctx[g][i];
    }
    __syncthreads();
    auto put = [&](int idx, float c, float sum) {
        const float v = __fmul_rn(c, __fdiv_rn(1.0f, __fadd_rn(sum, 1e-9f)));
        const size_t at = (head * G) * D + idx;
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        p.out_hi[at] = h;
        p.out_lo[at] = __float2bfloat16_rn(v - __bfloat162float(h));
    };
#pragma unroll 1
    for (int idx = tid; idx < G * D; idx += kArThreads) {
        const int g = idx / D;
        float M = -INFINITY, L = 0.f, c = 0.f;
#pragma unroll
        for (int w = 0; w < kArWarps; ++w) M = fmaxf(M, wm[w * G + g]);
#pragma unroll
        for (int w = 0; w < kArWarps; ++w) {
            const float mw = wm[w * G + g], f = mw == -INFINITY ? 0.f : expf(mw - M);
            L = fmaf(wl[w * G + g], f, L);
            c = fmaf(tiles[(w * G) * D + idx], f, c);
        }
        if (nsplit == 1) {
            put(idx, c, L);
        } else {
            cctx[idx] = c;
            if (idx % D == 0) {
                cm[g] = M;
                cl[g] = L;
            }
        }
    }
    if (nsplit == 1) return;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int idx = split * kArThreads + tid; idx < G * D; idx += nsplit * kArThreads) {
        const int g = idx / D;
        float mr[8], lr[8], cr[8], M = -INFINITY, L = 0.f, c = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (r < nsplit) {
                mr[r] = *cluster.map_shared_rank(cm + g, r);
                lr[r] = *cluster.map_shared_rank(cl + g, r);
                cr[r] = *cluster.map_shared_rank(cctx + idx, r);
            }
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (r < nsplit) M = fmaxf(M, mr[r]);
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (r < nsplit) {
                const float f = mr[r] == -INFINITY ? 0.f : expf(mr[r] - M);
                L = fmaf(lr[r], f, L);
                c = fmaf(cr[r], f, c);
            }
        put(idx, c, L);
    }
    cluster.sync();  // the others still read this CTA's part
}

template <int D, int G>
int launch_t(lumen_ctx *ctx, const AttnRowsArgs &a, size_t B, size_t Hkv, int splits, cudaStream_t s) {
    constexpr size_t smem = ArGeom<D, G>::kFloats * sizeof(float);
    auto kernel = attn_rows_kernel<D, G>;
    static bool attr_set[64] = {false};
    const int dev = ctx->device >= 0 && ctx->device < 64 ? ctx->device : 0;
    if (!attr_set[dev]) {
        LUMEN_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set[dev] = true;
    }
    return launch_pdl_cluster(ctx, kernel, (unsigned)splits, dim3((unsigned)splits, (unsigned)Hkv, (unsigned)B), dim3(kArThreads), smem, s, a);
}

}  // namespace

int launch_attn_rows(lumen_ctx *ctx, const AttnRowsArgs &a, size_t B, size_t Hq, size_t Hkv, size_t D, int splits, cudaStream_t s) {
    const size_t G = Hkv ? Hq / Hkv : 0;
#define LUMEN_AR(D_) (G == 8 ? launch_t<D_, 8>(ctx, a, B, Hkv, splits, s) : G == 4 ? launch_t<D_, 4>(ctx, a, B, Hkv, splits, s) \
                      : G == 2 ? launch_t<D_, 2>(ctx, a, B, Hkv, splits, s) : launch_t<D_, 1>(ctx, a, B, Hkv, splits, s))
    return D == 128 ? LUMEN_AR(128) : LUMEN_AR(64);
#undef LUMEN_AR
}

}  // namespace lumen
