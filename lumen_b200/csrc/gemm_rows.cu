// The products of a batched step (at most 64 rows: batched decode, short prompts), each with what follows it: one kernel per product, and
// nothing between two products but the attention.
//
//   C[M,N] = A[M,K] . W[N,K]^T as in gemm_tc.cu's swapped form: 128 rows of W fill the 128-row side of the MMA, the M activation rows
//   (bf16 hi and lo) the other one; f32 weights come as hi and lo too.
//
// What bounds a step is the chain of dependent kernels before the weights' way from HBM: TinyLlama with 16 sequences streams 4.4 GB
// (0.66 ms) but took 2.0 ms in eleven launches per block.  Hence
//   - the slices of K of one tile are the CTAs of a cluster: their accumulators meet in shared memory (each CTA adds its share
//     of the rows over the cluster) instead of in global memory and a second kernel;
//   - RMSNorm is a scalar per row, so it is left to the next product: a product's epilogue adds the residual, and writes x, the pair
//     (hi, lo) of x * gains, and its tile's sum of squares; the next product's epilogue multiplies by 1 / rms.  No kernel has to see a whole row;
//   - SwiGLU: a tile is 64 rows of gate and the 64 rows of up that go with them;
//   - programmatic dependent launch: a CTA asks for its first weights, then waits for the kernel before it.  The ring is small
//     enough (111 KB) for two CTAs per SM, so that the next product's CTAs find room before this one's end.  (Asking for the rest too, up to
//     64 MB for the L2, gained nothing with 16 rows and cost 3 % with 64: the way from the L2 to the SMs is busy enough);
//   - hi and lo of the activations are one operand of twice the columns: two MMAs per step of K with f32 weights, not three, and even
//     and odd steps have accumulators of their own, so that no MMA waits for the one before (by itself this moved nothing: the
//     operands' way is what a stage waits for).
//
// TinyLlama f32, 16 sequences: 40 steps and the prefill of 64 positions 84 -> 59.7 ms (a step 1.9 -> 1.3 ms); 9 layers of the Qwen3-8B
// shape, 64 sequences: a step 1.9 -> 1.5 ms.
//
// Thread 0 is the TMA producer, thread 32 issues the MMAs, warps 2 and 3 form 1 / rms meanwhile; all eight warps are the epilogue (its code runs
// once per CTA, so it is bound by latencies and by the way of the instructions themselves: short loops, little unrolling).
// Every wait is bounded; after a failure the CTA skips its arithmetic but takes part in every barrier of the cluster.
#include <algorithm>

#include <cooperative_groups.h>

#include "gemm_rows.cuh"
#include "row_finish.cuh"
#include "tc_common.cuh"

namespace lumen {
namespace {

using namespace tc;
namespace cg = cooperative_groups;

constexpr int kRowsThreads = 256;
constexpr int kRowsRing = 111 * 1024;

template <int NW, int BN>
struct RowsGeom {
    static constexpr uint32_t kHalfBytes = 64 * kBK * 2, kWBytes = 2 * kHalfBytes, kXBytes = BN * kBK * 2;
    static constexpr uint32_t kStageBytes = NW * kWBytes + 2 * kXBytes;
    static constexpr int kStages = kRowsRing / kStageBytes > 6 ? 6 : kRowsRing / kStageBytes;
    // accumulators of BN columns: W . x_hi and W . x_lo (side by side), W_lo . x_hi; for even and odd steps where they fit
    static constexpr int kParts = NW + 1, kSets = 2 * kParts * BN <= 256 ? 2 : 1, kAccs = kSets * kParts;
    static constexpr int kTmemCols = kAccs * BN <= 64 ? 64 : kAccs * BN <= 128 ? 128 : 256;
    static_assert(kStages >= 2 && kStages * kStageBytes >= BN * 128 * 4, "the ring holds the accumulator afterwards");
};

struct RowsParams {
    GemmRowsArgs a;
    int kb_per, splits;
    DeviceStatus *status;
};

// 16 consecutive accumulator columns of this thread's lane; usable after tmem_ld_wait().
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}

// EPI: GemmRowsArgs::Epi
template <int NW, int BN, int EPI>
__global__ void __launch_bounds__(kRowsThreads, 2)
gemm_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_wlo, const __grid_constant__ CUtensorMap map_x,
                 const __grid_constant__ CUtensorMap map_xlo, const RowsParams p) {
    using G = RowsGeom<NW, BN>;
    constexpr int kStages = G::kStages;
    constexpr uint32_t kIdescPair = idesc_bf16(128, 2 * BN), kIdescOne = idesc_bf16(128, BN);
    extern __shared__ unsigned char smem_raw[];
    unsigned char *ring = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[kStages], empty[kStages], done;
    __shared__ uint32_t tmem_base_s;
    __shared__ int failed;
    __shared__ float inv_s[64], ss_s[4][64];
    const GemmRowsArgs &a = p.a;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int splits = p.splits, tile = (int)blockIdx.x / splits, rank = (int)blockIdx.x - tile * splits;
    const int inter = a.N / 2;
    const int n0 = tile * (EPI == GemmRowsArgs::kSwiglu ? 64 : 128), n1 = EPI == GemmRowsArgs::kSwiglu ? inter + n0 : n0 + 64;  // rows of W of the two halves
    const int kb_all = (a.K + kBK - 1) / kBK, kb0 = rank * p.kb_per, nkb = max(0, min(kb_all, kb0 + p.kb_per) - kb0);
    // The tiles walk K from different steps on: they read the same activations, and all at once they would queue for the same lines of the L2.
    const int turn = nkb ? tile % nkb : 0;
    auto k_of = [&](int kb) { return (kb0 + (kb + turn < nkb ? kb + turn : kb + turn - nkb)) * kBK; };
    auto weights = [&](int kb) {
        unsigned char *st = ring + (size_t)(kb % kStages) * G::kStageBytes;
        uint64_t *bar = &full[kb % kStages];
        const int kx = k_of(kb);
        bar_expect(bar, G::kStageBytes);
        tma_load_2d(st, &map_w, kx, n0, bar);
        tma_load_2d(st + G::kHalfBytes, &map_w, kx, n1, bar);
        if (NW == 2) {
            tma_load_2d(st + G::kWBytes, &map_wlo, kx, n0, bar);
            tma_load_2d(st + G::kWBytes + G::kHalfBytes, &map_wlo, kx, n1, bar);
        }
    };
    const int ahead = min(nkb, kStages);
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            bar_init(&full[s], 1);
            bar_init(&empty[s], 1);
        }
        bar_init(&done, 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int kb = 0; kb < ahead; ++kb) weights(kb);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tmem_base_s)), "r"(G::kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    pdl_launch();  // (behind the allocation, as in gemm_pair_kernel: the next kernel takes tensor memory before it waits)
    int issued = 0;  // steps whose copies are on their way (thread 0)
    if (tid == 0) {
        pdl_wait();
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % kStages;
            if (kb >= ahead) {
                if (!bar_wait(&empty[s], (uint32_t)((kb / kStages - 1) & 1), p.status, 560)) {
                    failed = 1;
                    break;
                }
                weights(kb);
            }
            unsigned char *st = ring + (size_t)s * G::kStageBytes + NW * G::kWBytes;
            tma_load_2d(st, &map_x, k_of(kb), 0, &full[s]);
            tma_load_2d(st + G::kXBytes, &map_xlo, k_of(kb), 0, &full[s]);
            ++issued;  // (the weights requested ahead are all among these: nothing before step `ahead` can fail)
        }
    } else if (tid == 32) {
        bool ok = true;
        pdl_wait();  // (the limit of a wait is for this kernel's copies, not for the kernel before)
        for (int kb = 0; kb < nkb && ok; ++kb) {
            const int s = kb % kStages;
            ok = bar_wait(&full[s], (uint32_t)((kb / kStages) & 1), p.status, 561);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t st = saddr(ring + (size_t)s * G::kStageBytes);
            // (x_lo follows x_hi: together they are one operand of 2 * BN rows)
            const uint64_t dw = smem_desc(st), dwlo = smem_desc(st + G::kWBytes), dx = smem_desc(st + NW * G::kWBytes);
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk) {
                const uint32_t acc = tmem_base + (uint32_t)(kk % G::kSets * G::kParts * BN), add = (kb > 0 || kk >= G::kSets) ? 1u : 0u;
                umma_bf16(acc, dw + 2 * kk, dx + 2 * kk, kIdescPair, add);
                if (NW == 2) umma_bf16(acc + 2 * BN, dwlo + 2 * kk, dx + 2 * kk, kIdescOne, add);  // (lo . lo ~ 2^-18: dropped)
            }
            umma_commit(&empty[s]);
        }
        if (!ok) failed = 1;
        umma_commit(&done);
    } else if (warp == 2 || warp == 3) {
        pdl_wait();
        const int m = tid - 64;
        if (m < a.M) {
            float s = 0.f;
#pragma unroll 8
            for (int t = 0; t < a.n_ss; ++t) s += __ldcg(a.ss_in + t * 64 + m);
            inv_s[m] = a.n_ss ? __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(s, (float)a.K), a.eps))) : 1.0f;
        }
    }
    __syncwarp();
    pdl_wait();
    const bool have = bar_wait(&done, 0, p.status, 562);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool good = __syncthreads_and(have) && !failed;  // (waits of a CTA may end differently near their limit: one answer for all, there are barriers ahead)
    // The accumulator as red[m][column of the tile], where the ring was: every copy has landed and been read.
    float *red = reinterpret_cast<float *>(ring);
    if (good) {
        const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll 1
        for (int c0 = 16 * (warp >> 2); c0 < BN; c0 += 32) {  // (warps w and w + 4 read the same lanes)
            uint32_t v[G::kAccs][16];
#pragma unroll
            for (int q = 0; q < G::kAccs; ++q) tmem_ld16_issue(taddr + (uint32_t)(q * BN + c0), v[q]);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                float sum = __uint_as_float(v[0][j]);
#pragma unroll
                for (int q = 1; q < G::kAccs; ++q) sum += __uint_as_float(v[q][j]);
                if (c0 + j < a.M) red[(c0 + j) * 128 + (tid & 127)] = nkb ? sum : 0.f;
            }
        }
    } else if (tid == 0) {
        drain_ring(full, kStages, issued);
        drain_ring(&done, 1, 1);  // (the MMAs that were issued, before their tensor memory is given back)
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(G::kTmemCols) : "memory");
    cg::cluster_group cluster = cg::this_cluster();
    if (splits > 1) cluster.sync();
    // Rows m, m + by, ... of a column: the sum of the slices, in order.  The loads of a batch of rows from four CTAs are in flight
    // together: a trip to another SM's shared memory takes some 0.5 us.
    constexpr int kBatch = BN == 16 ? 2 : 4;
    auto sums = [&](float (&v)[kBatch], int m, int by, int col) {
#pragma unroll
        for (int q = 0; q < kBatch; ++q) v[q] = 0.f;
        if (splits == 1) {
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
                if (m + q * by < a.M) v[q] = red[(m + q * by) * 128 + col];
            return;
        }
#pragma unroll 1
        for (int r0 = 0; r0 < splits; r0 += 4) {
            float t[4][kBatch];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float *src = cluster.map_shared_rank(red, min(r0 + r, splits - 1));
#pragma unroll
                for (int q = 0; q < kBatch; ++q) t[r][q] = r0 + r < splits && m + q * by < a.M ? src[(m + q * by) * 128 + col] : 0.f;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int q = 0; q < kBatch; ++q) v[q] += t[r][q];
        }
    };
    if (good) {
        if constexpr (EPI == GemmRowsArgs::kSwiglu) {
            const int col = n0 + (tid & 63), by = 4 * splits;
#pragma unroll 1
            for (int m0 = rank * 4 + (tid >> 6); m0 < a.M; m0 += kBatch * by) {
                float g[kBatch], u[kBatch];
                sums(g, m0, by, tid & 63);
                sums(u, m0, by, 64 + (tid & 63));
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const int m = m0 + q * by;
                    if (m >= a.M || col >= inter) continue;
                    const float v = silu_mul1(__fmul_rn(g[q], inv_s[m]), __fmul_rn(u[q], inv_s[m]));
                    const __nv_bfloat16 h = __float2bfloat16_rn(v);
                    a.hi[(size_t)m * inter + col] = h;
                    a.lo[(size_t)m * inter + col] = __float2bfloat16_rn(v - __bfloat162float(h));
                }
            }
        } else if constexpr (EPI == GemmRowsArgs::kResidual) {
            const int col = n0 + (tid & 127), by = 2 * splits;
            const float g = col < a.N ? a.gain[col] : 0.f;
#pragma unroll 1
            for (int m0 = rank + splits * (tid >> 7); m0 < a.M; m0 += kBatch * by) {
                float v[kBatch], x[kBatch];
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const int m = m0 + q * by;
                    x[q] = m < a.M && col < a.N ? a.x[(size_t)m * a.N + col] : 0.f;
                }
                sums(v, m0, by, tid & 127);
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const int m = m0 + q * by;
                    if (m >= a.M) break;  // (the same in a warp)
                    float ss = 0.f;
                    if (col < a.N) {
                        const size_t at = (size_t)m * a.N + col;
                        const float h = __fadd_rn(x[q], v[q]);  // h = x + attn_out, out = h + mlp_out (llama.rs:110, :115)
                        a.x[at] = h;
                        const float y = __fmul_rn(h, g);
                        const __nv_bfloat16 b = __float2bfloat16_rn(y);
                        a.hi[at] = b;
                        a.lo[at] = __float2bfloat16_rn(y - __bfloat162float(b));
                        ss = h * h;
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                    if (lane == 0) ss_s[warp & 3][m] = ss;
                }
            }
            __syncthreads();
            if (tid < a.M && tid % splits == rank) a.ss_out[tile * 64 + tid] = (ss_s[0][tid] + ss_s[1][tid]) + (ss_s[2][tid] + ss_s[3][tid]);
            if (a.advance && blockIdx.x == 0 && tid == 0) *a.advance += 1;
        } else {
            const int col = n0 + (tid & 127), by = 2 * splits;
#pragma unroll 1
            for (int m0 = rank + splits * (tid >> 7); m0 < a.M; m0 += kBatch * by) {
                float v[kBatch];
                sums(v, m0, by, tid & 127);
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const int m = m0 + q * by;
                    if (m < a.M && col < a.N) a.c[(size_t)m * a.N + col] = __fmul_rn(v[q], inv_s[m]);
                }
            }
        }
    }
    if (splits > 1) cluster.sync();  // the others still read this CTA's accumulator
}

// The first product's operands: the pair of x * gains and the sums of squares (one per row).
__global__ void __launch_bounds__(256) rows_start_kernel(const float *x, const float *gain, int dim, __nv_bfloat16 *hi, __nv_bfloat16 *lo, float *ss_out) {
    __shared__ float red[8];
    const int tid = threadIdx.x;
    const size_t base = (size_t)blockIdx.x * dim;
    pdl_launch();
    pdl_wait();
    float ss = 0.f;
    for (int i = tid; i < dim / 4; i += 256) {
        const float4 v = __ldcg(reinterpret_cast<const float4 *>(x + base) + i), g = reinterpret_cast<const float4 *>(gain)[i];
        ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
        uint2 h, l;
        split4(make_float4(__fmul_rn(v.x, g.x), __fmul_rn(v.y, g.y), __fmul_rn(v.z, g.z), __fmul_rn(v.w, g.w)), &h, &l);
        reinterpret_cast<uint2 *>(hi + base)[i] = h;
        reinterpret_cast<uint2 *>(lo + base)[i] = l;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    if (tid == 0) {
        float t = 0.f;
        for (int w = 0; w < 8; ++w) t += red[w];
        ss_out[blockIdx.x] = t;
    }
}

template <int NW, int BN, int EPI>
int launch_rows_t(lumen_ctx *ctx, const GemmRowsArgs &a, cudaStream_t s) {
    using G = RowsGeom<NW, BN>;
    constexpr size_t smem = (size_t)G::kStages * G::kStageBytes + 1024;
    auto kernel = gemm_rows_kernel<NW, BN, EPI>;
    static bool attr_set[64] = {false};
    const int dev = ctx->device >= 0 && ctx->device < 64 ? ctx->device : 0;
    if (!attr_set[dev]) {
        LUMEN_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set[dev] = true;
    }
    CUtensorMap mw, mwlo, mx, mxlo;
    LUMEN_TRY(make_map(ctx, &mw, a.w_hi, a.N, a.K, 64));
    LUMEN_TRY(make_map(ctx, &mwlo, NW == 2 ? a.w_lo : a.w_hi, a.N, a.K, 64));
    LUMEN_TRY(make_map(ctx, &mx, a.x_hi, a.M, a.K, BN));
    LUMEN_TRY(make_map(ctx, &mxlo, a.x_lo, a.M, a.K, BN));
    const int tiles = EPI == GemmRowsArgs::kSwiglu ? (a.N / 2 + 63) / 64 : (a.N + 127) / 128, kb_all = (a.K + kBK - 1) / kBK;
    // Slices: until most SMs have a CTA (at least four steps of K each), as long as all CTAs are resident, two per SM.
    RowsParams p;
    p.a = a;
    p.status = ctx->d_status;
    p.splits = 1;
    while (p.splits < 8 && tiles * p.splits * 100 < ctx->num_sms * 85 && kb_all >= 8 * p.splits) p.splits *= 2;
    p.kb_per = (kb_all + p.splits - 1) / p.splits;
    return launch_pdl_cluster(ctx, kernel, (unsigned)p.splits, dim3((unsigned)(tiles * p.splits)), dim3(kRowsThreads), smem, s, mw, mwlo, mx, mxlo, p);
}

}  // namespace

bool gemm_rows_usable(lumen_dtype wdt, size_t M, size_t K, size_t N, const void *w) {
    return M <= (size_t)kGemmRowsMax && gemm_tc_usable(wdt, std::max<size_t>(M, 2), K, N, w) && N <= (1u << 30) && K <= (1u << 30);
}
size_t gemm_rows_ss_floats(size_t N) { return (N + 127) / 128 * 64; }

int launch_gemm_rows(lumen_ctx *ctx, const GemmRowsArgs &a, cudaStream_t s) {
    const int bn = a.M > 32 ? 64 : a.M > 16 ? 32 : 16;
#define LUMEN_ROWS_E(W_, B_)                                                                                   \
    (a.epi == GemmRowsArgs::kSwiglu ? launch_rows_t<W_, B_, GemmRowsArgs::kSwiglu>(ctx, a, s)                  \
     : a.epi == GemmRowsArgs::kResidual ? launch_rows_t<W_, B_, GemmRowsArgs::kResidual>(ctx, a, s)            \
                                        : launch_rows_t<W_, B_, GemmRowsArgs::kStore>(ctx, a, s))
#define LUMEN_ROWS(W_) (bn == 64 ? LUMEN_ROWS_E(W_, 64) : bn == 32 ? LUMEN_ROWS_E(W_, 32) : LUMEN_ROWS_E(W_, 16))
    return a.w_lo ? LUMEN_ROWS(2) : LUMEN_ROWS(1);
#undef LUMEN_ROWS
#undef LUMEN_ROWS_E
}

int launch_rows_start(lumen_ctx *ctx, const float *x, const float *gain, size_t rows, size_t dim, __nv_bfloat16 *hi, __nv_bfloat16 *lo, float *ss,
                      cudaStream_t s) {
    return launch_pdl(ctx, rows_start_kernel, dim3((unsigned)rows), dim3(256), 0, s, x, gain, (int)dim, hi, lo, ss);
}

}  // namespace lumen
