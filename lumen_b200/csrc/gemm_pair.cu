// C[M,N] = A[M,K] . W[N,K]^T (+ residual) for many rows (prefill): the same operands and arithmetic as gemm_tc.cu (f32
// activations as bf16 hi + lo, f32 weights likewise, products accumulated in the same order), by pairs of SMs.
//
// What bounds it: the tensor pipe and, before it, the operands' way from the L2 to shared memory.  With hi and lo every 64
// numbers of K bring 48 KB per 128 x 128 tile for 512 cycles of MMA, more than the L2 delivers per SM.  Here two CTAs of a
// cluster share one 256 x BN tile (tcgen05 cta_group::2): each loads its 128 rows of A and half of the columns' weights, and
// the tensor cores of both read the two halves, so the same 48 KB serve 1024 cycles.  The rest overlaps with the MMAs: one CTA
// per SM walks the tiles (groups of 8 tile rows share weights in the L2), a producer thread keeps a ring of stages full
// across tiles, and four epilogue warps empty one half of the tensor memory while the next tile accumulates in the other.
// Measured (8192 rows, K 4096, bf16 weights): the products of a block of 193 M weights 6.45 -> 4.42 ms, 490 -> 714 TFLOP/s of
// useful work, 1428 issued of 1667 measured for one bf16 product; f32 weights (1777 rows, K 2048 and 5632) 315 -> 418 useful,
// 945 -> 1254 issued.
//
// Roles per CTA (192 threads): warp 0 = TMA producer, warp 1 = MMA issuer (the first CTA of a pair only), warps 2-5 =
// epilogue.  Every wait is bounded; after a failure nobody waits any more and all threads meet at the closing barriers.
#include <algorithm>

#include "gemm_pair.cuh"
#include "row_finish.cuh"
#include "tc_common.cuh"

namespace lumen {
namespace {

using namespace tc;

constexpr int kPairThreads = 192;
constexpr int kPairRows = 256;          // rows of a tile, 128 per CTA
constexpr int kGroupRows = 8;           // tile rows walked together

template <int NA, int NB, int BN>
struct PairGeom {
    static constexpr uint32_t kABytes = 128 * kBK * 2, kBBytes = BN / 2 * kBK * 2;  // one bf16 part of one CTA's operands
    static constexpr uint32_t kStageBytes = NA * kABytes + NB * kBBytes;
    static constexpr int kStages = (200 * 1024 / kStageBytes) > 6 ? 6 : (200 * 1024 / kStageBytes);
    static constexpr uint32_t kIdesc = idesc_bf16(kPairRows, BN);
};

struct PairParams {
    float *c;               // [M, N], or [splits][M][N] partial sums
    const float *residual;  // [M, N] or null
    __nv_bfloat16 *hi, *lo; // SWIGLU: [M, N / 2]
    int M, N, K;            // SWIGLU: N = rows of gate and up together
    int kb_per_split, splits;
    DeviceStatus *status;
};

__device__ __forceinline__ uint32_t cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t in_first(const void *p) {  // shared::cluster address of the same variable in the pair's first CTA
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(saddr(p)));
    return a;
}
// 2-D tiled load into this CTA's shared memory that signals a barrier of the pair's first CTA (an address of in_first).
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(saddr(dst)), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n}"
                 ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// Arrives at the barrier of both CTAs when every MMA issued so far has completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(saddr(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void arrive_first(uint64_t *bar) {  // at the barrier of the pair's first CTA
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_first(bar)) : "memory");
}

struct PairTile {
    int m0, n0, split;  // n0: first column (SWIGLU: of the N / 2)
};
__device__ __forceinline__ PairTile pair_tile(int item, int tm, int tn, int cols) {
    PairTile t;
    const int tiles = tm * tn;
    t.split = item / tiles;
    const int i = item - t.split * tiles, g = i / (kGroupRows * tn), r = i - g * kGroupRows * tn;
    const int rows = min(kGroupRows, tm - g * kGroupRows);
    t.m0 = (g * kGroupRows + r % rows) * kPairRows;
    t.n0 = r / rows * cols;
    return t;
}

template <int NA, int NB, int BN, bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_ahi, const __grid_constant__ CUtensorMap map_alo,
                 const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_blo, const PairParams p) {
    using G = PairGeom<NA, NB, BN>;
    constexpr int kStages = G::kStages, kCols = SWIGLU ? BN / 2 : BN;
    static_assert(BN % 32 == 0 && BN <= 256, "columns of an MMA of two SMs; half of the weight rows end on a 1024-byte pattern");
    extern __shared__ unsigned char smem_raw[];
    unsigned char *ring = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[kStages], empty[kStages], tfull[2], tempty[2], quiet;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cta_rank();
    const int width = SWIGLU ? p.N / 2 : p.N;
    const int tm = (p.M + kPairRows - 1) / kPairRows, tn = (width + kCols - 1) / kCols;
    const int items = tm * tn * p.splits, first = blockIdx.x >> 1, step = gridDim.x >> 1;
    const int kb_all = (p.K + kBK - 1) / kBK;
    auto kb_range = [&](int split, int &kb0) {
        kb0 = split * p.kb_per_split;
        return min(kb_all, kb0 + p.kb_per_split) - kb0;
    };

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            bar_init(&full[s], 1);
            bar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            bar_init(&tfull[b], 1);
            bar_init(&tempty[b], 8);  // four epilogue warps of two CTAs
        }
        bar_init(&quiet, 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tmem_base_s)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();  // both CTAs' barriers exist before anything signals across
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    // The next kernel may start now, not earlier: its CTAs may take tensor memory before they wait for this kernel, so every CTA of this one must have its own.
    pdl_launch();
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            // ---- producer: this CTA's rows of A and its half of the tile's weight rows ----
            const uint32_t full0 = in_first(full);
            int i = 0;
            for (int item = first; item < items && !failed; item += step) {
                const PairTile t = pair_tile(item, tm, tn, kCols);
                int kb0;
                const int nkb = kb_range(t.split, kb0);
                const int ay = t.m0 + (int)rank * 128;
                const int by = SWIGLU ? t.n0 + (int)rank * width : t.n0 + (int)rank * (BN / 2);  // (gate in the first CTA, up in the second)
                for (int kb = 0; kb < nkb; ++kb, ++i) {
                    const int s = i % kStages;
                    if (!wait_or_failed(&empty[s], (uint32_t)(((i / kStages) & 1) ^ 1), &failed, p.status, 540)) break;
                    unsigned char *st = ring + (size_t)s * G::kStageBytes;
                    if (rank == 0) bar_expect(&full[s], 2 * G::kStageBytes);
                    const int kx = (kb0 + kb) * kBK;
                    const uint32_t bar = full0 + s * (uint32_t)sizeof(full[0]);
                    tma_load_2d_pair(st, &map_ahi, kx, ay, bar);
                    if (NA == 2) tma_load_2d_pair(st + G::kABytes, &map_alo, kx, ay, bar);
                    tma_load_2d_pair(st + NA * G::kABytes, &map_b, kx, by, bar);
                    if (NB == 2) tma_load_2d_pair(st + NA * G::kABytes + G::kBBytes, &map_blo, kx, by, bar);
                }
            }
            // the last stages have been read (and their copies landed) before the CTA may end
            for (int k = max(0, i - kStages); k < i; ++k) {
                if (failed) {
                    if (rank == 0) bar_wait(&full[k % kStages], (uint32_t)((k / kStages) & 1), p.status, 541);
                } else {
                    wait_or_failed(&empty[k % kStages], (uint32_t)((k / kStages) & 1), &failed, p.status, 542);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // ---- MMA issuer of the pair ----
            int i = 0, use = 0;
            for (int item = first; item < items && !failed; item += step, ++use) {
                const PairTile t = pair_tile(item, tm, tn, kCols);
                int kb0;
                const int nkb = kb_range(t.split, kb0);
                const int buf = use & 1;
                if (!wait_or_failed(&tempty[buf], (uint32_t)(((use >> 1) & 1) ^ 1), &failed, p.status, 543)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem_base + (uint32_t)(buf * 256);
                for (int kb = 0; kb < nkb; ++kb, ++i) {
                    const int s = i % kStages;
                    if (!wait_or_failed(&full[s], (uint32_t)((i / kStages) & 1), &failed, p.status, 544)) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t st = saddr(ring + (size_t)s * G::kStageBytes);
                    const uint64_t dhi = smem_desc(st), dlo = smem_desc(st + G::kABytes), db = smem_desc(st + NA * G::kABytes);
                    const uint64_t dblo = smem_desc(st + NA * G::kABytes + G::kBBytes);
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; ++kk) {
                        umma_bf16_pair(acc, dhi + 2 * kk, db + 2 * kk, G::kIdesc, (kb > 0 || kk > 0) ? 1u : 0u);
                        if (NA == 2) umma_bf16_pair(acc, dlo + 2 * kk, db + 2 * kk, G::kIdesc, 1u);
                        if (NB == 2) umma_bf16_pair(acc, dhi + 2 * kk, dblo + 2 * kk, G::kIdesc, 1u);
                    }
                    umma_commit_pair(&empty[s]);
                }
                umma_commit_pair(&tfull[buf]);
            }
        }
    } else {
        // ---- epilogue: a thread per row, its 32-lane quarter of the tensor memory by warp ----
        const int quarter = warp & 3;
        int use = 0;
        for (int item = first; item < items; item += step, ++use) {
            const PairTile t = pair_tile(item, tm, tn, kCols);
            const int buf = use & 1;
            const bool have = wait_or_failed(&tfull[buf], (uint32_t)((use >> 1) & 1), &failed, p.status, 545);
            if (__any_sync(0xffffffffu, !have)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row = t.m0 + (int)rank * 128 + quarter * 32 + lane;
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * 256);
            if constexpr (SWIGLU) {
#pragma unroll 1
                for (int c0 = 0; c0 < kCols; c0 += 32) {
                    uint32_t g[32], u[32];
                    __syncwarp();
                    tmem_ld32_issue(taddr + c0, g);
                    tmem_ld32_issue(taddr + kCols + c0, u);
                    tmem_ld_wait();
                    if (row < p.M) {
                        const size_t at = (size_t)row * width + t.n0 + c0;  // width is a multiple of 8
#pragma unroll
                        for (int j = 0; j < 32; j += 8) {
                            if (t.n0 + c0 + j >= width || c0 + j >= kCols) break;  // (kCols is a multiple of 16)
                            uint2 h[2], l[2];
#pragma unroll
                            for (int q = 0; q < 2; ++q) {
                                float x[4];
#pragma unroll
                                for (int e = 0; e < 4; ++e) x[e] = silu_mul1(__uint_as_float(g[j + 4 * q + e]), __uint_as_float(u[j + 4 * q + e]));
                                split4(make_float4(x[0], x[1], x[2], x[3]), &h[q], &l[q]);
                            }
                            *reinterpret_cast<uint4 *>(p.hi + at + j) = make_uint4(h[0].x, h[0].y, h[1].x, h[1].y);
                            *reinterpret_cast<uint4 *>(p.lo + at + j) = make_uint4(l[0].x, l[0].y, l[1].x, l[1].y);
                        }
                    }
                }
            } else {
                float *cbase = p.c + (size_t)t.split * p.M * p.N;
                const bool vec4 = (p.N & 3) == 0 && ((reinterpret_cast<uintptr_t>(cbase) | reinterpret_cast<uintptr_t>(p.residual)) & 15) == 0;
#pragma unroll 1
                for (int c0 = 0; c0 < BN; c0 += 32) {
                    uint32_t v[32];
                    __syncwarp();
                    tmem_ld32(taddr + c0, v);
                    const int col = t.n0 + c0;
                    if (row >= p.M || col >= p.N) continue;
                    float *crow = cbase + (size_t)row * p.N + col;
                    const float *rrow = p.residual ? p.residual + (size_t)row * p.N + col : nullptr;
                    if (vec4 && col + 32 <= p.N) {
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            float4 x = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                            if (rrow) x = add4(*reinterpret_cast<const float4 *>(rrow + j), x);
                            *reinterpret_cast<float4 *>(crow + j) = x;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (col + j < p.N) crow[j] = rrow ? __fadd_rn(rrow[j], __uint_as_float(v[j])) : __uint_as_float(v[j]);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_first(&tempty[buf]);
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (failed && rank == 0 && tid == 32) {  // a wait gave up: the MMAs under way end before their tensor memory is given back
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(&quiet)) : "memory");
        drain_ring(&quiet, 1, 1);
    }
    cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    cluster_sync();  // neither CTA ends while the other still frees the pair's tensor memory
}

template <int NA, int NB, int BN, bool SWIGLU>
int launch_pair_t(lumen_ctx *ctx, const GemmPairArgs &g, const PairParams &p, cudaStream_t s) {
    using G = PairGeom<NA, NB, BN>;
    constexpr size_t smem = (size_t)G::kStages * G::kStageBytes + 1024;
    auto kernel = gemm_pair_kernel<NA, NB, BN, SWIGLU>;
    static bool attr_set[64] = {false};
    const int dev = ctx->device >= 0 && ctx->device < 64 ? ctx->device : 0;
    if (!attr_set[dev]) {
        LUMEN_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set[dev] = true;
    }
    CUtensorMap ma, ma2, mb, mb2;
    LUMEN_TRY(make_map(ctx, &ma, g.a_hi, g.M, g.K, 128));
    LUMEN_TRY(make_map(ctx, &ma2, NA == 2 ? g.a_lo : g.a_hi, g.M, g.K, 128));
    LUMEN_TRY(make_map(ctx, &mb, g.w_hi, g.N, g.K, BN / 2));
    LUMEN_TRY(make_map(ctx, &mb2, NB == 2 ? g.w_lo : g.w_hi, g.N, g.K, BN / 2));
    const size_t width = SWIGLU ? g.N / 2 : g.N, cols = SWIGLU ? BN / 2 : BN;
    const size_t items = (g.M + kPairRows - 1) / kPairRows * ((width + cols - 1) / cols) * p.splits;
    const unsigned pairs = (unsigned)std::min<size_t>(items, std::max(1, ctx->num_sms / 2));
    return launch_pdl(ctx, kernel, 2 * pairs, kPairThreads, smem, s, ma, ma2, mb, mb2, p);
}

}  // namespace

int launch_gemm_pair(lumen_ctx *ctx, const GemmPairArgs &g, const GemmPairPlan &plan, cudaStream_t s) {
    PairParams p{};
    p.c = g.c; p.residual = g.residual; p.hi = g.out_hi; p.lo = g.out_lo;
    p.M = (int)g.M; p.N = (int)g.N; p.K = (int)g.K;
    p.kb_per_split = plan.kb_per_split; p.splits = plan.splits;
    p.status = ctx->d_status;
    const bool two = g.w_lo != nullptr, glu = g.out_hi != nullptr;
#define LUMEN_PAIR(NB_, BN_, GLU_) launch_pair_t<2, NB_, BN_, GLU_>(ctx, g, p, s)
#define LUMEN_PAIR_BN(BN_) (glu ? (two ? LUMEN_PAIR(2, BN_, true) : LUMEN_PAIR(1, BN_, true)) : (two ? LUMEN_PAIR(2, BN_, false) : LUMEN_PAIR(1, BN_, false)))
    switch (plan.bn) {
        case 256: return LUMEN_PAIR_BN(256);
        case 224: return LUMEN_PAIR_BN(224);
        case 192: return LUMEN_PAIR_BN(192);
        default: return LUMEN_PAIR_BN(128);
    }
#undef LUMEN_PAIR_BN
#undef LUMEN_PAIR
}

}  // namespace lumen
