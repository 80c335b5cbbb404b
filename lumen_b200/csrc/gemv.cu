// M = 1 (and small-M) vector-matrix kernels: y = W . x with W streamed once from HBM.
//
// Restates the M == 1 branch of ops::matmul::matmul (src/ops/matmul.rs:42-69 of the reference):
// one output element per weight row, f32 accumulation.  The reference sums in k order on one
// core; here a warp owns a row, every lane accumulates a strided slice with FMAs and the 32
// partial sums are combined by a shuffle tree, so results agree to rounding, not bitwise.
//
// Bandwidth design: each lane issues 128-bit streaming loads (ld.global.cs) and keeps
// kUnroll x kRowsPerWarp of them in flight; the activation vector is staged once per CTA in
// shared memory and read back as conflict-free 128-bit words.
#include <algorithm>

#include <cooperative_groups.h>

#include "decoder_kernels.cuh"
#include "gemv_rows.cuh"

namespace lumen {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// Stage x[M,K] into shared memory, optionally RMS-normalised: xs = (x * inv_rms) * norm_w, which is
// the element the reference's RMSNorm produces (src/layers/norm/rms_norm.rs:49-56) before its Linear.
// The CTA's warps share out the rows: one each where a pass has eight, all of them for a single one.  Every CTA does all of this, so it is
// paid per launch: with an index division per element and block-wide sums row after row the products of eight TinyLlama rows took 47
// (q, k, v), 43 (o), 65 (gate, up) and 103 us (down), most of it here.
// A step of 22 TinyLlama layers, f32, at 100 positions: 2401 -> 1747 us with 2 rows, 3443 -> 1943 with 4, 4884 -> 2252 with 8.
// (With one warp per row whatever their number, eight layers took 675 us with 2 rows, 747 with 4, now 658 and 733; a prompt of two tokens whose
// last row alone goes through an output matrix of bf16 [32000,4096], host to host, 149 us, now 141.)
template <int MB>
__device__ void stage_x(float *xs, const float *__restrict__ x, int M, size_t K, const float *__restrict__ norm_w, float eps) {
    static_assert(MB <= kWarps && kWarps % MB == 0, "whole warps per row");
    const int tid = threadIdx.x, n = (int)(M * K), all = (int)(MB * K);
    const bool vec = K % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    if (vec) {
#pragma unroll 8
        for (int i = tid; i < n / 4; i += kThreads) reinterpret_cast<float4 *>(xs)[i] = reinterpret_cast<const float4 *>(x)[i];
    } else {
        for (int i = tid; i < n; i += kThreads) xs[i] = x[i];
    }
    for (int i = n + tid; i < all; i += kThreads) xs[i] = 0.f;
    __syncthreads();
    if (norm_w == nullptr) return;
    constexpr int WPR = kWarps / MB, kStep = 32 * WPR;  // warps of a row
    __shared__ float red[kWarps];
    const int warp = tid >> 5, m = warp / WPR, at = tid % kStep;
    float *row = xs + (size_t)m * K;
    const bool vec_norm = vec && (reinterpret_cast<uintptr_t>(norm_w) & 15) == 0;
    const int n4 = (int)(K / 4);
    float ss = 0.f;
    if (m < M) {
        if (vec_norm) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);  // (four sums: short chains)
#pragma unroll 4
            for (int k = at; k < n4; k += kStep) {
                const float4 v = reinterpret_cast<const float4 *>(row)[k];
                acc = make_float4(fmaf(v.x, v.x, acc.x), fmaf(v.y, v.y, acc.y), fmaf(v.z, v.z, acc.z), fmaf(v.w, v.w, acc.w));
            }
            ss = (acc.x + acc.y) + (acc.z + acc.w);
        } else {
            for (size_t k = at; k < K; k += kStep) ss = fmaf(row[k], row[k], ss);
        }
    }
    ss = warp_sum(ss);
    if (WPR > 1) {
        if ((tid & 31) == 0) red[warp] = ss;
        __syncthreads();
        ss = 0.f;
#pragma unroll
        for (int w = 0; w < WPR; ++w) ss += red[m * WPR + w];
    }
    if (m < M) {
        const float inv = __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
        if (vec_norm) {
            float4 *r4 = reinterpret_cast<float4 *>(row);
            const float4 *g4 = reinterpret_cast<const float4 *>(norm_w);
#pragma unroll 4
            for (int k = at; k < n4; k += kStep) {
                const float4 v = r4[k], g = g4[k];
                r4[k] = make_float4(__fmul_rn(__fmul_rn(v.x, inv), g.x), __fmul_rn(__fmul_rn(v.y, inv), g.y), __fmul_rn(__fmul_rn(v.z, inv), g.z),
                                    __fmul_rn(__fmul_rn(v.w, inv), g.w));
            }
        } else {
            for (size_t k = at; k < K; k += kStep) row[k] = __fmul_rn(__fmul_rn(row[k], inv), norm_w[k]);
        }
    }
    __syncthreads();
}

template <typename WT, int MB>
__global__ void __launch_bounds__(kThreads)
gemv_nk_kernel(const float *__restrict__ x, const WT *__restrict__ w, float *__restrict__ y, int M, size_t K, size_t N,
               size_t ldy, const float *__restrict__ norm_w, float eps, const float *__restrict__ residual) {
    extern __shared__ __align__(16) float smem[];
    float *xs = smem;
    stage_x<MB>(xs, x, M, K, norm_w, eps);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int VEC = 16 / sizeof(WT);
    const bool vec_ok = (K % VEC == 0) && ((reinterpret_cast<uintptr_t>(w) & 15) == 0);
    if constexpr (MB > 1) {
        if (vec_ok) {  // several vectors: rows are taken RR at a time so that x is read once per RR rows
            constexpr int RR = MB >= 8 ? 2 : 4;
            for (size_t row0 = ((size_t)blockIdx.x * kWarps + warp) * RR; row0 < N; row0 += (size_t)gridDim.x * kWarps * RR) {
                const WT *rows[RR];
                float acc[RR][MB];
#pragma unroll
                for (int r = 0; r < RR; ++r) {
                    rows[r] = w + (row0 + r < N ? row0 + r : N - 1) * K;  // rows past the end repeat the last one (not stored)
#pragma unroll
                    for (int m = 0; m < MB; ++m) acc[r][m] = 0.f;
                }
                rows_dot<WT, MB, RR>(rows, xs, K, lane, acc);
#pragma unroll
                for (int r = 0; r < RR; ++r) {
#pragma unroll
                    for (int m = 0; m < MB; ++m) {
                        const float v = warp_sum(acc[r][m]);
                        if (lane == 0 && m < M && row0 + r < N) {
                            const size_t o = (size_t)m * ldy + row0 + r;
                            y[o] = residual ? __fadd_rn(residual[o], v) : v;
                        }
                    }
                }
            }
            return;
        }
    }
    for (size_t row = (size_t)blockIdx.x * kWarps + warp; row < N; row += (size_t)gridDim.x * kWarps) {
        float acc[MB];
#pragma unroll
        for (int m = 0; m < MB; ++m) acc[m] = 0.f;
        row_dot<WT, MB>(w + row * K, xs, K, lane, vec_ok, acc);
#pragma unroll
        for (int m = 0; m < MB; ++m) {
            float v = warp_sum(acc[m]);
            if (lane == 0 && m < M) {
                size_t o = (size_t)m * ldy + row;
                y[o] = residual ? __fadd_rn(residual[o], v) : v;
            }
        }
    }
}

// One vector, nothing before or behind the product, rows of whole 16-byte vectors: launched so that it may start while the call before it
// still runs (programmatic dependent launch).  Until that one is complete nothing is read - x and W may be its result - but the first
// rows are handed to the L2, which is where all SMs meet.  Then a warp has 2 x kAhead vectors of its rows in flight,
// the first of them requested before x is staged and the next row's while a row is summed up.  WPR warps share a row where rows
// are fewer than warps would be.
// What bounds it: launch, first bytes and staging for matrices of a few MB, HBM for large ones.  Calls behind one another, other weights every time:
// f32 [256,2048] 6.7 -> 2.65 us (three quarters of it the overlap), [4096,4096] 15.7 -> 12.1, [32000,4096] 79.9 -> 76.1 (6.9 TB/s);
// bf16 (fewer rows than warps, or rows below 2 KB; others go to the kernel behind this one) [256,2048] 4.6 -> 2.45, [2048,2048] 6.2 -> 4.0, [512,8192] 8.8 -> 4.8.
template <typename WT, int WPR>
__global__ void __launch_bounds__(kThreads, 4) gemv_vec_kernel(const float *x, const WT *w, float *y, int K, size_t N) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float red[kWarps];
    constexpr int VEC = 16 / sizeof(WT), kRows = kWarps / WPR;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = warp % WPR;
    const int nv = K / VEC, per = (nv + WPR - 1) / WPR, v0 = min(nv, part * per), vn = min(nv - v0, per);
    const size_t row0 = (size_t)blockIdx.x * kRows + warp / WPR, step = (size_t)gridDim.x * kRows;
    auto at = [&](size_t r) { return reinterpret_cast<const uint4 *>(w + r * K) + v0; };
    pdl_launch();
    if (row0 < N)
        for (int i = lane * 8; i < min(vn, 512); i += 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(at(row0) + i));
    pdl_wait();
    uint4 cur[kAhead];
    if (row0 < N) batch_load<true>(at(row0), 0, vn, lane, cur);
    if (K % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
#pragma unroll 4
        for (int k = tid; k < K / 4; k += kThreads) reinterpret_cast<float4 *>(smem)[k] = reinterpret_cast<const float4 *>(x)[k];
    } else {
        for (int k = tid; k < K; k += kThreads) smem[k] = x[k];
    }
    __syncthreads();
#pragma unroll 1
    for (size_t base = (size_t)blockIdx.x * kRows; base < N; base += step) {
        const size_t row = base + warp / WPR;
        float v = 0.f;
        if (row < N) v = row_dot_ahead<WT, true>(at(row), smem + v0 * VEC, vn, lane, cur, row + step < N ? at(row + step) : nullptr);
        v = warp_sum(v);
        if (WPR > 1) {  // the row's slices meet in its first warp
            if (lane == 0) red[warp] = v;
            __syncthreads();
            v = 0.f;
#pragma unroll
            for (int i = 0; i < WPR; ++i) v += red[(warp / WPR) * WPR + i];
            __syncthreads();
        }
        if (lane == 0 && part == 0 && row < N) y[row] = v;
    }
}

// The same for more bf16 rows than there are warps: two adjacent rows per warp at a time, so that the 32 bytes of x that go with 16 bytes of
// weights are read from shared memory once for both (the way to the registers, not HBM, bound it), and half as many CTAs stage x.  Rows
// shorter than a warp's batch (2 KB) lose by it, f32 rows (16 bytes of x for 16) gain nothing.
// bf16 [8448,2048] 8.9 -> 7.4 us, [11008,4096] 21.0 -> 16.8, [12288,12288] 54.6 -> 46.3 (6.5 TB/s); [20000,512] 6.9 -> 7.5, f32 [32000,4096] 76.1 -> 76.6.
__global__ void __launch_bounds__(kThreads, 2) gemv_vec_pair_kernel(const float *x, const __nv_bfloat16 *w, float *y, int K, size_t N) {
    using WT = __nv_bfloat16;
    extern __shared__ __align__(16) float smem[];
    constexpr int VEC = 16 / sizeof(WT);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nv = K / VEC;
    const size_t pairs = (N + 1) / 2, p0 = (size_t)blockIdx.x * kWarps + warp, step = (size_t)gridDim.x * kWarps;
    auto at = [&](size_t p, int r) { return reinterpret_cast<const uint4 *>(w + min(2 * p + r, N - 1) * K); };
    pdl_launch();
    if (p0 < pairs)
        for (int i = lane * 8; i < min(2 * p0 + 1 < N ? 2 * nv : nv, 512); i += 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(at(p0, 0) + i));
    pdl_wait();
    uint4 cur[2][kAhead];
    if (p0 < pairs) {
        batch_load<true>(at(p0, 0), 0, nv, lane, cur[0]);
        batch_load<true>(at(p0, 1), 0, nv, lane, cur[1]);
    }
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
#pragma unroll 4
        for (int k = tid; k < K / 4; k += kThreads) reinterpret_cast<float4 *>(smem)[k] = reinterpret_cast<const float4 *>(x)[k];
    } else {
        for (int k = tid; k < K; k += kThreads) smem[k] = x[k];
    }
    __syncthreads();
#pragma unroll 1
    for (size_t p = p0; p < pairs; p += step) {
        float v[2];
        const bool more = p + step < pairs;
        pair_dot_ahead<true>(at(p, 0), at(p, 1), smem, nv, lane, cur, more ? at(p + step, 0) : nullptr, more ? at(p + step, 1) : nullptr, v);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
            v[1] += __shfl_xor_sync(0xffffffffu, v[1], o);
        }
        if (lane < 2 && 2 * p + lane < N) y[2 * p + lane] = lane ? v[1] : v[0];
    }
}

// gate/up pair: out[m,i] = silu(gate_i . x_m) * (up_i . x_m)  (src/models/llama.rs:59-63,
// src/layers/activation.rs:143-146: sig = 1/(1+exp(-g)); g*sig).
template <typename WT, int MB>
__global__ void __launch_bounds__(kThreads)
gemv_gate_up_kernel(const float *__restrict__ x, const WT *__restrict__ wg, const WT *__restrict__ wu,
                    float *__restrict__ out, int M, size_t K, size_t I, const float *__restrict__ norm_w, float eps) {
    extern __shared__ __align__(16) float smem[];
    float *xs = smem;
    stage_x<MB>(xs, x, M, K, norm_w, eps);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int VEC = 16 / sizeof(WT);
    const bool vec_ok = (K % VEC == 0) && ((reinterpret_cast<uintptr_t>(wg) & 15) == 0) &&
                        ((reinterpret_cast<uintptr_t>(wu) & 15) == 0);
    if constexpr (MB > 1) {
        if (vec_ok) {  // the gate row and the up row of an output share every read of x
            for (size_t row = (size_t)blockIdx.x * kWarps + warp; row < I; row += (size_t)gridDim.x * kWarps) {
                const WT *rows[2] = {wg + row * K, wu + row * K};
                float acc[2][MB];
#pragma unroll
                for (int m = 0; m < MB; ++m) acc[0][m] = acc[1][m] = 0.f;
                rows_dot<WT, MB, 2>(rows, xs, K, lane, acc);
#pragma unroll
                for (int m = 0; m < MB; ++m) {
                    const float g = warp_sum(acc[0][m]);
                    const float u = warp_sum(acc[1][m]);
                    if (lane == 0 && m < M) {
                        const float sig = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-g)));
                        out[(size_t)m * I + row] = __fmul_rn(__fmul_rn(g, sig), u);
                    }
                }
            }
            return;
        }
    }
    for (size_t row = (size_t)blockIdx.x * kWarps + warp; row < I; row += (size_t)gridDim.x * kWarps) {
        float ag[MB], au[MB];
#pragma unroll
        for (int m = 0; m < MB; ++m) ag[m] = au[m] = 0.f;
        row_dot<WT, MB>(wg + row * K, xs, K, lane, vec_ok, ag);
        row_dot<WT, MB>(wu + row * K, xs, K, lane, vec_ok, au);
#pragma unroll
        for (int m = 0; m < MB; ++m) {
            float g = warp_sum(ag[m]);
            float u = warp_sum(au[m]);
            if (lane == 0 && m < M) {
                float sig = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-g)));
                out[(size_t)m * I + row] = __fmul_rn(__fmul_rn(g, sig), u);
            }
        }
    }
}

constexpr int kStepCtas = 4;  // of gemv_step_kernel per SM
constexpr int kHeld = 2;      // float4 of the input that a thread of it keeps in registers
// Numbers of gains that gemv_step_kernel keeps in shared memory (0: it reads them when it needs them).
__host__ __device__ inline size_t step_gains(const GemvStepArgs &a) {
    const bool fits = a.K % 4 == 0 && a.K <= (size_t)4 * kHeld * kThreads && ((reinterpret_cast<uintptr_t>(a.gain) | reinterpret_cast<uintptr_t>(a.norm_w)) & 15) == 0;
    return fits ? a.K * ((a.y ? 1 : 0) + (a.norm_w ? 1 : 0)) : 0;
}
// The input of a one-row product in shared memory: res, or res + RMSNorm(y) * gain (stored to x_out by the first CTA), then optionally
// RMSNorm * norm_w.  held: the gains are on their way to shared memory.
__device__ __forceinline__ void step_stage(const GemvStepArgs &a, float *xs, const float *gains, const float *norms, bool held, float *red, float *red2) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t K = a.K;
    auto inv_rms = [&](float ss) {
        ss = warp_sum(ss);
        if (lane == 0) red[warp] = ss;
        __syncthreads();
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) t += red[w];
        __syncthreads();
        return __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(t, (float)K), a.eps)));
    };
    // 32-bit indices and little unrolling: registers decide how many CTAs an SM holds
    const int k_n = (int)K;
    if (held) {
        const float4 *y4 = reinterpret_cast<const float4 *>(a.y), *r4 = reinterpret_cast<const float4 *>(a.res);
        const int n4 = k_n / 4;
        auto inv_of = [&](float ss, float *set) {
            ss = warp_sum(ss);
            if (lane == 0) set[warp] = ss;
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            float t = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) t += set[w];
            return __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(t, (float)K), a.eps)));
        };
        auto sq = [](const float4 &v, float ss) { return fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss)))); };
        float4 x[kHeld];
#pragma unroll
        for (int i = 0; i < kHeld; ++i) x[i] = tid + i * kThreads < n4 ? r4[tid + i * kThreads] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.y) {
            float4 y[kHeld];
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < kHeld; ++i) y[i] = tid + i * kThreads < n4 ? y4[tid + i * kThreads] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kHeld; ++i) ss = sq(y[i], ss);
            const float inv = inv_of(ss, red);
#pragma unroll
            for (int i = 0; i < kHeld; ++i) {
                const int k = tid + i * kThreads;
                if (k >= n4) break;
                const float4 g = reinterpret_cast<const float4 *>(gains)[k], v = y[i];
                x[i] = make_float4(__fadd_rn(x[i].x, __fmul_rn(__fmul_rn(v.x, inv), g.x)), __fadd_rn(x[i].y, __fmul_rn(__fmul_rn(v.y, inv), g.y)),
                                   __fadd_rn(x[i].z, __fmul_rn(__fmul_rn(v.z, inv), g.z)), __fadd_rn(x[i].w, __fmul_rn(__fmul_rn(v.w, inv), g.w)));
                if (blockIdx.x == 0) reinterpret_cast<float4 *>(a.x_out)[k] = x[i];
            }
        }
        if (a.norm_w) {
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < kHeld; ++i) ss = sq(x[i], ss);
            const float inv = inv_of(ss, red2);
#pragma unroll
            for (int i = 0; i < kHeld; ++i) {
                const int k = tid + i * kThreads;
                if (k >= n4) break;
                const float4 g = reinterpret_cast<const float4 *>(norms)[k];
                x[i] = make_float4(__fmul_rn(__fmul_rn(x[i].x, inv), g.x), __fmul_rn(__fmul_rn(x[i].y, inv), g.y), __fmul_rn(__fmul_rn(x[i].z, inv), g.z),
                                   __fmul_rn(__fmul_rn(x[i].w, inv), g.w));
            }
        }
#pragma unroll
        for (int i = 0; i < kHeld; ++i)
            if (tid + i * kThreads < n4) reinterpret_cast<float4 *>(xs)[tid + i * kThreads] = x[i];
    } else if (a.y) {
        float ss = 0.f;
        if (k_n % 4 == 0) {
            const float4 *y4 = reinterpret_cast<const float4 *>(a.y), *r4 = reinterpret_cast<const float4 *>(a.res), *g4 = reinterpret_cast<const float4 *>(a.gain);
            float4 *x4 = reinterpret_cast<float4 *>(xs);
            const int n4 = k_n / 4;
#pragma unroll 4
            for (int k = tid; k < n4; k += kThreads) {
                const float4 v = y4[k];
                x4[k] = v;
                ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
            }
            const float inv = inv_rms(ss);
#pragma unroll 1
            for (int k0 = tid; k0 < n4; k0 += 2 * kThreads) {  // two at a time: both loads before a store that might alias
                float4 r[2], g[2];
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (k0 + i * kThreads < n4) {
                        r[i] = r4[k0 + i * kThreads];
                        g[i] = g4[k0 + i * kThreads];
                    }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int k = k0 + i * kThreads;
                    if (k >= n4) break;
                    const float4 v = x4[k];
                    const float4 x = make_float4(__fadd_rn(r[i].x, __fmul_rn(__fmul_rn(v.x, inv), g[i].x)), __fadd_rn(r[i].y, __fmul_rn(__fmul_rn(v.y, inv), g[i].y)),
                                                 __fadd_rn(r[i].z, __fmul_rn(__fmul_rn(v.z, inv), g[i].z)), __fadd_rn(r[i].w, __fmul_rn(__fmul_rn(v.w, inv), g[i].w)));
                    x4[k] = x;
                    if (blockIdx.x == 0) reinterpret_cast<float4 *>(a.x_out)[k] = x;
                }
            }
        } else {
#pragma unroll 1
            for (int k = tid; k < k_n; k += kThreads) {
                const float v = a.y[k];
                xs[k] = v;
                ss = fmaf(v, v, ss);
            }
            const float inv = inv_rms(ss);
#pragma unroll 1
            for (int k = tid; k < k_n; k += kThreads) {
                const float x = __fadd_rn(a.res[k], __fmul_rn(__fmul_rn(xs[k], inv), a.gain[k]));
                xs[k] = x;
                if (blockIdx.x == 0) a.x_out[k] = x;
            }
        }
    } else if (k_n % 4 == 0) {
#pragma unroll 6
        for (int k = tid; k < k_n / 4; k += kThreads) reinterpret_cast<float4 *>(xs)[k] = reinterpret_cast<const float4 *>(a.res)[k];
    } else {
#pragma unroll 1
        for (int k = tid; k < k_n; k += kThreads) xs[k] = a.res[k];
    }
    if (a.norm_w && !held) {
        __syncthreads();
        float ss = 0.f;
        if (k_n % 4 == 0) {
            float4 *x4 = reinterpret_cast<float4 *>(xs);
            const float4 *g4 = reinterpret_cast<const float4 *>(a.norm_w);
#pragma unroll 2
            for (int k = tid; k < k_n / 4; k += kThreads) {
                const float4 v = x4[k];
                ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
            }
            const float inv = inv_rms(ss);
#pragma unroll 2
            for (int k = tid; k < k_n / 4; k += kThreads) {
                const float4 v = x4[k], g = g4[k];
                x4[k] = make_float4(__fmul_rn(__fmul_rn(v.x, inv), g.x), __fmul_rn(__fmul_rn(v.y, inv), g.y), __fmul_rn(__fmul_rn(v.z, inv), g.z),
                                    __fmul_rn(__fmul_rn(v.w, inv), g.w));
            }
        } else {
#pragma unroll 1
            for (int k = tid; k < k_n; k += kThreads) ss = fmaf(xs[k], xs[k], ss);
            const float inv = inv_rms(ss);
#pragma unroll 1
            for (int k = tid; k < k_n; k += kThreads) xs[k] = __fmul_rn(__fmul_rn(xs[k], inv), a.norm_w[k]);
        }
    }
    __syncthreads();
}
// Requests the gains (before pdl_wait); returns whether there are any to keep.
__device__ __forceinline__ bool step_request_gains(const GemvStepArgs &a, float *gains, float *norms) {
    if (step_gains(a) == 0) return false;
    for (int k = threadIdx.x; k < (int)a.K / 4; k += kThreads) {
        if (a.y) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(gains + 4 * k)), "l"(a.gain + 4 * k) : "memory");
        if (a.norm_w) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(norms + 4 * k)), "l"(a.norm_w + 4 * k) : "memory");
    }
    return true;
}
// What the last product of a step does besides (see GemvStepArgs).
__device__ __forceinline__ void step_end(const GemvStepArgs &a) {
    if (!a.d_lens || blockIdx.x != gridDim.x - 1) return;
    for (int l = threadIdx.x; l < a.layers; l += kThreads) a.d_lens[l] += 1;
    if (threadIdx.x == 0) *a.last_tok = (int)id_to_index(a.ids[0]);
}
template <typename WT>
__device__ __forceinline__ float step_act(const GemvStepArgs &a, float v, size_t row) {
    if (a.act != StepFinish::kStore) v = gelu_tanh(v);
    if (a.act == StepFinish::kSideGate) {
        const unsigned long long tok = id_to_index(a.ids[0]);
        v *= tok < a.table_rows ? to_f32(static_cast<const WT *>(a.table)[tok * a.table_ld + row]) : 0.f;
    }
    return v;
}

// One row whose input may still owe the norm of a sublayer's output (post-norm models): x = res + RMSNorm(y) * gain is
// formed by every CTA while it stages x, so that the norm, the residual sum and the product are one launch.  WPR warps share a
// weight row (a slice of K each) where there are too few rows to keep enough loads in flight.
// GATED: N gate rows and the N up rows that go with them (in blocks, see kGateBlock) are walked as pairs; out = gelu_tanh(gate) * up.
template <typename WT, int WPR, bool GATED>
__global__ void __launch_bounds__(kThreads, kStepCtas) gemv_step_kernel(const GemvStepArgs a) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float red[kWarps], red2[kWarps];
    float *xs = smem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int VEC = 16 / sizeof(WT), kRows = kWarps / WPR;
    const int part = warp % WPR;
    const size_t K = a.K, n_rows = GATED ? 2 * a.N : a.N, row0 = (size_t)blockIdx.x * kRows + warp / WPR;
    const WT *w = static_cast<const WT *>(a.w);
    // where row r of the walk is stored (GATED: r = 2 * i for gate row i, 2 * i + 1 for up row i)
    auto stored = [&](size_t r) {
        if (!GATED) return r;
        const size_t i = r >> 1;
        return i / kGateBlock * (2 * kGateBlock) + i % kGateBlock + (r & 1) * kGateBlock;
    };
    const bool vec_ok = (K % VEC == 0) && ((reinterpret_cast<uintptr_t>(w) & 15) == 0);
    // this warp's slice of K, in whole vectors
    const int nv = (int)(K / VEC), per = (nv + WPR - 1) / WPR, v0 = min(nv, part * per), vn = min(nv - v0, per);
    uint4 pre[kAhead];
    if (vec_ok && row0 < n_rows) row_ahead(reinterpret_cast<const uint4 *>(w + stored(row0) * K) + v0, vn, lane, pre);
    // Rows of up to 2048 numbers with norms: the gains are in shared memory before the wait ends, and what there is to read behind it
    // (y and the residual) is one batch of loads held in registers, with one barrier per sum.  A step of six Fekorax layers 183 -> 173 us, of eight
    // Fegetar layers 428 -> 417 (with the end of the step in its last product).
    float *gains = smem + K, *norms = gains + (a.y ? K : 0);
    const bool held = step_request_gains(a, gains, norms);
    pdl_launch();
    pdl_wait();
    step_stage(a, xs, gains, norms, held, red, red2);
#pragma unroll 1
    for (size_t base = (size_t)blockIdx.x * kRows; base < n_rows; base += (size_t)gridDim.x * kRows) {
        const size_t row = base + warp / WPR;
        float v = 0.f;
        if (row < n_rows) {
            if (vec_ok) {
                const size_t after = row + (size_t)gridDim.x * kRows;
                const uint4 *wrow = reinterpret_cast<const uint4 *>(w + stored(row) * K) + v0;
                const uint4 *next = after < n_rows ? reinterpret_cast<const uint4 *>(w + stored(after) * K) + v0 : nullptr;
                v = row_dot_ahead<WT>(wrow, xs + v0 * VEC, vn, lane, pre, next);
            } else if (part == 0) {
                v = row_dot_scalar<WT>(w + stored(row) * K, xs, (int)K, lane);
            }
        }
        v = warp_sum(v);
        if (GATED) {  // slices and the two rows of a pair meet in the pair's first warp (kRows is even, so a pair shares a CTA)
            if (lane == 0) red[warp] = v;
            __syncthreads();
            if (lane == 0 && part == 0 && (row & 1) == 0 && row < n_rows) {
                float g = 0.f, u = 0.f;
#pragma unroll
                for (int i = 0; i < WPR; ++i) {
                    g += red[warp + i];
                    u += red[warp + WPR + i];
                }
                a.out[row >> 1] = gelu_tanh(g) * u;
            }
            __syncthreads();
            continue;
        }
        if (WPR > 1) {  // the row's slices meet in its first warp
            if (lane == 0) red[warp] = v;
            __syncthreads();
            v = 0.f;
#pragma unroll
            for (int i = 0; i < WPR; ++i) v += red[(warp / WPR) * WPR + i];
            __syncthreads();
        }
        if (lane == 0 && part == 0 && row < n_rows) {
            a.out[row] = step_act<WT>(a, v, row);
        }
    }
    step_end(a);
}

// The same for many rows of bf16 weights: a warp (or WPR warps, a slice of K each) takes two rows at a time, as in gemv_vec_pair_kernel.
// GATED: a gate row and the up row that goes with it, so that nothing but the slices has to meet in shared memory.
// What bounds it: HBM for the matrices of a few MB, and the way of x through shared memory, which two rows share.  A step of eight Fegetar
// layers 416 -> 381 us at 96 positions (442 -> 406 at 1900), of six Fekorax layers 165 -> 149.
template <int WPR, bool GATED>
__global__ void __launch_bounds__(kThreads, 2) gemv_step_pair_kernel(const GemvStepArgs a) {
    using WT = __nv_bfloat16;
    extern __shared__ __align__(16) float smem[];
    __shared__ float red[kWarps], red2[kWarps];
    __shared__ float2 part_s[kWarps];
    constexpr int VEC = 16 / sizeof(WT), kPairs = kWarps / WPR;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = warp % WPR;
    const size_t K = a.K, N = a.N, pairs = GATED ? N : (N + 1) / 2, p0 = (size_t)blockIdx.x * kPairs + warp / WPR, step = (size_t)gridDim.x * kPairs;
    const int nv = (int)(K / VEC), per = (nv + WPR - 1) / WPR, v0 = min(nv, part * per), vn = min(nv - v0, per);
    const WT *w = static_cast<const WT *>(a.w);
    auto at = [&](size_t p, int r) {
        const size_t row = GATED ? p / kGateBlock * (2 * kGateBlock) + p % kGateBlock + r * kGateBlock : min(2 * p + r, N - 1);
        return reinterpret_cast<const uint4 *>(w + row * K) + v0;
    };
    uint4 cur[2][kAhead];
    if (p0 < pairs)
#pragma unroll
        for (int r = 0; r < 2; ++r) row_ahead(at(p0, r), vn, lane, cur[r]);
    float *xs = smem, *gains = smem + K, *norms = gains + (a.y ? K : 0);
    const bool held = step_request_gains(a, gains, norms);
    pdl_launch();
    pdl_wait();
    step_stage(a, xs, gains, norms, held, red, red2);
#pragma unroll 1
    for (size_t base = (size_t)blockIdx.x * kPairs; base < pairs; base += step) {
        const size_t p = base + warp / WPR;
        float v[2] = {0.f, 0.f};
        if (p < pairs) {
            const bool more = p + step < pairs;
            pair_dot_ahead(at(p, 0), at(p, 1), xs + v0 * VEC, vn, lane, cur, more ? at(p + step, 0) : nullptr, more ? at(p + step, 1) : nullptr, v);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
            v[1] += __shfl_xor_sync(0xffffffffu, v[1], o);
        }
        if (WPR > 1) {  // the rows' slices meet in their first warp
            if (lane == 0) part_s[warp] = make_float2(v[0], v[1]);
            __syncthreads();
            v[0] = v[1] = 0.f;
#pragma unroll
            for (int i = 0; i < WPR; ++i) {
                v[0] += part_s[warp / WPR * WPR + i].x;
                v[1] += part_s[warp / WPR * WPR + i].y;
            }
            __syncthreads();
        }
        if (part != 0 || p >= pairs) continue;
        if (GATED) {
            if (lane == 0) a.out[p] = gelu_tanh(v[0]) * v[1];
        } else if (lane < 2 && 2 * p + lane < N) {
            a.out[2 * p + lane] = step_act<WT>(a, lane ? v[1] : v[0], 2 * p + lane);
        }
    }
    step_end(a);
}

// ---- [K,N] row-major layout ---------------------------------------------------------------------
// y[n] = sum_k w[k,n] x[k].  A warp walks rows of a tile of columns, LW lanes side by side (16 bytes each: VEC adjacent columns a
// lane) and 32 / LW rows at once; the CTA's eight warps take the rows in turn, the CTAs of a cluster take a slice of K each.  Partial
// sums meet in shared memory and, across the slices, in `part` (slices added in order: deterministic, no atomics).
// Rows that do not start on 16 bytes (N not a multiple of VEC) are read in whole aligned vectors all the same: a thread's rows
// lie a multiple of eight apart, so all of them are `shift` elements off alignment, and its sums belong `shift` columns further
// left; a tile is one vector narrower than what a warp reads.
// Why this split: HBM wants some 45 KB in flight per SM (two or three CTAs of 256 threads with eight 16-byte loads each), in lines
// of 128 bytes or more; everything behind that is overhead: calls overlap like those of gemv_vec_kernel.  [4096,11008] bf16, calls behind one
// another: 18.4 us (4.9 TB/s; 21.9 without the overlap, 34.8 with 108 slices per column, whose sums a second kernel had to read back).
constexpr int kKnWarps = 8, kKnUnroll = 8, kKnChunk = 2048, kKnSplits = 8;
__host__ __device__ constexpr int kn_tile_cols(int lw, int vec, bool whole) { return (whole ? lw : lw - 1) * vec; }

template <typename WT, int LW>
__global__ void __launch_bounds__(kKnWarps * 32, 3)
gemv_kn_kernel(const float *x, const WT *w, float *part, float *y, size_t K, size_t N, size_t k_per_split) {
    constexpr int VEC = 16 / sizeof(WT), RPW = 32 / LW, ROWS = kKnWarps * RPW;
    static_assert(ROWS % 8 == 0, "a thread's rows share their alignment");
    __shared__ float xs[kKnChunk];
    __shared__ __align__(16) float red[kKnWarps * 32 * VEC];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = lane % LW, row = warp * RPW + lane / LW;
    const bool aligned = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
    const int tile = kn_tile_cols(LW, VEC, N % VEC == 0);
    const size_t c0 = (size_t)blockIdx.x * tile, k0 = min(K, (size_t)blockIdx.y * k_per_split), k1 = min(K, k0 + k_per_split), total = K * N;
    auto shift_of = [&](int r) { return (int)(((k0 + r) % VEC * (N % VEC) + c0) % VEC); };
    const int shift = shift_of(row);
    const bool active = c0 + (size_t)sub * VEC < N + shift;
    const size_t first = (k0 + row) * N + c0 - shift + (size_t)sub * VEC;  // of this thread's elements
    auto fetch = [&](size_t kk) {  // row k0 + row + kk
        const size_t at = first + kk * N;
        if (aligned && at + VEC <= total) return ld_live_u4(reinterpret_cast<const uint4 *>(w + at));
        uint4 v = make_uint4(0u, 0u, 0u, 0u);  // the last elements of the matrix, or a matrix that starts anywhere
        WT *e = reinterpret_cast<WT *>(&v);
        for (int i = 0; i < VEC; ++i)
            if (at + i < total) e[i] = w[at + i];
        return v;
    };
    if (active && k0 + row < k1)
#pragma unroll 1
        for (int u = 0; u < kKnUnroll && k0 + row + u * ROWS < k1; ++u) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + min(first + (size_t)u * ROWS * N, total - 1)));
    pdl_wait();
    float acc[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (size_t kb = k0; kb < k1; kb += kKnChunk) {
        const int kn = (int)min((size_t)kKnChunk, k1 - kb);
        uint4 wv[kKnUnroll];
#pragma unroll
        for (int u = 0; u < kKnUnroll; ++u) wv[u] = active && row + u * ROWS < kn ? fetch(kb - k0 + u * ROWS) : zero;
        __syncthreads();
        for (int i = tid; i < kn; i += kKnWarps * 32) xs[i] = x[kb + i];
        __syncthreads();
        for (int r = row; r < kn;) {
#pragma unroll
            for (int u = 0; u < kKnUnroll; ++u) {
                const float xv = r + u * ROWS < kn ? xs[r + u * ROWS] : 0.f;
                if constexpr (sizeof(WT) == 4) {
                    acc[0] = fmaf(__uint_as_float(wv[u].x), xv, acc[0]);
                    acc[1] = fmaf(__uint_as_float(wv[u].y), xv, acc[1]);
                    acc[2] = fmaf(__uint_as_float(wv[u].z), xv, acc[2]);
                    acc[3] = fmaf(__uint_as_float(wv[u].w), xv, acc[3]);
                } else {
                    acc[0] = fmaf(bf16_lo(wv[u].x), xv, acc[0]);
                    acc[1] = fmaf(bf16_hi(wv[u].x), xv, acc[1]);
                    acc[2] = fmaf(bf16_lo(wv[u].y), xv, acc[2]);
                    acc[3] = fmaf(bf16_hi(wv[u].y), xv, acc[3]);
                    acc[4] = fmaf(bf16_lo(wv[u].z), xv, acc[4]);
                    acc[5] = fmaf(bf16_hi(wv[u].z), xv, acc[5]);
                    acc[6] = fmaf(bf16_lo(wv[u].w), xv, acc[6]);
                    acc[7] = fmaf(bf16_hi(wv[u].w), xv, acc[7]);
                }
            }
            r += kKnUnroll * ROWS;
#pragma unroll
            for (int u = 0; u < kKnUnroll; ++u) wv[u] = active && r + u * ROWS < kn ? fetch(kb - k0 + (r - row) + u * ROWS) : zero;
        }
    }
    pdl_launch();  // (from the start on, the next call's CTAs would take turns with this one's: [4096,32000] bf16 58.2 us instead of 55.8)
#pragma unroll
    for (int v = 0; v < VEC; v += 4)
        *reinterpret_cast<float4 *>(red + (warp * 32 + lane) * VEC + v) = make_float4(acc[v], acc[v + 1], acc[v + 2], acc[v + 3]);
    __syncthreads();
    const bool sliced = gridDim.y > 1;
    for (int c = tid; c < tile && c0 + c < N; c += kKnWarps * 32) {
        float s = 0.f;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) s += red[r * LW * VEC + c + shift_of(r)];
        if (sliced) part[(size_t)blockIdx.y * N + c0 + c] = s;
        else y[c0 + c] = s;
    }
    if (!sliced) return;
    __threadfence();
    cooperative_groups::this_cluster().sync();  // (grid.y is the cluster)
    const int per = (tile + gridDim.y - 1) / gridDim.y, end = min(tile, (int)(blockIdx.y + 1) * per);
    for (int c = blockIdx.y * per + tid; c < end && c0 + c < N; c += kKnWarps * 32) {
        float s = 0.f;
#pragma unroll 8
        for (int i = 0; i < (int)gridDim.y; ++i) s += __ldcg(part + (size_t)i * N + c0 + c);
        y[c0 + c] = s;
    }
}

struct KnPlan {
    int lanes, col_blocks, splits;
    size_t k_per_split;
};

// Tiles as wide as leave two CTAs per SM with K cut in eight; no more slices than that takes (a slice has at least four
// rows per thread), and no more CTAs than are resident, three per SM (500 CTAs for [4096,32000] bf16 took 63 us, 250 take 57).
KnPlan plan_kn(size_t K, size_t N, int vec, int num_sms) {
    KnPlan p;
    const size_t want = 2 * (size_t)num_sms;
    size_t blocks = 0;
    for (p.lanes = 32; p.lanes >= 8; p.lanes /= 2) {
        const size_t tile = kn_tile_cols(p.lanes, vec, N % vec == 0);
        blocks = (N + tile - 1) / tile;
        if (blocks * kKnSplits >= want || p.lanes == 8) break;
    }
    p.col_blocks = (int)blocks;
    const size_t rows = (size_t)kKnWarps * 32 / p.lanes;
    p.splits = 1;
    while (p.splits < kKnSplits && blocks * p.splits < want && 2 * blocks * p.splits <= 3 * (size_t)num_sms && K > (size_t)p.splits * rows * 4) p.splits *= 2;
    p.k_per_split = ((K + p.splits - 1) / p.splits + rows - 1) / rows * rows;
    return p;
}

int pick_grid(lumen_ctx *ctx, size_t rows, size_t smem_bytes) {
    // Resident CTAs per SM limited by shared memory (227 KB) and by 2048 threads.
    int per_sm = (int)std::min<size_t>(8, (227 * 1024) / std::max<size_t>(smem_bytes + 1024, 1));
    per_sm = std::max(per_sm, 1);
    size_t want = (rows + kWarps - 1) / kWarps;
    size_t cap = (size_t)ctx->num_sms * per_sm;
    return (int)std::max<size_t>(1, std::min(want, cap));
}

template <typename WT, int MB>
int launch_nk_t(lumen_ctx *ctx, const GemvArgs &a, cudaStream_t s) {
    size_t smem = (size_t)MB * a.K * sizeof(float);
    auto kern = gemv_nk_kernel<WT, MB>;
    LUMEN_TRY(allow_smem(ctx, kern, smem));
    int grid = pick_grid(ctx, a.N, smem);
    kern<<<grid, kThreads, smem, s>>>(a.x, static_cast<const WT *>(a.w), a.y, a.M, a.K, a.N, a.ldy, a.norm_w,
                                      a.norm_eps, a.residual);
    LUMEN_LAUNCHED(ctx);
    return LUMEN_OK;
}

template <typename WT, int MB>
int launch_gate_up_t(lumen_ctx *ctx, const float *x, const void *wg, const void *wu, float *out, int M, size_t K,
                     size_t I, const float *norm_w, float eps, cudaStream_t s) {
    size_t smem = (size_t)MB * K * sizeof(float);
    auto kern = gemv_gate_up_kernel<WT, MB>;
    LUMEN_TRY(allow_smem(ctx, kern, smem));
    int grid = pick_grid(ctx, I, smem);
    kern<<<grid, kThreads, smem, s>>>(x, static_cast<const WT *>(wg), static_cast<const WT *>(wu), out, M, K, I, norm_w,
                                      eps);
    LUMEN_LAUNCHED(ctx);
    return LUMEN_OK;
}

}  // namespace

int launch_gemv_nk(lumen_ctx *ctx, const GemvArgs &a, cudaStream_t s) {
    if (a.M < 1 || a.M > 8) return set_error(ctx, LUMEN_ERR_INVALID, "gemv: M=%d outside 1..8", a.M);
    if ((size_t)a.M * a.K * 4 > 200 * 1024) return set_error(ctx, LUMEN_ERR_UNSUPPORTED, "gemv: M*K too large for staging");
    const int mb = a.M == 1 ? 1 : a.M == 2 ? 2 : a.M <= 4 ? 4 : 8;
    const bool f32 = a.wdt == LUMEN_F32;
    switch (mb) {
        case 1: return f32 ? launch_nk_t<float, 1>(ctx, a, s) : launch_nk_t<__nv_bfloat16, 1>(ctx, a, s);
        case 2: return f32 ? launch_nk_t<float, 2>(ctx, a, s) : launch_nk_t<__nv_bfloat16, 2>(ctx, a, s);
        case 4: return f32 ? launch_nk_t<float, 4>(ctx, a, s) : launch_nk_t<__nv_bfloat16, 4>(ctx, a, s);
        default: return f32 ? launch_nk_t<float, 8>(ctx, a, s) : launch_nk_t<__nv_bfloat16, 8>(ctx, a, s);
    }
}

// y = W x for one vector (see gemv_vec_kernel); false: not a call for it.
bool gemv_vec_usable(const void *w, lumen_dtype wdt, size_t K) {
    return K % (wdt == LUMEN_F32 ? 4 : 8) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && K * 4 <= 100 * 1024;
}
int launch_gemv_vec(lumen_ctx *ctx, const float *x, const void *w, lumen_dtype wdt, float *y, size_t K, size_t N, cudaStream_t s) {
    const size_t smem = K * sizeof(float), row_bytes = K * (wdt == LUMEN_F32 ? 4 : 2), want = (size_t)ctx->num_sms * 4 * kWarps;
    // warps per row: enough warps for four CTAs per SM, a slice of at least 1 KB each
    int wpr = 1;
    while (wpr < 8 && N * wpr * 2 <= want && row_bytes >= 2048u * wpr) wpr *= 2;
    const int grid = std::min(pick_grid(ctx, N * wpr, smem), ctx->num_sms * 4);
    const bool pdl = ctx->pdl;
    ctx->pdl = true;
    int rc;
    if (wpr == 1 && wdt == LUMEN_BF16 && row_bytes >= 2048) {
        const int pairs = (int)std::min<size_t>(((N + 1) / 2 + kWarps - 1) / kWarps, (size_t)ctx->num_sms * 2);
        rc = allow_smem(ctx, gemv_vec_pair_kernel, smem);
        if (rc == LUMEN_OK) rc = launch_pdl(ctx, gemv_vec_pair_kernel, pairs, kThreads, smem, s, x, static_cast<const __nv_bfloat16 *>(w), y, (int)K, N);
        ctx->pdl = pdl;
        return rc;
    }
#define LUMEN_VEC(T_, W_) rc = allow_smem(ctx, gemv_vec_kernel<T_, W_>, smem); if (rc == LUMEN_OK) rc = launch_pdl(ctx, gemv_vec_kernel<T_, W_>, grid, kThreads, smem, s, x, static_cast<const T_ *>(w), y, (int)K, N)
#define LUMEN_VEC_T(T_) do { if (wpr == 8) { LUMEN_VEC(T_, 8); } else if (wpr == 4) { LUMEN_VEC(T_, 4); } else if (wpr == 2) { LUMEN_VEC(T_, 2); } else { LUMEN_VEC(T_, 1); } } while (0)
    if (wdt == LUMEN_F32) LUMEN_VEC_T(float);
    else LUMEN_VEC_T(__nv_bfloat16);
#undef LUMEN_VEC_T
#undef LUMEN_VEC
    ctx->pdl = pdl;
    return rc;
}

int launch_gemv_gate_up(lumen_ctx *ctx, const float *x, const void *w_gate, const void *w_up, lumen_dtype wdt,
                        float *out, int M, size_t K, size_t I, const float *norm_w, float norm_eps, cudaStream_t s) {
    if (M < 1 || M > 8) return set_error(ctx, LUMEN_ERR_INVALID, "gate_up: M=%d outside 1..8", M);
    if ((size_t)M * K * 4 > 200 * 1024) return set_error(ctx, LUMEN_ERR_UNSUPPORTED, "gate_up: M*K too large for staging");
    const int mb = M == 1 ? 1 : M == 2 ? 2 : M <= 4 ? 4 : 8;
    const bool f32 = wdt == LUMEN_F32;
#define GU(T, B) launch_gate_up_t<T, B>(ctx, x, w_gate, w_up, out, M, K, I, norm_w, norm_eps, s)
    switch (mb) {
        case 1: return f32 ? GU(float, 1) : GU(__nv_bfloat16, 1);
        case 2: return f32 ? GU(float, 2) : GU(__nv_bfloat16, 2);
        case 4: return f32 ? GU(float, 4) : GU(__nv_bfloat16, 4);
        default: return f32 ? GU(float, 8) : GU(__nv_bfloat16, 8);
    }
#undef GU
}

int launch_gemv_step(lumen_ctx *ctx, const GemvStepArgs &a, cudaStream_t s) {
    const size_t smem = (a.K + step_gains(a)) * sizeof(float);
    if (smem > 200 * 1024) return set_error(ctx, LUMEN_ERR_UNSUPPORTED, "gemv_step: row of %zu elements", a.K);
    // warps per row: enough warps for about three CTAs per SM, a slice of at least 1 KB each
    const size_t row_bytes = a.K * (a.wdt == LUMEN_F32 ? 4 : 2), want = (size_t)ctx->num_sms * 3 * kWarps;
    const bool gated = a.act == StepFinish::kGated;
    const size_t rows = gated ? 2 * a.N : a.N;
    // Two rows per warp where there are more pairs than half of its warps, or where their long rows make up for it
    const size_t pair_warps = (size_t)ctx->num_sms * 2 * kWarps, pairs = gated ? a.N : (a.N + 1) / 2;
    const bool split = pairs * 2 <= pair_warps && row_bytes >= 8192;
    if (a.wdt == LUMEN_BF16 && a.K % 8 == 0 && (reinterpret_cast<uintptr_t>(a.w) & 15) == 0 && row_bytes >= 2048 && (split || pairs * 2 > pair_warps)) {
        const int g2 = (int)std::min((pairs * (split ? 2 : 1) + kWarps - 1) / kWarps, pair_warps / kWarps);
#define LUMEN_PAIR(W_, G_)                                                                            \
    do {                                                                                              \
        LUMEN_TRY(allow_smem(ctx, gemv_step_pair_kernel<W_, G_>, smem));                                \
        return launch_pdl(ctx, gemv_step_pair_kernel<W_, G_>, g2, kThreads, smem, s, a);              \
    } while (0)
        if (gated) {
            if (split) LUMEN_PAIR(2, true);
            LUMEN_PAIR(1, true);
        }
        if (split) LUMEN_PAIR(2, false);
        LUMEN_PAIR(1, false);
#undef LUMEN_PAIR
    }
    const int wpr = rows * 4 <= want && row_bytes >= 4096 ? 4 : rows * 2 <= want && row_bytes >= 2048 ? 2 : row_bytes >= 8192 && rows * 2 <= 2 * want ? 2 : 1;
    // as many CTAs as the device holds: each stages its input once
    const int grid = std::min(pick_grid(ctx, rows * wpr, smem), ctx->num_sms * kStepCtas);
#define LUMEN_STEP_G(T_, W_, G_)                                                               \
    do {                                                                                       \
        LUMEN_TRY(allow_smem(ctx, gemv_step_kernel<T_, W_, G_>, smem));                          \
        return launch_pdl(ctx, gemv_step_kernel<T_, W_, G_>, grid, kThreads, smem, s, a);      \
    } while (0)
#define LUMEN_STEP(T_, W_)                                                                     \
    do {                                                                                       \
        if (gated) LUMEN_STEP_G(T_, W_, true);                                                 \
        LUMEN_STEP_G(T_, W_, false);                                                           \
    } while (0)
    if (a.wdt == LUMEN_F32) {
        if (wpr == 4) LUMEN_STEP(float, 4);
        if (wpr == 2) LUMEN_STEP(float, 2);
        LUMEN_STEP(float, 1);
    }
    if (wpr == 4) LUMEN_STEP(__nv_bfloat16, 4);
    if (wpr == 2) LUMEN_STEP(__nv_bfloat16, 2);
    LUMEN_STEP(__nv_bfloat16, 1);
#undef LUMEN_STEP
#undef LUMEN_STEP_G
}

size_t gemv_kn_scratch_bytes_for(size_t K, size_t N, lumen_dtype wdt, int num_sms) {
    return (size_t)plan_kn(K, N, wdt == LUMEN_F32 ? 4 : 8, num_sms).splits * N * sizeof(float);
}

size_t gemv_kn_scratch_bytes(size_t K, size_t N, int num_sms) {
    KnPlan p4 = plan_kn(K, N, 4, num_sms), p8 = plan_kn(K, N, 8, num_sms);
    return (size_t)std::max(p4.splits, p8.splits) * N * sizeof(float);
}

int launch_gemv_kn(lumen_ctx *ctx, const float *x, const void *w, lumen_dtype wdt, float *y, size_t K, size_t N,
                   float *scratch, cudaStream_t s) {
    const KnPlan p = plan_kn(K, N, wdt == LUMEN_F32 ? 4 : 8, ctx->num_sms);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.col_blocks, p.splits);
    cfg.blockDim = dim3(kKnWarps * 32);
    cfg.stream = s;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {1, (unsigned)p.splits, 1};
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
#define LUMEN_KN(T_, L_) cudaLaunchKernelEx(&cfg, gemv_kn_kernel<T_, L_>, x, static_cast<const T_ *>(w), scratch, y, K, N, p.k_per_split)
    if (wdt == LUMEN_F32) LUMEN_CUDA(ctx, p.lanes == 32 ? LUMEN_KN(float, 32) : p.lanes == 16 ? LUMEN_KN(float, 16) : LUMEN_KN(float, 8));
    else LUMEN_CUDA(ctx, p.lanes == 32 ? LUMEN_KN(__nv_bfloat16, 32) : p.lanes == 16 ? LUMEN_KN(__nv_bfloat16, 16) : LUMEN_KN(__nv_bfloat16, 8));
#undef LUMEN_KN
    LUMEN_LAUNCHED(ctx);
    return LUMEN_OK;
}

}  // namespace lumen
