// Nucleus sampling on the device: `sample_top_p` of the reference's chat loop (src/main.rs:74-137), so that
// one token id crosses PCIe per step instead of the logits vector.
//
// Same steps as the reference: repetition penalty over the recent tokens (one division per occurrence),
// temperature (floored at 1e-5), softmax with 1/(sum + 1e-9), stable descending sort, nucleus cut at the
// first rank where the cumulative probability reaches top_p (clamped to [1e-6, 1]), inverse-CDF walk over
// probs[i] / cumulative with the caller's uniform draw.  The cumulative sums carry the roundings of the reference's
// sequential f32 loops; the softmax denominator is a tree sum (the reference adds it sequentially), which
// moves every probability by the same last-ulp factor and the result only when the draw sits on a boundary.
// One kernel on a cluster of eight SMs serves what chat loops ask for (sample_nucleus_kernel).  What it cannot hold
// (nuclei that reach into probabilities below 2^-24, hundreds of nearly equal probabilities, vocabularies of more than
// kNucleusMaxVocab, NaN) takes a kernel that forms the probabilities, cub::DeviceRadixSort (a library sort: not the hot
// path) and a kernel that walks the sorted list.
#include <chrono>
#include <climits>
#include <thread>

#include <cooperative_groups.h>

#include <cub/cub.cuh>

#include "common.cuh"

namespace lumen {
namespace {

constexpr int kPrepThreads = 1024;
constexpr int kMaxRecent = 256;  // the reference keeps a window of 96 tokens (src/main.rs:300-313)

__device__ __forceinline__ float block_reduce(float v, float *red, bool is_max) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float t = __shfl_xor_sync(0xffffffffu, v, o);
        v = is_max ? fmaxf(v, t) : v + t;
    }
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float x = lane < (int)(blockDim.x >> 5) ? red[lane] : (is_max ? -INFINITY : 0.f);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float t = __shfl_xor_sync(0xffffffffu, x, o);
            x = is_max ? fmaxf(x, t) : x + t;
        }
        if (lane == 0) red[32] = x;
    }
    __syncthreads();
    const float out = red[32];
    __syncthreads();
    return out;
}

// One CTA: probabilities of the adjusted logits and the identity permutation.
__global__ void __launch_bounds__(kPrepThreads)
sample_prep_kernel(const float *__restrict__ logits, int n, float temperature, float penalty, const int *__restrict__ recent,
                   int n_recent, float *__restrict__ probs, int *__restrict__ idx) {
    __shared__ float red[33];
    __shared__ int rec[kMaxRecent];
    const int tid = threadIdx.x;
    for (int i = tid; i < n; i += kPrepThreads) probs[i] = logits[i];
    for (int i = tid; i < n_recent; i += kPrepThreads) rec[i] = recent[i];
    __syncthreads();
    if (penalty > 1.0f && tid < n_recent) {
        // the first occurrence of a token applies one division per occurrence (main.rs:83-89)
        const int t = rec[tid];
        bool first = t >= 0 && t < n;
        for (int k = 0; k < tid && first; ++k) first = rec[k] != t;
        if (first) {
            float x = probs[t];
            for (int k = tid; k < n_recent; ++k)
                if (rec[k] == t) x = __fdiv_rn(x, penalty);
            probs[t] = x;
        }
    }
    __syncthreads();
    const float temp = fmaxf(temperature, 1e-5f);
    float mx = -INFINITY;
    for (int i = tid; i < n; i += kPrepThreads) {
        const float x = __fdiv_rn(probs[i], temp);
        probs[i] = x;
        mx = fmaxf(mx, x);
    }
    mx = block_reduce(mx, red, true);
    float sum = 0.f;
    for (int i = tid; i < n; i += kPrepThreads) {
        const float e = expf(__fsub_rn(probs[i], mx));
        probs[i] = e;
        sum += e;
    }
    sum = block_reduce(sum, red, false);
    const float inv = __fdiv_rn(1.0f, __fadd_rn(sum, 1e-9f));
    for (int i = tid; i < n; i += kPrepThreads) {
        probs[i] = __fmul_rn(probs[i], inv);
        idx[i] = i;
    }
}

// The reference adds the sorted probabilities one by one in f32 and stops at the first index where the running sum
// reaches a threshold (main.rs:113-121 and :126-134).  With a flat distribution the rounding of that sequential sum
// decides the index, so its roundings are kept, but not its order in time: while the sum stays within a binade, its
// unit in the last place u is fixed and run / u is a whole number R, so that adding v >= 0 adds round(v / u) - which
// depends on R only where v / u lies halfway between two whole numbers (the even sum wins), that is on R's parity.  A value is
// therefore a function (parity of R) -> increment, the functions of consecutive values compose associatively, and a
// block-wide scan gives every running sum exactly.  The value that takes R past 2^24 is added in f32 and the scan starts over
// behind it with the next u: about one scan per doubling of the sum and one per 4096 values.  The first 256
// values, over which the sum doubles most often, are added one by one.  (One thread adding everything takes 4 cycles a value:
// 90 us for the two walks of a nucleus of 28800; a scan takes about 1 us.)
constexpr int kPickThreads = 1024;
constexpr int kPickWarps = kPickThreads / 32;
constexpr int kPickHead = 256;             // values added one by one first
constexpr uint32_t kPickFull = 1u << 24;   // R of the next binade
constexpr uint32_t kPickSat = 1u << 30;    // increments saturate here: past the end of the binade they are not used

struct PickShared {
    __align__(16) float head[kPickHead];
    uint2 total[2][kPickWarps];  // increments of a warp's values, for even and odd R (two sets: one is read while the next is written)
    int at[2][kPickWarps];       // a warp's first value that ends the scan (INT_MAX: none),
    uint32_t before[2][kPickWarps];  // R before it
    float val[2][kPickWarps];        // and the value
    int found;
    float run;
};

__device__ __forceinline__ uint2 pick_then(uint2 f, uint2 g) {  // f's values, then g's
    return make_uint2(min(f.x + ((f.x & 1) ? g.y : g.x), kPickSat), min(f.y + ((f.y & 1) ? g.x : g.y), kPickSat));
}
__device__ __forceinline__ uint2 pick_inc(float w) {  // w = v / u < 2^24
    const uint32_t q = (uint32_t)w;
    const float frac = w - (float)q;
    const uint32_t up = frac > 0.5f, tie = frac == 0.5f, odd = q & 1;
    return make_uint2(q + (up | (tie & odd)), q + (up | (tie & (odd ^ 1))));
}
__device__ __forceinline__ uint2 pick_scan(uint2 f, int lane) {  // inclusive, over the warp's lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint2 g = make_uint2(__shfl_up_sync(0xffffffffu, f.x, o), __shfl_up_sync(0xffffffffu, f.y, o));
        if (lane >= o) f = pick_then(g, f);
    }
    return f;
}

// First index < n whose running sum of vals[i] / scale is >= threshold (n if none), and that running sum (the total if none).
// vals is in descending order, all >= 0.  All kPickThreads threads call; the answers are the same in all of them.
template <bool SHARED>  // where the list is
__device__ __forceinline__ int first_reaching(const float *vals, int n, float scale, float threshold, PickShared &sh, float *sum_out) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float run = 0.f;
    int start = 0, turn = 0;  // values before `start` are in `run`
    for (int base = 0; base < n; base += 4 * kPickThreads) {
        const int i0 = base + 4 * tid;
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = i0 + q < n ? __fdiv_rn(SHARED ? vals[i0 + q] : __ldcg(vals + i0 + q), scale) : 0.f;
        if (base == 0) {
            if (4 * tid < kPickHead) *reinterpret_cast<float4 *>(sh.head + 4 * tid) = make_float4(v[0], v[1], v[2], v[3]);
            __syncthreads();
            if (tid == 0) {
                // 32 values per test of the threshold: eight 128-bit loads, then the dependent chain of 32 additions
                const int m = min(n, kPickHead);
                int found = -1;
                for (int i = 0; i < m && found < 0; i += 32) {
                    float4 x[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) x[j] = *reinterpret_cast<const float4 *>(sh.head + i + 4 * j);
                    float t = run;
#pragma unroll
                    for (int j = 0; j < 8; ++j) t = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(t, x[j].x), x[j].y), x[j].z), x[j].w);
                    if (!(t >= threshold)) {
                        run = t;
                        continue;
                    }
                    for (int j = i; j < m && found < 0; ++j) {  // the sums only grow: the crossing is inside these 32
                        run = __fadd_rn(run, sh.head[j]);
                        if (run >= threshold) found = j;
                    }
                }
                sh.found = found;
                sh.run = run;
            }
            __syncthreads();
            run = sh.run;
            start = kPickHead;
            const int found = sh.found;
            __syncthreads();  // everybody has read the words before the next walk writes them
            if (found >= 0 || n <= kPickHead || !(run > 0.f)) {  // (NaN reaches nothing; behind a sum of zero there are only zeros)
                *sum_out = run;
                return found >= 0 ? found : n;
            }
        }
        while (start < min(n, base + 4 * kPickThreads)) {
            // run in [2^(e-127), 2^(e-126)): u = 2^(e-150).  1 / n <= first value <= run < 2, so both powers are normal
            const uint32_t e = __float_as_uint(run) >> 23;
            const float per_u = __uint_as_float((277u - e) << 23), u = __uint_as_float((e - 23u) << 23);
            const uint32_t r0 = (uint32_t)(run * per_u);
            uint2 own[4], f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                own[q] = i0 + q >= start ? pick_inc(v[q] * per_u) : make_uint2(0u, 0u);
                f = q == 0 ? own[0] : pick_then(f, own[q]);
            }
            const uint2 in = pick_scan(f, lane);
            uint2 ex = make_uint2(__shfl_up_sync(0xffffffffu, in.x, 1), __shfl_up_sync(0xffffffffu, in.y, 1));
            if (lane == 0) ex = make_uint2(0u, 0u);
            if (lane == 31) sh.total[turn][warp] = in;
            __syncthreads();
            const uint2 w_in = pick_scan(sh.total[turn][lane], lane);
            const int prev = max(warp - 1, 0);
            uint2 w_ex = make_uint2(__shfl_sync(0xffffffffu, w_in.x, prev), __shfl_sync(0xffffffffu, w_in.y, prev));
            if (warp == 0) w_ex = make_uint2(0u, 0u);
            const uint2 all = make_uint2(__shfl_sync(0xffffffffu, w_in.x, 31), __shfl_sync(0xffffffffu, w_in.y, 31));
            ex = pick_then(w_ex, ex);
            uint32_t r = r0 + ((r0 & 1) ? ex.y : ex.x), before = r;
            int at = INT_MAX;
            float val = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t next = r + ((r & 1) ? own[q].y : own[q].x);
                if (at == INT_MAX && (next >= kPickFull || (float)next * u >= threshold)) {
                    at = i0 + q;
                    before = r;
                    val = v[q];
                }
                r = next;
            }
            const uint32_t hit = __ballot_sync(0xffffffffu, at != INT_MAX);
            if (hit ? lane == __ffs(hit) - 1 : lane == 0) {
                sh.at[turn][warp] = at;
                sh.before[turn][warp] = before;
                sh.val[turn][warp] = val;
            }
            __syncthreads();
            const uint32_t hits = __ballot_sync(0xffffffffu, sh.at[turn][lane] != INT_MAX);
            if (!hits) {
                run = (float)(r0 + ((r0 & 1) ? all.y : all.x)) * u;
                start = base + 4 * kPickThreads;
            } else {
                const int w = __ffs(hits) - 1;
                run = __fadd_rn((float)sh.before[turn][w] * u, sh.val[turn][w]);
                start = sh.at[turn][w] + 1;
                if (run >= threshold) {
                    *sum_out = run;
                    __syncthreads();  // (the next walk starts with the same set)
                    return start - 1;
                }
            }
            turn ^= 1;
        }
    }
    *sum_out = run;
    __syncthreads();
    return n;
}

// Rank of the drawn token in the sorted list.  `all`: the list is complete; otherwise -1 where it ends before the nucleus does.
template <bool SHARED>
__device__ __forceinline__ int pick_rank(const float *sorted_p, int n, bool all, float target, float r, PickShared &sh) {
    float cumulative, acc;
    const int at = first_reaching<SHARED>(sorted_p, n, 1.0f, target, sh, &cumulative);  // main.rs:113-121
    if (at == n && !all) return -1;
    const int cut = max(1, min(n, at + 1));
    // main.rs:126-134: acc += probs[i] / cumulative; the first i with r <= acc, else the last of the nucleus
    return min(first_reaching<SHARED>(sorted_p, cut, cumulative, r, sh, &acc), cut - 1);
}

__global__ void __launch_bounds__(kPickThreads)
sample_pick_kernel(const float *__restrict__ sorted_p, const int *__restrict__ sorted_i, int n, float target, float r, int *__restrict__ token_out) {
    __shared__ PickShared sh;
    const int pick = pick_rank<false>(sorted_p, n, true, target, r, sh);
    if (threadIdx.x == 0) *token_out = sorted_i[pick];
}

// ---- one kernel ---------------------------------------------------------------------------------------------------
// A cluster of eight CTAs holds the vocabulary in shared memory: CTA c owns the columns [128 c, 128 c + 128) of every 1024
// logits, the columns whose partial sums sample_prep_kernel's threads 128 c .. 128 c + 127 form, so that both kernels add the softmax
// denominator in the same order and agree on every bit of a probability.
// Only the nucleus is sorted.  The probabilities are counted by exponent and seven bits of mantissa (128 bins per octave, 24
// octaves); from the counts and the bins' lower edges every CTA finds the bin that certainly completes the nucleus, and the
// offsets of the bins in descending order.  The candidates are scattered into their bins (up to 2048 into CTA 0's shared memory, which
// ranks them alone; longer lists in global memory, tens of KB in the L2, ranked by all CTAs), and
// a candidate's rank within its bin is the number of larger ones (an equal probability of a smaller index is larger: the sort
// is stable).  CTA 0 then walks the list as the general path does.
// What bounds it is the chain of passes and cluster barriers, not bytes: hence one barrier per reduction (every warp hands its number to
// every CTA), counts of 16 bits (eight remote reads a thread), no trip to the L2 for short lists, and an answer that the
// host picks up by itself.  32000 logits of which some hundred to a thousand make the nucleus: 29 us a call (49 with remote reads behind
// local reductions, lists in the L2, and a copy and a wait for the stream behind the kernel; 140 with the seven kernels of the general path).
namespace cg = cooperative_groups;
constexpr int kCluster = 8;
constexpr int kNucleusBins = 24 * 128;
constexpr int kBinsPerThread = 4, kBinThreads = kNucleusBins / kBinsPerThread;
constexpr int kNear = 2048;  // a list of up to this many stays in the first CTA's shared memory
constexpr uint32_t kTopBin = 0x3f800000u >> 16;  // of probability 1
constexpr int kMaxBin = 512;                      // ranking is quadratic in a bin's size
constexpr int kNucleusMaxVocab = 256 * 1024;      // 128 KB of shared memory per CTA
static_assert(kPrepThreads == kPickThreads && kBinsPerThread * kBinThreads == kNucleusBins && kBinThreads <= kPrepThreads && kBinThreads % 32 == 0, "");
static_assert(kNucleusMaxVocab / kCluster < 65536, "a CTA's counts take 16 bits");

struct NucleusArgs {
    const float *logits;
    int n;
    float temperature, penalty, target, r;
    unsigned long long *cand;  // [n] probability bits : ~index
    float *sorted_p;           // [n]
    int *sorted_i;             // [n]
    const int *status;         // what kernels before this one reported
    unsigned long long *answer;  // pinned host memory: turn << 32 | token; the token is -1 where it is not served here, -2 after a report
    unsigned int turn;
    int n_recent;
    int recent[kMaxRecent];
};

struct NucleusShared {
    __align__(16) unsigned int hist[kNucleusBins / 2];          // counts here, two bins to a word
    int cursor[kNucleusBins], first[kNucleusBins + 1];          // next place; first place of a bin
    __align__(16) unsigned long long window[kPrepThreads / 32][32];
    __align__(16) unsigned long long cand[kNear];               // the first CTA's: candidates in their bins,
    float near_p[kNear];                                        // in order
    int near_i[kNear];
    float top[kCluster * kPrepThreads / 32], part[kCluster * 4];  // every warp's, of all CTAs
    int recent[kMaxRecent];
    int scan_n[32];
    float scan_m[32];
    int last_bin, crowded;
    PickShared pick;
};

__device__ __forceinline__ int bin_of(float p) { return (int)kTopBin - (int)(__float_as_uint(p) >> 16); }

__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kPrepThreads) sample_nucleus_kernel(const __grid_constant__ NucleusArgs a) {
    extern __shared__ __align__(16) unsigned char nucleus_smem[];
    NucleusShared &sh = *reinterpret_cast<NucleusShared *>(nucleus_smem);
    float *vals = reinterpret_cast<float *>(nucleus_smem + sizeof(NucleusShared));
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)cluster.block_rank(), n = a.n;
    const int slots = (n + 1023) / 1024 * 128;
    auto index_of = [&](int s) { return (s >> 7) * 1024 + rank * 128 + (s & 127); };
    auto answer = [&](int token) {  // one word, so that its turn says that the token is there
        const unsigned int t = __ldcg(a.status) ? (unsigned int)-2 : (unsigned int)token;
        asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(a.answer), "l"((unsigned long long)a.turn << 32 | t) : "memory");
    };
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");  // (this CTA runs: the others may write to its shared memory)
    for (int s = tid; s < slots; s += kPrepThreads) {
        if (index_of(s) < n)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(vals + s)), "l"(a.logits + index_of(s)) : "memory");
        else vals[s] = -INFINITY;
    }
    for (int b = tid; b < kNucleusBins / 2; b += kPrepThreads) sh.hist[b] = 0;
    if (tid < a.n_recent) sh.recent[tid] = a.recent[tid];
    if (tid == 0) {
        sh.last_bin = INT_MAX;
        sh.crowded = 0;
    }
    __syncthreads();
    // (the recent tokens are counted while the logits are on their way)
    int times = 0, token = -1;  // occurrences of thread t's recent token, if it is the first and in this CTA's columns
    if (a.penalty > 1.0f && tid < a.n_recent) {
        // the first occurrence of a token applies one division per occurrence (main.rs:83-89)
        token = sh.recent[tid];
        int before = 0;
#pragma unroll 8
        for (int k = 0; k < a.n_recent; ++k) {
            const int same = sh.recent[k] == token;
            times += same;
            before += k < tid ? same : 0;
        }
        if (before != 0 || token < 0 || token >= n || ((token >> 7) & (kCluster - 1)) != rank) token = -1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (token >= 0) {
        float x = vals[(token >> 10) * 128 + (token & 127)];
        for (int k = 0; k < times; ++k) x = __fdiv_rn(x, a.penalty);
        vals[(token >> 10) * 128 + (token & 127)] = x;
    }
    __syncthreads();
    const float temp = fmaxf(a.temperature, 1e-5f);
    float mx = -INFINITY;
    for (int s = tid; s < slots; s += kPrepThreads) {
        const float x = __fdiv_rn(vals[s], temp);
        vals[s] = x;
        if (index_of(s) < n) mx = fmaxf(mx, x);
    }
    // Every warp hands its maximum to every CTA, so that one barrier is all that lies between.
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (lane < kCluster) *cluster.map_shared_rank(&sh.top[rank * (kPrepThreads / 32) + warp], lane) = mx;
    cluster.sync();
#pragma unroll
    for (int q = 0; q < kCluster; ++q) mx = fmaxf(mx, sh.top[q * 32 + lane]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    for (int s = tid; s < slots; s += kPrepThreads) vals[s] = index_of(s) < n ? expf(__fsub_rn(vals[s], mx)) : 0.f;
    __syncthreads();
    if (tid < 128) {
        float sum = 0.f;
#pragma unroll 8
        for (int s = tid; s < slots; s += 128) sum += vals[s];  // (adding the zeros behind the end changes nothing)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane < kCluster) *cluster.map_shared_rank(&sh.part[rank * 4 + warp], lane) = sum;
    }
    cluster.sync();
    float sum = sh.part[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float inv = __fdiv_rn(1.0f, __fadd_rn(sum, 1e-9f));
    const bool finite = inv > 0.f && inv < INFINITY;  // (the same in every CTA)
    for (int s = tid; s < slots; s += kPrepThreads) {
        const float p = __fmul_rn(vals[s], inv);
        vals[s] = p;
        const int b = bin_of(p);
        if (finite && b < kNucleusBins && index_of(s) < n) atomicAdd(&sh.hist[b >> 1], b & 1 ? 0x10000u : 1u);
    }
    cluster.sync();
    // Thread t's bins; all CTAs form the same totals in the same order.
    int total[kBinsPerThread], lower[kBinsPerThread], count = 0;  // lower: of the CTAs before this one
    float mass = 0.f;
#pragma unroll
    for (int j = 0; j < kBinsPerThread; ++j) total[j] = lower[j] = 0;
    if (tid < kBinThreads) {
        uint2 h[kCluster];
#pragma unroll
        for (int c = 0; c < kCluster; ++c) h[c] = *cluster.map_shared_rank(reinterpret_cast<uint2 *>(sh.hist) + tid, c);
#pragma unroll
        for (int c = 0; c < kCluster; ++c) {
            const int n_c[kBinsPerThread] = {(int)(h[c].x & 0xffffu), (int)(h[c].x >> 16), (int)(h[c].y & 0xffffu), (int)(h[c].y >> 16)};
#pragma unroll
            for (int j = 0; j < kBinsPerThread; ++j) {
                if (c < rank) lower[j] += n_c[j];
                total[j] += n_c[j];
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kBinsPerThread; ++j) {
        count += total[j];
        mass += (float)total[j] * __uint_as_float((kTopBin - (uint32_t)(tid * kBinsPerThread + j)) << 16);
    }
    int count_in = count;
    float mass_in = mass;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int c = __shfl_up_sync(0xffffffffu, count_in, o);
        const float m = __shfl_up_sync(0xffffffffu, mass_in, o);
        if (lane >= o) {
            count_in += c;
            mass_in += m;
        }
    }
    if (lane == 31) {
        sh.scan_n[warp] = count_in;
        sh.scan_m[warp] = mass_in;
    }
    __syncthreads();
    int w_count = sh.scan_n[lane];  // the 32 warps' totals, scanned by every warp
    float w_mass = sh.scan_m[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int c = __shfl_up_sync(0xffffffffu, w_count, o);
        const float m = __shfl_up_sync(0xffffffffu, w_mass, o);
        if (lane >= o) {
            w_count += c;
            w_mass += m;
        }
    }
    const int counted = __shfl_sync(0xffffffffu, w_count, 31), n_before = __shfl_sync(0xffffffffu, w_count, max(warp - 1, 0));
    const float m_before = __shfl_sync(0xffffffffu, w_mass, max(warp - 1, 0));
    int at = (warp ? n_before : 0) + count_in - count;
    float reached = (warp ? m_before : 0.f) + mass_in - mass;
    const float need = a.target * (1.0f + 1.0f / 4096);  // (the sequential sum may round down a little; checked by the walk)
#pragma unroll
    for (int j = 0; j < kBinsPerThread; ++j) {
        const int b = tid * kBinsPerThread + j;
        if (tid >= kBinThreads) break;
        sh.first[b] = at;
        sh.cursor[b] = at + lower[j];
        at += total[j];
        reached += (float)total[j] * __uint_as_float((kTopBin - (uint32_t)b) << 16);
        if (reached >= need) atomicMin(&sh.last_bin, b);
    }
    if (tid == kBinThreads - 1) sh.first[kNucleusBins] = at;
    __syncthreads();
    int last = sh.last_bin;
    const bool all = last == INT_MAX;  // the whole vocabulary is the list, if the bins hold it
    if (all) last = kNucleusBins - 1;
#pragma unroll
    for (int j = 0; j < kBinsPerThread; ++j)
        if (tid * kBinsPerThread + j <= last && total[j] > kMaxBin) sh.crowded = 1;
    __syncthreads();
    if (!finite || sh.crowded || (all && counted != n)) {
        if (rank == 0 && tid == 0) answer(-1);
        cluster.sync();  // the others may still read this CTA's counts
        return;
    }
    const int cands = sh.first[last + 1];
    if (cands <= kNear) {
        // The first CTA alone: candidates into their bins over its shared memory, ranked and walked there.
        for (int s = tid; s < slots; s += kPrepThreads) {
            const float p = vals[s];
            const int b = bin_of(p), i = index_of(s);
            if (b <= last && i < n)
                *cluster.map_shared_rank(&sh.cand[atomicAdd(&sh.cursor[b], 1)], 0) = ((unsigned long long)__float_as_uint(p) << 32) | (uint32_t)~i;
        }
        cluster.sync();
        if (rank != 0) return;
        for (int c = tid; c < cands; c += kPrepThreads) {
            const unsigned long long own = sh.cand[c];
            const int b = bin_of(__uint_as_float((uint32_t)(own >> 32))), w0 = sh.first[b], w1 = sh.first[b + 1];
            int larger = 0;
#pragma unroll 4
            for (int w = w0; w < w1; ++w) larger += sh.cand[w] > own;
            sh.near_p[w0 + larger] = __uint_as_float((uint32_t)(own >> 32));
            sh.near_i[w0 + larger] = (int)~(uint32_t)own;
        }
        __syncthreads();
        const int pick = pick_rank<true>(sh.near_p, cands, all, a.target, a.r, sh.pick);
        if (tid == 0) answer(pick < 0 ? -1 : sh.near_i[pick]);
        return;
    }
    for (int s = tid; s < slots; s += kPrepThreads) {
        const float p = vals[s];
        const int b = bin_of(p), i = index_of(s);
        if (b <= last && i < n) a.cand[atomicAdd(&sh.cursor[b], 1)] = ((unsigned long long)__float_as_uint(p) << 32) | (uint32_t)~i;
    }
    __threadfence();
    cluster.sync();
    // A warp ranks 32 neighbours at a time against the bins that they lie in.
    for (int p0 = (rank * (kPrepThreads / 32) + warp) * 32; p0 < cands; p0 += kCluster * kPrepThreads) {
        const int live = min(32, cands - p0);
        const unsigned long long own = lane < live ? __ldcg(a.cand + p0 + lane) : 0;
        const int b = bin_of(__uint_as_float((uint32_t)(own >> 32)));
        const int w0 = sh.first[__shfl_sync(0xffffffffu, b, 0)], w1 = sh.first[__shfl_sync(0xffffffffu, b, live - 1) + 1];
        int larger = 0;
        unsigned long long next = w0 + lane < w1 ? __ldcg(a.cand + w0 + lane) : 0;
        for (int w = w0; w < w1; w += 32) {
            sh.window[warp][lane] = next;
            __syncwarp();
            next = w + 32 + lane < w1 ? __ldcg(a.cand + w + 32 + lane) : 0;
#pragma unroll 8
            for (int j = 0; j < 32; j += 2) {
                const ulonglong2 k = *reinterpret_cast<const ulonglong2 *>(&sh.window[warp][j]);
                larger += (k.x > own) + (k.y > own);
            }
            __syncwarp();
        }
        if (lane < live) {
            a.sorted_p[w0 + larger] = __uint_as_float((uint32_t)(own >> 32));
            a.sorted_i[w0 + larger] = (int)~(uint32_t)own;
        }
    }
    __threadfence();
    cluster.sync();
    if (rank != 0) return;
    const int pick = pick_rank<false>(a.sorted_p, cands, all, a.target, a.r, sh.pick);
    if (tid == 0) answer(pick < 0 ? -1 : __ldcg(a.sorted_i + pick));
}

}  // namespace

// logits_dev[vocab] -> *token.  Waits for the token: everything enqueued before the call has run by then, the stream itself may not be idle yet (the end of
// the sampling kernel).  The answer does not release what earlier work wrote to host memory: a fence of the system in the kernel costs 1.2 us a draw (8 draws
// 223 -> 234 us), and who needs that can wait for the stream.
int sample_top_p(lumen_ctx *ctx, const float *logits_dev, size_t vocab, const lumen_sample_params &sp, int32_t *token, cudaStream_t s) {
    if (vocab == 0 || vocab > (size_t)1 << 30) return set_error(ctx, LUMEN_ERR_SHAPE, "sample: vocabulary of %zu", vocab);
    if (sp.n_recent > (size_t)kMaxRecent) return set_error(ctx, LUMEN_ERR_UNSUPPORTED, "sample: %zu recent tokens, at most %d", sp.n_recent, kMaxRecent);
    const int n = (int)vocab;
    const size_t nf = ((size_t)n + 63) & ~(size_t)63, list_bytes = 4 * nf * 4 + kMaxRecent * sizeof(int);
    // scratch kept with the context (grown when a larger vocabulary comes along): no allocation per token
    auto ensure_ws = [&](size_t bytes) -> int {
        if (ctx->sampler_ws_bytes >= bytes) return LUMEN_OK;
        LUMEN_CUDA(ctx, cudaStreamSynchronize(s));
        if (ctx->sampler_ws) cudaFree(ctx->sampler_ws);
        ctx->sampler_ws = nullptr;
        ctx->sampler_ws_bytes = 0;
        LUMEN_CUDA(ctx, cudaMalloc(&ctx->sampler_ws, bytes));
        ctx->sampler_ws_bytes = bytes;
        return LUMEN_OK;
    };
    int *token_dev = &ctx->d_status->token;  // comes back with the status
    const float target = fmaxf(fminf(fmaxf(sp.top_p, 0.f), 1.f), 1e-6f);
    // A nucleus of (nearly) everything reaches into the probabilities that the bins leave out.
    if (n <= kNucleusMaxVocab && target < 0.999f) {
        LUMEN_TRY(ensure_ws(list_bytes));
        const size_t smem = sizeof(NucleusShared) + (size_t)(n + 1023) / 1024 * 128 * sizeof(float);
        static bool attr_set[64] = {false};
        const int dev = ctx->device >= 0 && ctx->device < 64 ? ctx->device : 0;
        if (!attr_set[dev]) {
            const size_t most = sizeof(NucleusShared) + kNucleusMaxVocab / kCluster * sizeof(float);
            LUMEN_CUDA(ctx, cudaFuncSetAttribute(sample_nucleus_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
            attr_set[dev] = true;
        }
        char *ws = static_cast<char *>(ctx->sampler_ws);
        NucleusArgs a;
        a.logits = logits_dev; a.n = n; a.temperature = sp.temperature; a.penalty = sp.repetition_penalty; a.target = target; a.r = sp.uniform;
        a.cand = reinterpret_cast<unsigned long long *>(ws);
        a.sorted_p = reinterpret_cast<float *>(ws + 8 * nf); a.sorted_i = reinterpret_cast<int *>(ws + 12 * nf);
        a.status = &ctx->d_status->code;
        a.answer = ctx->h_answer; a.turn = ++ctx->answer_turn;
        a.n_recent = (int)sp.n_recent;
        for (size_t i = 0; i < sp.n_recent; ++i) a.recent[i] = sp.recent_tokens[i];
        sample_nucleus_kernel<<<kCluster, kPrepThreads, smem, s>>>(a);
        LUMEN_LAUNCHED(ctx);
        // The kernel stores its answer to pinned memory of the host, which watches the word, so that no copy and no wait for
        // the stream follow the kernel.  It spins at first, then gives way to other threads; behind a backlog of more than 20 ms, and
        // where a failure left no answer, it waits for the stream as everything else does (as the device's scheduling flags say).
        int got = -1;
        const auto asked = std::chrono::steady_clock::now();
        for (unsigned int spins = 1;; ++spins) {
            unsigned long long v = __atomic_load_n(ctx->h_answer, __ATOMIC_ACQUIRE);
            bool last = false;
            if ((spins & 63) == 0 && (unsigned int)(v >> 32) != a.turn) {
                const auto waited = std::chrono::steady_clock::now() - asked;
                if (waited > std::chrono::milliseconds(20)) {
                    LUMEN_TRY(check_device_status(ctx));
                    v = __atomic_load_n(ctx->h_answer, __ATOMIC_ACQUIRE);
                    last = true;
                } else if (waited > std::chrono::microseconds(50)) {
                    std::this_thread::yield();
                }
            }
            if ((unsigned int)(v >> 32) == a.turn) {
                got = (int)(unsigned int)v;
                break;
            }
            if (last) break;
#if defined(__x86_64__)
            __builtin_ia32_pause();
#endif
        }
        if (got >= 0) {
            *token = got;
            return LUMEN_OK;
        }
        if (got == -2) LUMEN_TRY(check_device_status(ctx));
    }
    size_t sort_bytes = 0;
    LUMEN_CUDA(ctx, cub::DeviceRadixSort::SortPairsDescending(nullptr, sort_bytes, (const float *)nullptr, (float *)nullptr, (const int *)nullptr,
                                                              (int *)nullptr, n, 0, 32, s));
    LUMEN_TRY(ensure_ws(list_bytes + ((sort_bytes + 255) & ~(size_t)255)));
    void *ws = ctx->sampler_ws;
    float *probs = static_cast<float *>(ws), *probs_sorted = probs + nf;
    int *idx = reinterpret_cast<int *>(probs_sorted + nf), *idx_sorted = idx + nf;
    int *recent_dev = idx_sorted + nf;
    void *sort_ws = recent_dev + kMaxRecent;
    if (sp.n_recent) LUMEN_CUDA(ctx, cudaMemcpyAsync(recent_dev, sp.recent_tokens, sp.n_recent * sizeof(int), cudaMemcpyHostToDevice, s));
    sample_prep_kernel<<<1, kPrepThreads, 0, s>>>(logits_dev, n, sp.temperature, sp.repetition_penalty, recent_dev, (int)sp.n_recent, probs, idx);
    LUMEN_LAUNCHED(ctx);
    LUMEN_CUDA(ctx, cub::DeviceRadixSort::SortPairsDescending(sort_ws, sort_bytes, probs, probs_sorted, idx, idx_sorted, n, 0, 32, s));
    sample_pick_kernel<<<1, kPickThreads, 0, s>>>(probs_sorted, idx_sorted, n, target, sp.uniform, token_dev);
    LUMEN_LAUNCHED(ctx);
    LUMEN_TRY(check_device_status(ctx));
    *token = ctx->h_status->token;
    return LUMEN_OK;
}

}  // namespace lumen
