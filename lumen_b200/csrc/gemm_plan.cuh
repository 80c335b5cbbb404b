// Which kernel multiplies many rows, in tiles of which width and in how many slices of K: plain arithmetic, also for programs of the host.
#pragma once

#include <algorithm>
#include <cstddef>

namespace lumen {

// Tile width, slices of K and 64-number blocks of K per slice; bn == 0: 128 x 128 tiles of single SMs (gemm_tc.cu).
struct GemmPairPlan {
    int bn = 0, splits = 1, kb_per_split = 0;
};

// Microseconds of a plain product but for what its kernels have in common: a fixed part, and for every 64 numbers of K a full wave of tiles, or a last one
// (a part of its own and one that grows with its share of the device).  Fitted to 272 sizes each (129 to 8192 rows, K 512 to 12288, 256 to
// 32000 columns; 5 % rms).  The kernel of the smallest estimate is 0.1 % slower than the fastest in the mean and 8 % at worst; pairs
// of SMs alone, whose 256-row tiles leave most of the device idle where there are few, were 10 % slower in the mean with bf16
// weights (1025 x 4096 x 4096: 81 us by single SMs, 113 by pairs; 256 x 4096 x 12288: 77 and 63).
struct GemmTileCost {
    int rows, cols, sms;
    double fixed, full, last, last_share;
};

inline GemmPairPlan plan_gemm_plain(size_t M, size_t K, size_t N, bool bf16, int num_sms) {
    static const GemmTileCost costs[2][3] = {{{128, 128, 1, 0.0, 0.78, 0.43, 0.08}, {256, 128, 2, 1.7, 0.67, 0.51, 0.03}, {256, 256, 2, 4.9, 1.05, 0.75, 0.08}},
                                             {{128, 128, 1, 0.0, 0.51, 0.34, 0.05}, {256, 128, 2, 1.6, 0.49, 0.43, 0.02}, {256, 256, 2, 4.4, 0.66, 0.53, 0.04}}};
    const size_t kb = (K + 63) / 64;
    GemmPairPlan best;
    double best_cost = 0;
    for (const GemmTileCost &c : costs[bf16]) {
        const size_t slots = (size_t)std::max(1, num_sms / c.sms), tiles = (M + c.rows - 1) / c.rows * ((N + c.cols - 1) / c.cols);
        const double share = (double)(tiles % slots) / slots;
        const double cost = c.fixed + kb * ((double)(tiles / slots) * c.full + (share > 0 ? c.last + share * c.last_share : 0));
        if (!best.kb_per_split || cost < best_cost) {
            best.bn = c.sms == 2 ? c.cols : 0;
            best.kb_per_split = (int)std::max<size_t>(kb, 1);
            best_cost = cost;
        }
    }
    return best;
}

// The same for products that pairs of SMs serve anyway: SwiGLU in the epilogue, or (may_split) a reader that adds slices of K.
// Cycles of the fullest pair of SMs: its tiles one after the other, and what is not overlapped (ring fill, last epilogue).
// A 128-wide tile takes more than half of a 256-wide one's time (its operands are 40 KB per 64 numbers of K instead of 48).
inline GemmPairPlan plan_gemm_pair(size_t M, size_t K, size_t N, int products, bool swiglu, bool may_split, int num_sms) {
    const size_t pairs = (size_t)std::max(1, num_sms / 2), kb_all = (K + 63) / 64, tm = (M + 255) / 256;
    const size_t width = swiglu ? N / 2 : N;
    GemmPairPlan best;
    double best_cost = 0;
    for (int bn : {256, 128}) {
        const size_t cols = swiglu ? bn / 2 : bn, tiles = tm * ((width + cols - 1) / cols);
        for (size_t splits = 1; splits <= (may_split ? 4 : 1); ++splits) {
            const size_t per = (kb_all + splits - 1) / splits;
            if (splits > 1 && (per < 8 || (kb_all + per - 1) / per != splits)) continue;
            const size_t waves = (tiles * splits + pairs - 1) / pairs;
            const double cost = (double)waves * per * products * (bn == 256 ? 512 : 330) + 4000 +
                                (splits > 1 ? (double)(splits + 1) * M * N * 4 / 2500 : 0);  // slices written and read again
            if (!best.bn || cost < best_cost) {
                best = GemmPairPlan{bn, (int)splits, (int)per};
                best_cost = cost;
            }
        }
    }
    return best;
}

// Columns of a tile where 256 were chosen above: 224 or 192 where the last wave of 256 would leave most pairs idle (512 x 4096 x 12288: 96 tiles for 74
// pairs, two waves; 128 tiles of 192 columns take two shorter ones).  Cycles of a tile as above: 512, and 330 for 128 columns; 224
// and 192 lie on the line between them: of 124 sizes for which this takes them (M 257 to 4096, K 1024 to 12288, N 1024 to 32000, both weight types) none was slower
// than with 256, and all but a few were 4 to 17 % faster (bf16 1777 x 5632 x 2048: 83.6, 78.1, 116.7 us with 256, 224, 192; 1280 x 12288 x 4096: 277, 250, 242).
// A prompt of four TinyLlama layers, 1777 positions, f32: 2153 -> 2047 us; of four Llama-2-7B layers, 512 positions, bf16: 1810 -> 1717.
inline int pair_width(size_t M, size_t N, bool swiglu, int splits, int num_sms) {
    const size_t pairs = (size_t)std::max(1, num_sms / 2), tm = (M + 255) / 256 * splits, width = swiglu ? N / 2 : N;
    int best = 256;
    double best_cost = 0;
    for (int bn : {256, 224, 192}) {
        const size_t cols = swiglu ? bn / 2 : bn, waves = (tm * ((width + cols - 1) / cols) + pairs - 1) / pairs;
        const double cost = (double)waves * (148 + 1.42 * bn);
        if (bn == 256 || cost < 0.97 * best_cost) {
            best = bn;
            best_cost = cost;
        }
    }
    return best;
}

}  // namespace lumen
