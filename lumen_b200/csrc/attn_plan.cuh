// Which kernel attends in a batched decode step, and in how many parts of the context: plain arithmetic, also for programs of the host.
#pragma once

#include <cstddef>

namespace lumen {

// Parts of the context for attn_rows.cu; 0: the general kernel (attention.cu).
// Up to eight parts: as many as leave every SM two CTAs and a part 96 rows (a tile of rows per warp takes about 3 us; a step of
// four TinyLlama layers, 16 sequences at 1900 positions: 383 us with eight parts, 479 with four, 402 with the general kernel and its merge).
// Longer contexts of few sequences want more parts than a cluster has: they take the general kernel.
// So do long contexts of heads of 64 in groups of four or eight, where the general kernel has tiles of 32 rows in three stages per warp and this one 16 rows in
// one.  Steps of four layers of width 2048 at 500 / 1000 / 2000 / 4096 positions, here and there: 64 sequences of 4 KV heads, groups of 8:
// 318 / 412 / 595 / 927 us and 344 / 406 / 516 / 770; 64 of 8 KV heads, groups of 4: 344 / 490 / 710 / 1163 and 398 / 498 / 661 / 1025; 8 of 4 KV heads, groups
// of 8: 169 / 192 / 238 / 326 and 215 / 227 / 246 / 272.
// Heads of 128 gain up to 4096 positions (64 sequences of 8 KV heads: 478 / 654 / 1012 / 1742 us and 588 / 824 / 1219 / 2047).
inline int attn_rows_splits(size_t B, size_t Hq, size_t Hkv, size_t D, size_t len, int num_sms) {
    if ((D != 64 && D != 128) || Hkv == 0 || Hq % Hkv) return 0;
    const size_t G = Hq / Hkv, base = B * Hkv, sms = (size_t)num_sms;
    if (G != 1 && G != 2 && G != 4 && G != 8) return 0;
    if (base * 8 < sms && len > 4096) return 0;
    if (D == 64 && G >= 4 && base * 8 >= sms) {
        const bool eight = base * 4 < 2 * sms;  // (eight parts share a context)
        if (len > (size_t)(G == 8 ? (eight ? 2600 : 1200) : (eight ? 3500 : 1750))) return 0;
    }
    int n = 1;
    while (n < 8 && base * n < 2 * sms && len >= 96 * (size_t)n) n *= 2;
    return n;
}

}  // namespace lumen
