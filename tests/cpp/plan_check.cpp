// Prints the plans of products and of decode attention, one per line of its input:
//   plain M K N bf16   ->  bn splits kb_per_split          (bn 0: 128 x 128 tiles of single SMs)
//   pair M K N products swiglu may_split   ->  the same
//   width M N swiglu splits   ->  columns of a tile where the plan has 256
//   attn B Hq Hkv D len   ->  parts of a batched decode step's context (0: the general kernel)
#include <cstdio>
#include <cstring>

#include "attn_plan.cuh"
#include "gemm_plan.cuh"

int main() {
    char kind[16];
    size_t m, k, n;
    while (std::scanf("%15s %zu %zu %zu", kind, &m, &k, &n) == 4) {
        int a = 0, b = 0, c = 0;
        if (!std::strcmp(kind, "width")) {
            if (std::scanf("%d", &a) != 1) return 1;
            std::printf("%d\n", lumen::pair_width(m, k, n != 0, a, 148));
            continue;
        }
        if (!std::strcmp(kind, "attn")) {
            size_t d, len;
            if (std::scanf("%zu %zu", &d, &len) != 2) return 1;
            std::printf("%d\n", lumen::attn_rows_splits(m, k, n, d, len, 148));
            continue;
        }
        lumen::GemmPairPlan p;
        if (!std::strcmp(kind, "plain")) {
            if (std::scanf("%d", &a) != 1) return 1;
            p = lumen::plan_gemm_plain(m, k, n, a != 0, 148);
        } else {
            if (std::scanf("%d %d %d", &a, &b, &c) != 3) return 1;
            p = lumen::plan_gemm_pair(m, k, n, a, b != 0, c != 0, 148);
        }
        std::printf("%d %d %d\n", p.bn, p.splits, p.kb_per_split);
    }
    return 0;
}
