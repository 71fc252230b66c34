// Host build of the tensor-core launch plan (qwen38_metal_b200/csrc/q4_decomp.h) for CPU tests: walks every worker's
// items as the kernel does and checks that each (tile, K stage) is visited once and scratch indices stay in bounds.
#include <algorithm>
#include <vector>

#include "../qwen38_metal_b200/csrc/q4_decomp.h"

// 0: fine; otherwise the number of the rule that is broken
extern "C" int shim_gemm_plan(uint32_t m, uint32_t k, uint32_t row_tiles, uint32_t pairs) {
    Q4GemmPlan p;
    q4_gemm_plan(m, k, row_tiles, pairs, &p);
    const uint32_t ks = q4_gemm_k_stages(k);
    if (p.partial_floats > q4_gemm_most_partial_floats(pairs) || p.counters > q4_gemm_most_counters(pairs)) return 8;
    if (p.bn % 32 || p.bn < 32 || p.bn > 256 || p.accs * p.bn + 64 * p.stages > 512 || p.stages < 4) return 1;
    if (p.tiles != row_tiles * p.tiles_m || p.tiles_m * p.bn < m || (p.tiles_m - 1) * p.bn >= m) return 2;
    if (p.workers == 0 || p.workers > pairs || p.tail_workers > p.workers) return 3;
    std::vector<int> seen((size_t)p.tiles * ks, 0);
    const uint32_t done = p.full_rounds * p.workers;
    for (uint32_t w = 0; w < p.workers; ++w) {
        for (uint32_t r = 0; r < p.full_rounds; ++r) {
            const uint32_t t = w + r * p.workers;
            for (uint32_t i = 0; t < p.tiles && i < ks; ++i) ++seen[(size_t)t * ks + i];
        }
        if (p.tiles <= done || w >= p.tail_workers) continue;
        const Q4Split s{(uint64_t)(p.tiles - done) * ks, ks, p.tail_workers};
        uint32_t u = (uint32_t)q4_split_begin(s, w), cuts = 0;
        const uint32_t end = (uint32_t)q4_split_begin(s, w + 1);
        while (u < end) {
            const uint32_t tt = u / ks, k0 = u - tt * ks, n = std::min(ks - k0, end - u);
            for (uint32_t i = 0; i < n; ++i) ++seen[(size_t)(done + tt) * ks + k0 + i];
            if (n != ks) {
                uint32_t first, last;
                q4_split_contributors(s, tt, &first, &last);
                if (w < first || w > last || first == last) return 4;
                if ((uint64_t)(q4_split_slot(s, w, tt) + 1) * p.bn * 256 > p.partial_floats) return 5;
                if ((tt + 1) * 8 > p.counters || ++cuts > 2) return 6;
            }
            u += n;
        }
    }
    for (int v : seen)
        if (v != 1) return 7;
    return 0;
}
