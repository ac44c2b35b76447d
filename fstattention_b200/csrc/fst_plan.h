// Choices that the library makes inside a call and the Python host path has to know before it (workspace
// sizes, which kernels a call launches).  Plain host arithmetic.
#pragma once

#include <algorithm>
#include <cstdint>

namespace fst {

// Query heads whose rows share one 128-row tile of the tcgen05 prefix kernel: heads of one grouped-query
// group read the same K and V, so a small tree's rows of two, four or eight of them make one tile
// (n_q <= 64, 32, 16) instead of as many tiles that are mostly padding.
inline int prefix_heads_per_tile(int64_t H, int64_t H_kv, int64_t n_q) {
    const int64_t group = H_kv > 0 ? H / H_kv : 1;
    int pack = 1;
    while (pack < 8 && group % (pack * 2) == 0 && n_q * pack * 2 <= 128) pack *= 2;
    return pack;
}

// Runs of column tiles that a call behind a shared prefix is cut into: one CTA per 128 query rows, head (or pack of
// heads), batch element and run, one CTA per SM.  The choice minimises waves x (tiles of a run + kFixed), with a
// charge for merging more than one run: loading the first tiles, merging the two softmax groups and writing the
// result take as long as some eight tiles of the steady state (0.95 us each at D 128), the merge kernel as four
// and more, and a grid of 1.2 waves takes two.
inline int prefix_runs(int64_t Z, int64_t H, int64_t H_kv, int64_t n_q, int64_t prefix, int sms) {
    const int64_t ctas = std::max<int64_t>(1, Z * (H / prefix_heads_per_tile(H, H_kv, n_q)) * ((n_q + 127) / 128));
    const int64_t tiles = (prefix + 127) / 128 + 2, cap = std::min<int64_t>({prefix / 256, 16, 65535 / std::max<int64_t>(Z, 1)});
    constexpr int64_t kFixed = 8, kMerge = 4;
    int64_t best = 1, best_cost = INT64_MAX;
    for (int64_t runs = 1; runs <= std::max<int64_t>(cap, 1); ++runs) {
        const int64_t waves = (ctas * runs + sms - 1) / sms,
                      cost = waves * ((tiles + runs - 1) / runs + kFixed) + (runs > 1 ? kMerge + runs : 0);
        if (cost < best_cost) {
            best_cost = cost;
            best = runs;
        }
    }
    return int(best);
}

// When the tcgen05 tree kernel beats the mma.sync one.  Measured on B200, fp16, six kinds of trees, from 64
// items (128 query rows of one head) up, ratios of old to new time:
//   D 128, block_m 128   1.15 - 1.46 from 256 items, up to 1.95 at 4096; 0.73 - 0.98 below 100
//   D 128, block_m 64    1.06 - 1.28 from 256 items where the ancestor lists run to several tiles (bound of
//                        four blocks), 1.05 - 1.25 from 1024 items with a bound of two; 0.93 - 1.04 with one
//   D 128, block_m 32    1.38 - 1.74 at 256 items, 0.98 - 1.09 above; 0.82 - 0.99 with long lists
//   D 64, block_m 128    1.16 - 1.32 from 288 to 1248 items, 0.95 - 1.29 above
//   D 64, block_m 64     1.08 - 1.40 from 1024 items with a bound of two blocks or more, 1.05 - 1.14 from
//                        4096 with one
//   D 64, block_m 32     1.12 - 1.33 from 4096 items; 0.53 - 0.88 with long lists
// Small grids are bound by one CTA's latency, which is longer here; with one short tile of ancestors per
// 64 rows at D 128 both kernels wait for the same HBM bytes.
inline bool tree_umma_pays(int64_t Z, int64_t H, int64_t n_q, int D, int bm, int ma) {
    const int64_t items = (n_q + 127) / 128 * H * Z;
    const int bound = ma / bm;                        // tiles of ancestors the caller allows for
    if (D == 128) {
        if (bm == 128) return items >= 200;
        if (bm == 64) return bound >= 4 ? items >= 256 : bound >= 2 && items >= 1024;
        return items >= 200 && (bound < 8 || items <= 400);
    }
    if (bm == 128) return items >= 280;
    if (bm == 64) return bound >= 2 ? items >= 1024 : items >= 3000;
    return bound < 8 && items >= 2000;
}

}  // namespace fst
