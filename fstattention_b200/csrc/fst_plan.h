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

// How a call behind a shared prefix is laid out: whether a CTA has two query tiles (pair), and into how many runs
// the column tiles are cut, the runs of a query tile being a cluster of CTAs.  One CTA per SM.
// The choice minimises waves x (tiles of a run x a tile's time + a CTA's fixed time) + merging.  In tenths of a
// microsecond at D 128 (4096 prefix rows, 32 heads of 256 query rows; 3001 rows in pages of 16, 8 K/V heads): a tile 10
// for one query tile and 22 for two, but 18 for one where the tile comes in small pages (a page of 16 rows
// is a TMA box per 64 columns, and the boxes are what takes the time: two query tiles share them);
// 140 for loading the first tiles, the last tile's chain and the output; 7 for every run to be merged.
constexpr int kMaxPrefixRuns = 8;      // portable cluster size
struct PrefixPlan {
    int runs;
    bool pair;
};
inline PrefixPlan prefix_plan(int64_t Z, int64_t H, int64_t H_kv, int64_t n_q, int64_t prefix, int sms, int64_t asked = 0,
                              int64_t page = 128) {
    const int64_t kv_tiles = H / H_kv / prefix_heads_per_tile(H, H_kv, n_q) * ((n_q + 127) / 128);
    const int64_t tiles = (prefix + 127) / 128 + 2;
    const int64_t cap = std::max<int64_t>(1, std::min<int64_t>({kMaxPrefixRuns, tiles / 2, 65535 / std::max<int64_t>(Z, 1)}));
    const int64_t lo = asked > 0 ? std::min<int64_t>(asked, kMaxPrefixRuns) : 1, hi = asked > 0 ? lo : cap;
    PrefixPlan best{int(lo), false};
    int64_t best_cost = INT64_MAX;
    for (int64_t pair = 0; pair < (kv_tiles > 1 ? 2 : 1); ++pair)
        for (int64_t runs = lo; runs <= hi; ++runs) {
            const int64_t ctas = Z * H_kv * ((kv_tiles + pair) / (1 + pair)) * runs;
            const int64_t fit = runs > 4 ? sms * 7 / 8 : runs > 2 ? sms * 9 / 10 : sms;      // clusters stay within a GPC
            const int64_t waves = (ctas + fit - 1) / fit;
            const int64_t cost = waves * ((tiles + runs - 1) / runs * (pair ? 22 : page < 32 ? 18 : 10) + 140) + (runs > 1 ? 10 + 7 * runs : 0);
            if (cost < best_cost) {
                best_cost = cost;
                best = {int(runs), pair != 0};
            }
        }
    return best;
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
