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

// How a call behind a shared prefix is laid out: whether a CTA has two query tiles (pair), into how many runs the
// column tiles are cut, and whether the runs of a query tile are a cluster of CTAs that merges them through
// distributed shared memory, or spread over the GPU, with partial results in a workspace and a merge kernel.
// One CTA per SM.  A cluster stays within a GPC, of which there are eight with 16 SMs or more, not all of them
// with 18: 7 CTAs to a cluster use 112 SMs of 148, and few query tiles behind a long prefix are better
// spread (18 query tiles, 15100 rows: 47 us as clusters of seven in two waves, 25 spread).
// The choice minimises waves x (tiles of a run x a tile's time + a CTA's fixed time) + merging, in tenths of a
// microsecond at D 128 (4096 prefix rows, 32 heads of 256 query rows; 3001 rows in pages of 16, 8 K/V heads): a tile 8
// for one query tile and 17 for two, but 15 for one where the tile comes in small pages (a page of 16 rows
// is a TMA box per 64 columns, and the boxes are what takes the time: two query tiles share them);
// 120 for loading the first tiles, the last tile's chain and the output; 10 and 7 for every run to merge a
// cluster's, 45 and 3 for every run to spread them.
constexpr int kMaxClusterRuns = 8;     // portable cluster size
constexpr int kMaxSpreadRuns = 16;
constexpr int kGpcSms = 18;
struct PrefixPlan {
    int runs;
    bool pair, spread;
};
inline PrefixPlan prefix_plan(int64_t Z, int64_t H, int64_t H_kv, int64_t n_q, int64_t prefix, int sms, bool may_spread,
                              int64_t asked = 0, int64_t page = 128) {
    const int64_t kv_tiles = H / H_kv / prefix_heads_per_tile(H, H_kv, n_q) * ((n_q + 127) / 128);
    const int64_t tiles = (prefix + 127) / 128 + 2, per_z = 65535 / std::max<int64_t>(Z, 1);
    const int64_t most = may_spread ? per_z : std::min<int64_t>(kMaxClusterRuns, per_z);
    const int64_t lo = asked > 0 ? std::min(asked, most) : 1,
                  hi = asked > 0 ? lo : std::max<int64_t>(1, std::min<int64_t>({may_spread ? kMaxSpreadRuns : kMaxClusterRuns, tiles / 2, per_z}));
    PrefixPlan best{int(lo), false, lo > kMaxClusterRuns};
    int64_t best_cost = INT64_MAX;
    for (int spread = 0; spread < (may_spread ? 2 : 1); ++spread)
        for (int pair = 0; pair < (kv_tiles > 1 ? 2 : 1); ++pair)
            for (int64_t runs = std::max<int64_t>(lo, spread ? 2 : 1); runs <= (spread ? hi : std::min<int64_t>(hi, kMaxClusterRuns)); ++runs) {
                const int64_t ctas = Z * H_kv * ((kv_tiles + pair) / (1 + pair)) * runs;
                const int64_t gpcs = sms / kGpcSms;         // (a slice of a GPU may have less than one)
                const int64_t fit = std::max<int64_t>(1, spread || runs == 1 ? sms : runs == 2 ? gpcs * kGpcSms : gpcs * (16 / runs) * runs);
                const int64_t waves = (ctas + fit - 1) / fit, tile = pair ? 17 : page < 32 ? 15 : 8;
                const int64_t merge = runs == 1 ? 0 : spread ? 45 + 3 * runs : 10 + 7 * runs;
                const int64_t cost = waves * ((tiles + runs - 1) / runs * tile + 120) + merge;
                if (cost < best_cost) {
                    best_cost = cost;
                    best = {int(runs), pair != 0, spread != 0};
                }
            }
    return best;
}

// Whether a call behind a shared prefix goes to the tcgen05 prefix kernel (head_dim 64 or 128, block_m 32 and up) or the
// tree kernel walks the prefix.  Measured at 33 to 255 prefix rows, ratio of the tree kernel's time to the other's:
// block_m 128 (250 nodes) 0.85 - 1.09 at 33 rows, 1.02 - 1.32 at 96, 1.30 - 1.61 at 200; block_m 64 (100
// nodes) 0.74 - 0.91 up to 128, 0.98 - 1.18 at 200; block_m 32 (20 nodes) 0.45 - 0.96 up to 128, 1.00 - 1.22
// at 200, but 0.60 - 0.64 where more query tiles than SMs are filled to a quarter or less.
inline bool prefix_umma_pays(int64_t Z, int64_t H, int64_t H_kv, int64_t n_q, int64_t prefix, int64_t bm, int sms) {
    const int64_t pack = prefix_heads_per_tile(H, H_kv, n_q);
    const bool sparse = n_q * pack <= 32 && Z * H / pack > sms;
    return prefix >= (sparse ? 256 : bm >= 128 ? 96 : 192);
}

// Columns of a column tile of the TMA tree kernel, 32 or 64.  64 halve the rounds of softmax that a warp runs one after the
// other, but leave room for fewer CTAs on an SM: two instead of three (one instead of two at block_m 128, D 64; one either
// way at D 128).  So what counts is whether 32 need fewer waves, and how many gathered tiles there can be.  Us per
// call, 32 / 64 columns, by CTAs; "bound": ancestors allowed for, in blocks:
//   block_m 64, bound 1    D 128: 384 8.8 / 10.7, 512 12.9 / 12.1, 768 15.7 / 17.1, 1024 19.4 / 21.8; D 64: 384 6.1 / 7.5, 512 9.1 / 8.5, 768 10.5 / 12.0
//   block_m 64, bound 2    D 128: 384 11.8 / 13.1, 512 18.1 / 14.5, 1024 28.1 / 26.2; bound 5: 384 19.9 / 19.0, 512 27.5 / 23.7
//   block_m 32, 64 slots   D 128: 128 3.9 / 5.2, 512 6.3 / 10.1, 1024 11.1 / 18.9; D 64: 128 2.9 / 3.8, 512 4.6 / 4.5, 1024 7.8 / 8.6
//                          a few CTAs more than fit at once, 304: deep trees D 128 11.1 / 9.5, D 64 8.2 / 6.8, scored ones 9.6 / 9.6,
//                          6.9 / 6.9; 320: deep 11.3 / 12.2, 8.2 / 8.7
//   block_m 128, bound 1   D 64: 128 7.1 / 5.3, 256 8.8 / 10.1, 384 14.4 / 14.5, 512 15.6 / 18.8; D 128: 192 14.7 / 13.4
//   block_m 128, bound 2   D 64: 192 10.3 / 11.4, 256 10.8 / 12.3; bound 3: 192 18.1 / 13.2
// Above eight CTAs per SM 32 win at block_m 64 and 128 (64 batched trees of 256 nodes: 104 / 142).  Longer lists at block_m 32:
//   D 128, 128 slots       scored trees 128 4.0 / 5.3, 256 5.6 / 5.5, 512 6.6 / 10.3; deep ones 5.5 / 5.7, 7.2 / 5.8, 8.2 / 11.1
//   D 64, 128 slots        scored 128 3.2 / 3.8, 512 4.8 / 4.6, 1024 8.5 / 8.8, 1536 11.9 / 12.5, 4096 26.5 / 29.4; deep 4.1 / 4.1, 6.0 / 5.0,
//                          10.7 / 9.6, 15.1 / 13.5, 34.1 / 31.7: they part above eight CTAs per SM, where scored (and Medusa)
//                          trees lose 5 to 20 % by 64 columns and deep ones 3 to 12 % by 32
//   D 64, 320 slots        window trees 512 9.9 / 8.7, 1024 17.7 / 14.8, 2048 30.5 / 28.5, 8192 101 / 100
inline int tma_tile_cols(int64_t ctas, int D, int bm, int ma, int sms) {
    if (bm == 32) {
        if (D == 128) return ma > 64 && ctas <= 2LL * sms ? 64 : 32;
        if (ma <= 64) return ctas > 3LL * sms && ctas <= 4LL * sms ? 64 : 32;     // two waves either way
        return ma > 256 || ctas <= 8LL * sms ? 64 : 32;
    }
    if (ctas > 8LL * sms) return 32;
    if (bm == 128 && D == 128) return 64;
    const int64_t fit = (bm == 64 ? 2LL : 1LL) * sms;     // CTAs at once with 64 columns; with 32 one more per SM
    if (ctas <= fit + (ma > bm ? sms / 16 : 0)) return 64;
    if (ctas <= fit + sms) return ma <= 2 * bm ? 32 : 64;
    return ma > bm || (ctas + fit - 1) / fit <= (ctas + fit + sms - 1) / (fit + sms) ? 64 : 32;
}

// When the tcgen05 tree kernel beats the mma.sync one.  Measured on B200, fp16, six kinds of trees of 64 to 4096 nodes, 30 to 4130
// items (128 query rows of one head), in graphs of calls; ratios of the mma.sync kernel's time (with the better of its
// tiles) to the other's; "bound" is the ancestor bound in blocks:
//   D 128, block_m 128   0.69 - 1.15 up to one item per SM, 1.01 - 1.29 at 150 to 170, 1.06 - 1.67 up to 420, 1.32 - 2.28 above
//   D 128, block_m 64    64 slots: 0.55 - 1.02 up to 900, 1.02 - 1.15 above, but 1.01 in a program whose inputs come from HBM (64 x 256
//                        nodes 114.6 / 113.4 us), and errors against 64 bits of 1.003 of the other kernel's: not there.
//                        96 slots: 0.84 - 1.02 up to 420, 0.97 - 1.08 at 500, 1.06 - 1.21 above.  Bound 2 and 3: 0.56 - 1.08 up to 224; deep trees
//                        1.07 at 250 to 310, others 0.83 - 1.00; 0.86 - 1.16 up to 420, 0.93 - 1.21 at 500, 0.98 - 1.43 above.  Bound 4 and
//                        up: 0.63 - 1.11 up to 224; with 700 nodes and more 1.02 - 1.18 at 250 to 310 (in a decode step of 1024 window
//                        nodes, 256 items, 1.00 - 1.04 on five GPUs), 0.98 - 1.22 up to 420 (scored trees 0.90 at 312), 1.01 - 1.44 above; with fewer
//                        0.86 - 1.17 up to 420, 1.00 - 1.22 at 500, 1.05 - 1.39 above
//   D 128, block_m 32    64 slots: 0.53 - 0.99 up to 530, 1.00 - 1.03 up to 900, 1.09 - 1.23 above; bound 4 to 7: 0.54 - 1.03 up to 420, 0.88 - 1.07 at 500,
//                        0.96 - 1.10 up to 900, 0.98 - 1.27 above (256-node deep trees 0.93 - 1.04); 0.62 - 1.01 with 320 slots.  64 nodes
//                        0.55 - 0.75 at any size, 300 nodes 0.54 - 1.00 up to 900 and 1.05 - 1.13 above
//   D 64, block_m 128    bound 1: 0.58 - 1.04 up to 310, 1.04 - 1.47 above; bound 2: 0.69 - 0.80 up to one per SM, 0.96 - 1.05 up to 310, 1.08 - 1.39
//                        above; bound 3: 0.85 - 1.00 up to 170, 1.03 - 1.67 above
//   D 64, block_m 64     64 slots: 0.54 - 1.01 up to 900, 1.07 - 1.21 above (64 nodes 0.52 - 0.91); bound 2 and 3: 0.54 - 0.96 up to 310, 0.84 - 1.06 up to
//                        420, 0.98 - 1.18 at 500 and 1.03 - 1.47 above (Medusa trees 0.92 - 1.00, 0.94 at 640, 1.02 - 1.18); bound 4 and up:
//                        0.55 - 1.08 up to 420, 0.92 - 1.20 at 500, 1.04 - 1.46 above (512 window nodes 0.94 - 0.96 from 1200 on: four row tiles
//                        to a head in a grid of 148, so that the longest lists fall to the same CTAs); 300 nodes in short lists
//                        0.54 - 0.94 up to 900 and 1.01 - 1.09 above, in long ones 0.58 - 0.97 up to 700, 1.04 - 1.18 above
//   D 64, block_m 32     64 slots: 0.47 - 0.99 up to 420, 0.93 - 1.07 at 500, 1.07 - 1.31 above; bound 4 to 7: scored and Medusa trees 0.49 - 1.05 up to 420,
//                        0.96 - 1.12 at 500, 1.12 - 1.34 above, deep ones 0.81 - 0.92 at 250 to 900 and 0.92 - 1.00 above (the line is where
//                        they lose next to nothing against the columns that the others want); 0.53 - 1.03 with a bound of 8 and
//                        up (scored trees 1.07 - 1.25 from 500).  64 nodes 0.45 - 0.70 at any size, 300 nodes 0.50 - 1.02 up to
//                        900 and 1.09 - 1.16 above
// Rows of an item for which there is no node cost as much as the others here and nothing there.
// Small grids are bound by one CTA's latency, which is longer here.
inline bool tree_umma_pays(int64_t Z, int64_t H, int64_t n_q, int D, int bm, int ma) {
    const int64_t slots = (n_q + 127) / 128 * 128, items = slots / 128 * H * Z;
    const int bound = ma / bm;                        // tiles of ancestors the caller allows for
    if (bm == 128) return items >= (D == 128 || bound == 2 ? 150 : bound > 2 ? 166 : 300);
    if (D == 128 && bm == 64) return ma > 64 && items >= (bound < 2 ? 650 : bound < 4 || n_q >= 700 ? 250 : 600);
    if (4 * n_q < 3 * slots || (bm == 32 && bound >= 8)) return false;
    if (5 * n_q < 4 * slots) return items >= (bm == 64 && bound >= 4 ? 700 : 1000);
    if (D == 128) return items >= (bound >= 4 ? 500 : 600);
    if (bm == 64) return items >= (bound >= 4 ? (n_q >= 700 ? 500 : 600) : bound >= 2 ? 450 : 1000);
    return items >= (bound < 4 ? 700 : n_q >= 700 ? 500 : 1000);
}

}  // namespace fst
