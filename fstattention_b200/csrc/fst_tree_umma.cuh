// Tree attention on the 5th-generation tensor cores (tcgen05 + TMEM): persistent, one CTA per SM.
//
// Same mathematics as attn_tma_kernel (reference fstattention.py:21-151, no shared prefix); what
// differs is who does the work.  A block is 64 rows of at most some 130 columns, so with mma.sync
// a warp's sixteen rows are one chain of some 1500 dependent instructions, and twelve warps - all that fit an
// SM's registers - cannot interleave enough of them: large grids ran at half the copy bandwidth
// with every pipe half idle.  Here the products are a handful of tcgen05.mma issued by one thread,
// a row's scores come back to one thread (no shuffles), and loads run tiles ahead of everything.
//
//   item     128 query rows of one head: 128 / BM consecutive blocks of the tree
//   tile     128 columns of K and V rows, BM columns for each of the item's blocks.  Tile 0 is
//            the item's own rows (contiguous, TMA boxes); tile t > 0 holds ancestor slots
//            [(t-1) BM, t BM) of every block (gathered row by row; padding slots are zeros).  The last
//            tile is narrow - BM / 2 columns for each block - when the lists end in its first half.
//   round    the tiles whose scores are computed at once (see Round)
//   S = Q K^T     M 128, N 128 (64), both operands in shared memory (128-byte swizzle)
//   softmax       thread r of a group owns row r and looks only at its block's columns; 32-column
//                 words in which no row of its warp has a mask bit are not even read; P goes back
//                 over S in tensor memory
//   O += P V      A = P from tensor memory, V from shared memory (MN-major); 16-column steps
//                 beyond every block's list are left out, and a step adds to the rows that have a column in it
//                 and to no others (O starts as zeros): zero times a V that is not finite would be NaN in rows
//                 that do not attend to it, 128 of them.  Nor need P then be cleared where a warp has no column
//
// Sixteen warps.  Warps 0-3 and 4-7 are two softmax groups: group g takes the CTA's items g, g + 2, ... and
// owns an S/P buffer and an accumulator (TMEM: 128 or 192 columns, and D), so that one group's latencies hide
// behind the other's work (one group with a tile of lookahead in the products was bound by its own
// instruction stream: 7000 cycles per 128 rows at D 64).  One lane of warp 8 + g issues the products of
// group g.  Warp 10 loads Q and the own tiles, warps 11-14 gather (cp.async, 16 bytes a lane; TMA's gather4
// fills the same layout but takes the engine about 100 cycles for its four rows, 6500 per item of 64
// trees against the 5700 that its HBM bytes take), warp 15 stores O.  All tiles share one pool of 128-row
// buffers (seven at D 128): warp 10 hands them out in item order - K, Q, a gathered tile, V, the others (a narrow
// tile's K and V in one buffer) - as they come free, in whatever order that is, so that the next items'
// 96 KB are on their way while these are used up; O leaves through its item's Q buffer.
//
// Five roles share an instruction cache: waits loop out of line and long loops are kept rolled, but for the
// issue of products.  At 96 KB of code instead of fifty the 64-tree forest took 199 us instead of 125.
//
// All hand-offs are mbarriers with bounded waits; whoever times out records FST_DEV_TIMEOUT and stops.
// A parity wait can tell a phase only from its neighbours, so no waiter may be two phases off: every group's
// loads have positions of their own, with a "full" barrier for each of the last sixteen, and at most a
// pool of tiles (14) is outstanding; one thread consumes a group's positions in order.
//
// The exponent's reference point is the row's largest score so far; when a later tile has a larger one, O is
// rescaled in tensor memory.  So the weight that dominates a row is exactly 1 and loses nothing when P is
// rounded to 16 bits, as in attn_tma_kernel: errors against 64 bits over six kinds of trees are 1.000 of that
// kernel's (0.991 - 1.008; 1.002 - 1.006 where the scores of both tiles come at once).  Moving it only past 2^8 saved
// 2 to 3 % of the time and cost 9 to 20 % in error.
// When S(t) has landed every earlier product of the group has too (one thread issues them in order), so
// the group may rescale O without asking; where S(1) comes with S(0) it asks bar_m.
//
// Measured against attn_tma_kernel (us per call, fp16): 4096-node deep tree, 64 heads, D 128 84 -> 60 (4.5 TB/s
// over Q, K, V and O); 64 x 300-node dynamic trees, D 128, block_m 128 381 -> 146; 16 x 1000-node deep
// trees, D 64 120 -> 82; the create_tree forest of 65532 nodes, 4 x 48 heads, D 64, block_m 128 2190 -> 1360.
// What bounds it is the chain of a group's round - product, softmax, (rescale,) product - and at D 128 the pool: a 96 KB item
// in use, one on its way, and the last one's O.  Items of one tile run at HBM's rate (D 128: 83 us where 64 trees of
// 256 nodes take 101; D 64: 1165 where the forest takes 1360), so the ancestors are what the rest pays for.
//
// The scores of both tiles of an item at once (Round::BOTH), for bounds of up to 64 at D 64 and block_m 128: their columns
// fit beside one another, so the second tile's are there when the softmax of the first is done, and the first's product
// with V runs under the second's exponentials: forest of 65532 nodes 1745 -> 1360 us, of 8188 218 -> 175 (1400 and 179 with O
// rescaled ahead of the exponentials, as in the other rounds).  The roundings are those of the tiles one by one.  One
// softmax over both (1335 us) rounded the own tile's largest weight too, 1.2 to 2.8 % more error; with the second tile's
// output in columns of its own, scaled when O is read, it had the error of now and the speed, but not the bits.  One
// softmax lost elsewhere: longer lists (dynamic trees of 1024 nodes, D 128 54.4 / 56.0; further rounds of 64 or 128 slots
// 24.4 / 27.1 and 68 / 79), block_m 64 at D 64 (140 / 155), block_m 32 (104 / 118).
// tree_umma_pays (fst_plan.h) has the line between the two kernels.
#pragma once

#include <algorithm>

#include "fst_umma.cuh"

namespace fst {

namespace tree_umma {

constexpr int ROWS = 128;              // query rows per item, K/V rows per tile
constexpr int GATHER = 4;              // gathering warps
constexpr int THREADS = (12 + GATHER) * 32;
constexpr int FULL_COUNT = GATHER * 32;   // arrivals that complete a K or V tile: the gathering lanes', or one for all of them
constexpr int POSITIONS = 16;          // load positions of a group with a barrier of their own
constexpr int TURNS = 16;              // hand-overs to the gathering warps that may be outstanding
constexpr int ITEMS = 16;              // items whose Q or O may be outstanding (the pool holds fewer)

template <int D>
struct Geo {
    static constexpr int TILE = ROWS * D * 2;
    static constexpr int POOL = D == 128 ? 7 : 14;            // tile buffers
    static constexpr int COLS = 256 - D;                      // columns of S: 2 x (COLS + D) are all of tensor memory
    static constexpr int OFF_BAR = POOL * TILE;
    static constexpr int N_BAR = 2 * POSITIONS + POOL + TURNS + 2 * ITEMS + 8;
    static constexpr int OFF_INFO = OFF_BAR + (N_BAR + 1) / 2 * 16;   // ItemInfo per item in flight
    static constexpr int OFF_ROWS = OFF_INFO + ITEMS * 32;            // [group][16 columns of S][warp] rows with a column there
    static constexpr int OFF_WHERE = OFF_ROWS + 2 * COLS;             // which buffer a position's tile is in; then the TMEM address
    static constexpr int SMEM_BYTES = OFF_WHERE + 2 * POSITIONS + 16 + 1024;  // + slack to align the base to 1 KB
    static_assert(SMEM_BYTES <= 227 * 1024, "one CTA's shared memory");
};

// What one round of scores takes.  TILE: a column tile.  BOTH: the two tiles of an item whose lists end in the first half of a
// gathered tile (D 64, block_m 128: 128 + 64 of S's 192 columns).
enum class Round { TILE, BOTH };

// what the loading warp tells a group and its issuing thread about their next item
struct ItemInfo {
    int tiles;                         // column tiles
    int at;                            // position of the first K tile in the group's load sequence
    int count[4];                      // external ancestors of the item's blocks
    int narrow;                        // the last tile is a narrow one
    int q_buf;                         // buffer of Q, later of O
};

// 16-column steps of gathered tile t that hold slots of some block (bit ks: rows 16 ks .. of the buffer); seg: slots per block
template <int BM>
__device__ __forceinline__ uint32_t live_steps(int t, int seg, const int (&count)[ROWS / BM]) {
    uint32_t steps = 0;
#pragma unroll
    for (int s = 0; s < ROWS / BM; ++s) {
        const int left = min(count[s] - (t - 1) * BM, seg), n = left > 0 ? (left + 15) >> 4 : 0;
        steps |= ((1u << n) - 1u) << (s * seg >> 4);
    }
    return steps;
}

// column tiles of an item whose longest ancestor list has `longest` entries, and whether the last is narrow
template <int BM>
__device__ __forceinline__ int tiles_of(int longest, bool *narrow) {
    const int tiles = 1 + (longest + BM - 1) / BM;
    *narrow = BM > 32 && tiles > 1 && longest - (tiles - 2) * BM <= BM / 2;
    return tiles;
}

__device__ __forceinline__ void arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// arrives when the calling thread's cp.async copies so far have landed
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}
// what cp.async has written, for the tensor core to read through the async proxy
__device__ __forceinline__ void fence_copied() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void arrive_n(uint32_t bar, int n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(n) : "memory");
}

}  // namespace tree_umma

// Arguments beyond AttnArgs: the grid's items.
struct TreeUmmaArgs {
    int n_items, row_tiles;            // row_tiles: items per head
    int heads_first;                   // item order: heads fastest and the last rows first
};

template <typename T, int D, int BM, tree_umma::Round ROUND>
__global__ void __launch_bounds__(tree_umma::THREADS, 1)
tree_umma_kernel(const AttnArgs a, const TreeUmmaArgs ta, const __grid_constant__ CUtensorMap tm_q,
                 const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                 const __grid_constant__ CUtensorMap tm_o) {
    using namespace tree_umma;
    using namespace umma;
    using MT = MmaTraits<T>;
    using G = Geo<D>;
    constexpr bool BF16 = !std::is_same<T, __half>::value;
    constexpr int DH = D / 64, TILE = G::TILE, POOL = G::POOL;
    constexpr bool BOTH = ROUND == Round::BOTH;
    static_assert(!BOTH || (BM == 128 && D == 64), "room in tensor memory for the columns of both tiles");
    constexpr int SUB = ROWS / BM;                        // blocks per item
    constexpr int NW = BM / 32;                           // mask words per row and tile
    constexpr int EW = BOTH ? 2 : NW;                     // of them in a gathered tile

    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    extern __shared__ unsigned char smem_raw[];
    const uint32_t s_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *smem = smem_raw + (s_base - smem_u32(smem_raw));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar_full = s_base + G::OFF_BAR, bar_empty = bar_full + 2 * POSITIONS * 8, bar_go = bar_empty + POOL * 8,
                   bar_q = bar_go + TURNS * 8, bar_ob = bar_q + ITEMS * 8, bar_s = bar_ob + ITEMS * 8, bar_p = bar_s + 16, bar_o = bar_s + 32, bar_m = bar_s + 48;
    int4 *info = reinterpret_cast<int4 *>(smem + G::OFF_INFO);        // ItemInfo, read and written in two halves
    volatile unsigned char *buf_at = smem + G::OFF_WHERE;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + G::OFF_WHERE + 2 * POSITIONS);

    if (warp == 10 && lane == 0) {
        for (int i = 0; i < 2 * POSITIONS; ++i) mbar_init(bar_full + i * 8, FULL_COUNT);
        for (int i = 0; i < POOL + TURNS + ITEMS; ++i) mbar_init(bar_empty + i * 8, 1);
        for (int i = 0; i < ITEMS; ++i) mbar_init(bar_ob + i * 8, ROWS);
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_s + i * 8, 1);
            mbar_init(bar_p + i * 8, ROWS);
            mbar_init(bar_o + i * 8, 1);
            mbar_init(bar_m + i * 8, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 9) tmem_alloc_all(smem_u32(tmem_slot));
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;                // S/P of group g at g * COLS, O at 2 * COLS + g * D

    const PackedLayout L = packed_layout(a.nb, BM, a.ma);
    const int maw = L.maw, stride = gridDim.x;
    // Item numbers in mixed radix: row tiles, heads, batch (or heads, row tiles from the last down, batch), so
    // that a role's step to its CTA's next item is three additions with carries.
    struct Where {
        int d0, d1, z;
    };
    const bool hf_order = ta.heads_first != 0;
    const int r0 = hf_order ? a.H : ta.row_tiles, r1 = hf_order ? ta.row_tiles : a.H;
    auto digits = [&](int v) -> Where {
        Where w;
        const int rest = v / r0;
        w.d0 = v - rest * r0;
        w.z = rest / r1;
        w.d1 = rest - w.z * r1;
        return w;
    };
    auto tile_of = [&](const Where &w) { return hf_order ? ta.row_tiles - 1 - w.d1 : w.d0; };
    auto head_of = [&](const Where &w) { return hf_order ? w.d0 : w.d1; };
    auto plus = [&](Where w, const Where &step) -> Where {
        w.d0 += step.d0;
        w.d1 += step.d1;
        w.z += step.z;
        if (w.d0 >= r0) { w.d0 -= r0; ++w.d1; }
        if (w.d1 >= r1) { w.d1 -= r1; ++w.z; }
        return w;
    };
    // one after another, or - the roles of a group - every other one
    const bool alternate = warp < 10;
    const Where first = digits(blockIdx.x + (alternate && (warp < 8 ? warp >> 2 : warp - 8) ? stride : 0)),
                step = digits(alternate ? 2 * stride : stride);
    if (!a.meta_stable) asm volatile("griddepcontrol.wait;\n" ::: "memory");

    // external ancestors of the item's block `lane`
    auto count_of = [&](const Where &w) -> int {
        if (w.z >= a.Z || lane >= SUB) return 0;
        const int b = tile_of(w) * SUB + lane;
        if (b >= a.nb) return 0;
        const unsigned char *blob = a.packed + size_t(w.z) * a.meta_stride;
        return min(max(__ldg(reinterpret_cast<const int32_t *>(blob + L.off_count) + b), 0), a.ma);
    };
    auto spread = [&](int cnt_lane, int (&cnt)[SUB]) -> int {
        int longest = 0;
#pragma unroll
        for (int s = 0; s < SUB; ++s) {
            cnt[s] = __shfl_sync(0xffffffffu, cnt_lane, s);
            longest = max(longest, cnt[s]);
        }
        return longest;
    };
    // positions of group g: their barrier, and which buffer the tile is in
    auto full_of = [&](int g, int at) { return bar_full + (g * POSITIONS + at % POSITIONS) * 8; };
    auto buf_of = [&](int g, int at) -> volatile unsigned char & { return buf_at[g * POSITIONS + at % POSITIONS]; };
    auto full_parity = [&](int at) { return uint32_t(at / POSITIONS) & 1u; };
    auto q_of = [&](int n) { return bar_q + (n % ITEMS) * 8; };
    auto q_parity = [&](int n) { return uint32_t(n / ITEMS) & 1u; };

    if (warp == 10) {
        // ================================ loads: Q and own tiles ================================
        Where w = first;
        int cnt_lane = count_of(w);
        if (a.meta_stable) asm volatile("griddepcontrol.wait;\n" ::: "memory");
        int ahead[2] = {0, 0}, n = 0, turn = 0;           // the groups' positions, item number, hand-overs so far
        bool alive = true, used = false;
        uint32_t parity = 0;                              // lane b: has buffer b been handed out, parity of its next release
        auto take = [&]() -> int {                        // a free buffer; every lane looks at its own
            unsigned long long since = 0;
#pragma unroll 1
            for (int spin = 1; alive; ++spin) {
                const uint32_t ready = __ballot_sync(0xffffffffu, lane < POOL && (!used || over(bar_empty + lane * 8, parity)));
                if (ready != 0u) {
                    const int b = __ffs(ready) - 1;
                    if (lane == b) {
                        parity ^= uint32_t(used);
                        used = true;
                    }
                    return b;
                }
                __nanosleep(32);                          // leave the issue slots to the others
                if ((spin & 255) == 0) {                  // as long as any other wait
                    const unsigned long long now = global_ns();
                    if (since == 0) since = now;
                    else if (now - since > 50000000ull) {
                        if (lane == 0) report(a.status, FST_DEV_TIMEOUT, n, turn);
                        alive = false;
                    }
                }
                alive = __all_sync(0xffffffffu, alive);
            }
            return 0;
        };
#pragma unroll 1
        for (int item = blockIdx.x; item < ta.n_items && alive; item += stride, ++n) {
            const Where next = plus(w, step);
            const int p = tile_of(w), h = head_of(w), hk = h / a.kv_group;
            int cnt[SUB];
            bool narrow;
            const int tiles = tiles_of<BM>(spread(cnt_lane, cnt), &narrow);
            cnt_lane = count_of(next);                    // one item ahead
            const int g = n & 1, pos = g ? ahead[1] : ahead[0];
            const int end = pos + 2 * tiles - int(narrow);    // positions: two for a tile, one where K and V share a buffer
            // Own K, Q, the first gathered tile, own V, the other gathered ones: buffers come free one by one, some 1000
            // cycles apart where the pool is what bounds the kernel, the first product needs Q and the first gathered tile
            // takes longest to come (with V second and Q third: 64 x 256 nodes D 128 115.8 -> 106.5 us, block_m 128 103.6 ->
            // 99.5, block_m 32 104.5 -> 92.7, 4096-node deep tree 63.0 -> 58.0).  BOTH keeps Q last: its pool has room,
            // and this order took 1485 -> 1500 us.
            const int gathered = end - pos - 2, q_at = BOTH ? 2 : 1, v_at = BOTH ? 1 : 2 + min(gathered, narrow && tiles == 2 ? 1 : 2);
            int at = pos + 2;
#pragma unroll 1
            for (int i = 0; i < 3 + gathered; ++i) {
                const int b = take();
                if (!alive) break;
                if (i == 0 || i == q_at || i == v_at) {
                    if (elect_one()) {
                        const bool q = i == q_at;
                        const int own = i == 0 ? pos : pos + 1;
                        const uint32_t bar = q ? q_of(n) : full_of(g, own);
                        if (!q) {
                            buf_of(g, own) = (unsigned char)b;
                            arrive_n(bar, FULL_COUNT - 1);
                        } else {
                            info[(n % ITEMS) * 2] = make_int4(tiles, pos, narrow, b);
                            info[(n % ITEMS) * 2 + 1] =
                                make_int4(cnt[0], SUB > 1 ? cnt[1 % SUB] : 0, SUB > 2 ? cnt[2 % SUB] : 0, SUB > 2 ? cnt[3 % SUB] : 0);
                        }
                        mbar_arrive_expect_tx(bar, TILE);
                        const CUtensorMap *map = q ? &tm_q : i == 0 ? &tm_k : &tm_v;
                        const int row = (q ? 0 : a.prefix) + p * ROWS, head = q ? h : hk;
#pragma unroll
                        for (int hf = 0; hf < DH; ++hf)
                            tma_load_4d(s_base + b * TILE + hf * HALF, map, hf * 64, row, head, w.z, bar);
                    }
                } else {
                    if (elect_one()) {
                        buf_of(g, at) = (unsigned char)b;
                        arrive(bar_go + (turn % TURNS) * 8);
                    }
                    ++at;
                    ++turn;
                }
                __syncwarp();
            }
            (g ? ahead[1] : ahead[0]) = end;
            w = next;
        }
    } else if (warp >= 11 && warp < 11 + GATHER) {
        // ================================ gathered tiles ================================
        // A tile's live 16-row steps are dealt to the warps in turn; a warp gets at most two, the rows of the
        // first in lanes 0-15 and those of the second in lanes 16-31.
        const int gw = warp - 11;
        int cnt[SUB] = {};
        Where w{}, next = first;
        int t = 0, tiles = 0, pos = 0, n = -1, other_pos = 0;   // pos: of item n's group, other_pos: of the other
        bool narrow = false;
        int cnt_lane = count_of(next);
        struct Tile {
            int g, pos, z, hk, row_a, row_b, node, b, slot;  // row_a, row_b: first tile row of my steps, -1: none
            bool one;                                     // K and V share a buffer
        };
        auto advance = [&](Tile &x) -> bool {             // the next gathered tile of my CTA
            while (++t >= tiles) {
                w = next;
                if (w.z >= a.Z) return false;
                ++n;
                const int swap = pos;
                pos = other_pos;
                other_pos = swap;
                next = plus(w, step);
                const int longest = spread(cnt_lane, cnt);
                cnt_lane = count_of(next);
                tiles = tiles_of<BM>(longest, &narrow);
                pos += 2;                                 // the own tile's slots
                t = 0;
            }
            x.one = narrow && t + 1 == tiles;
            const int seg = x.one ? BM / 2 : BM;
            uint32_t steps = live_steps<BM>(t, seg, cnt);
            x.row_a = x.row_b = -1;
            for (int i = 0; steps != 0; ++i) {
                const int row = (__ffs(steps) - 1) * 16;
                steps &= steps - 1;
                if (i == gw) x.row_a = row;
                if (i == gw + GATHER) x.row_b = row;
            }
            const int mine = lane < 16 ? x.row_a : x.row_b;
            x.node = -1;
            x.b = x.slot = 0;
            if (mine >= 0) {
                const int s = mine / seg;
                x.b = tile_of(w) * SUB + s;
                x.slot = (t - 1) * BM + mine - s * seg + (lane & 15);
                int c = 0;
#pragma unroll
                for (int i = 0; i < SUB; ++i)
                    if (i == s) c = cnt[i];
                if (x.slot < c)
                    x.node = __ldg(reinterpret_cast<const int32_t *>(a.packed + size_t(w.z) * a.meta_stride + L.off_idx) +
                                   size_t(x.b) * a.ma + x.slot);
            }
            x.z = w.z;
            x.hk = head_of(w) / a.kv_group;
            x.g = n & 1;
            x.pos = pos;
            pos += x.one ? 1 : 2;
            return true;
        };
        Tile cur{}, nxt{};
        if (a.meta_stable) asm volatile("griddepcontrol.wait;\n" ::: "memory");
        constexpr int CH = D / 8, RPP = 32 / CH;          // 16-byte chunks per row, rows per pass of a warp
        const int lr = lane / CH, lc = lane % CH;
        int turn = 0;                                     // tiles handed to us so far
        bool alive = true, have = false;
#pragma unroll 1
        for (bool more = true; more || have;) {           // index lists are fetched one tile ahead
            more = more && advance(nxt);
            const bool now = have;
            have = more;
            if (!now) {
                cur = nxt;
                continue;
            }
            int node = cur.node;
            if (node >= a.n_q) report(a.status, FST_DEV_INDEX_RANGE, cur.b, cur.slot);
            if (unsigned(node) >= unsigned(a.n_q)) node = -1;         // padding: zeros
            const T *kp = static_cast<const T *>(a.k) + cur.z * a.ks_z + cur.hk * a.ks_h + a.prefix * a.ks_n + lc * 8;
            const T *vp = static_cast<const T *>(a.v) + cur.z * a.vs_z + cur.hk * a.vs_h + a.prefix * a.vs_n + lc * 8;
            const int half = cur.one ? HALF / 2 : HALF;
            auto claim = [&](int at) {
                const uint32_t bar = bar_go + (turn % TURNS) * 8, parity = (turn / TURNS) & 1;
                ++turn;
                alive = __all_sync(0xffffffffu, wait(bar, parity, a.status, at));
            };
#pragma unroll 1
            for (int kv = 0; kv < 2 && alive; ++kv) {
                const int at = cur.pos + (cur.one ? 0 : kv);
                if (kv == 0 || !cur.one) claim(at);
                if (!alive) break;
                const uint32_t d0 = s_base + buf_of(cur.g, at) * TILE + (kv && cur.one ? TILE / 2 : 0) + (lc >> 3) * half;
                const T *src = kv ? vp : kp;
                const int64_t row_stride = kv ? a.vs_n : a.ks_n;
#pragma unroll 1
                for (int st = 0; st < 2; ++st) {
                    const int row0 = st ? cur.row_b : cur.row_a;
                    if (row0 < 0) break;
#pragma unroll 2
                    for (int i = 0; i < 16 / RPP; ++i) {
                        const int rr = i * RPP + lr, row = row0 + rr;
                        const int nd = __shfl_sync(0xffffffffu, node, st * 16 + rr);
                        cp_async16(d0 + row * 128 + (((lc & 7) ^ (row & 7)) << 4), src + (nd < 0 ? 0 : nd) * row_stride, nd >= 0);
                    }
                }
                if (kv == 0 && cur.one) continue;
                cp_async_arrive(full_of(cur.g, at));      // by every lane, once its copies have landed
            }
            if (!alive) break;
            cur = nxt;
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    } else if (warp == 8 || warp == 9) {
        // ================================ products ================================
        const int g = warp - 8;
        // (as every role does before its first bounded wait: the grid ahead may run longer than the bound)
        if (a.meta_stable) asm volatile("griddepcontrol.wait;\n" ::: "memory");
        if (elect_one()) {
            const uint64_t dk = smem_desc(s_base, 16), dv = smem_desc(s_base, HALF), dv_one = smem_desc(s_base + TILE / 2, HALF / 2);
            const uint32_t idesc_pv = instr_desc(BF16, true, D), s_col = tmem_base + g * G::COLS, o_col = tmem_base + 2 * G::COLS + g * D;
            const uint4 *rows = reinterpret_cast<const uint4 *>(smem + G::OFF_ROWS) + g * (G::COLS / 16);
            bool alive = true;
            int round = 0, n = g;
            Where w = first;
#pragma unroll 1
            for (int item = blockIdx.x + g * stride; item < ta.n_items && alive; item += 2 * stride, n += 2, w = plus(w, step)) {
                const int own_rows = a.n_q - tile_of(w) * ROWS;
                alive = wait(q_of(n), q_parity(n), a.status, item);
                if (!alive) break;
                const int4 in = info[(n % ITEMS) * 2], counts = info[(n % ITEMS) * 2 + 1];
                const int tiles = in.x, four[4] = {counts.x, counts.y, counts.z, counts.w};
                const uint64_t dqs = dk + uint64_t(in.w * (TILE >> 4));
                int cnt[SUB];
#pragma unroll
                for (int s = 0; s < SUB; ++s) cnt[s] = four[s];
                if constexpr (BOTH) {
                    // the own tile and, when there are ancestors, one narrow tile: both products of S, then those of O as P comes
                    const int at = in.y, steps0 = min((own_rows + 15) >> 4, ROWS / 16), steps1 = (cnt[0] + 15) >> 4;
                    alive = wait(full_of(g, at), full_parity(at), a.status, item);
                    if (!alive) break;
                    int b = buf_of(g, at);
                    auto scores = [&](uint32_t to, uint64_t dks, int steps) {
                        const uint32_t idesc_s = instr_desc(BF16, false, 16 * steps);
                        fence_after_sync();
#pragma unroll
                        for (int ks = 0; ks < D / 16; ++ks) mma_f16(to, dqs + ks * 2, dks + ks * 2, idesc_s, ks > 0);
                    };
                    scores(s_col, dk + uint64_t(b * (TILE >> 4)), steps0);
                    int b1 = 0;
                    if (tiles > 1) {
                        alive = wait(full_of(g, at + 2), full_parity(at + 2), a.status, item);
                        if (!alive) break;
                        b1 = buf_of(g, at + 2);
                        fence_copied();
                        scores(s_col + BM, dk + uint64_t(b1 * (TILE >> 4)), steps1);
                    }
                    mma_commit(bar_s + g * 8);
                    mma_commit(bar_empty + b * 8);
                    // (V is usually there long before P)
                    alive = wait(full_of(g, at + 1), full_parity(at + 1), a.status, item) && wait(bar_p + g * 8, round & 1, a.status, item);
                    if (!alive) break;
                    ++round;
                    b = buf_of(g, at + 1);
                    fence_after_sync();
                    auto output = [&](auto most, int col, uint64_t dvs, int steps) {
                        constexpr int MOST = decltype(most)::value;
                        uint4 off[MOST];
#pragma unroll
                        for (int ks = 0; ks < MOST; ++ks) off[ks] = rows[(col >> 4) + ks];
#pragma unroll
                        for (int ks = 0; ks < MOST; ++ks)
                            if (ks < steps) mma_f16_ts_but(o_col, s_col + (col >> 1) + ks * 8, dvs + uint64_t((ks * 16 * 128) >> 4), idesc_pv, off[ks]);
                    };
                    output(std::integral_constant<int, 8>{}, 0, dv + uint64_t(b * (TILE >> 4)), steps0);
                    mma_commit(bar_empty + b * 8);
                    if (tiles > 1) {
                        mma_commit(bar_m + g * 8);        // O may be rescaled
                        alive = wait(bar_p + g * 8, round & 1, a.status, item);
                        if (!alive) break;
                        ++round;
                        fence_after_sync();
                        output(std::integral_constant<int, 4>{}, BM, dv_one + uint64_t(b1 * (TILE >> 4)), steps1);
                        mma_commit(bar_empty + b1 * 8);
                    }
                    mma_commit(bar_o + g * 8);
                } else {
                    // 16-column steps of tile t that some block has (bit ks: rows 16 ks .. of the buffer)
                    auto steps_of = [&](int t, int seg) -> uint32_t {
                        return t == 0 ? (1u << min((own_rows + 15) >> 4, ROWS / 16)) - 1u : live_steps<BM>(t, seg, cnt);
                    };
                    int at = in.y;                            // position of the tile's K rows
#pragma unroll 1
                    for (int t = 0; t < tiles; ++t, ++round) {
                        const bool narrow = in.z != 0 && t + 1 == tiles;
                        const uint32_t steps = steps_of(t, narrow ? BM / 2 : BM);
                        const uint32_t idesc_s = instr_desc(BF16, false, 16 * (32 - __clz(steps)));
                        alive = wait(full_of(g, at), full_parity(at), a.status, item);
                        if (!alive) break;
                        int b = buf_of(g, at);
                        const uint64_t dks = dk + uint64_t(b * (TILE >> 4)),
                                       half16 = (narrow ? HALF / 2 : HALF) >> 4;
                        if (t > 0) fence_copied();
                        fence_after_sync();
#pragma unroll
                        for (int ks = 0; ks < D / 16; ++ks)
                            mma_f16(s_col, dqs + uint64_t(((ks >> 2) * HALF + (ks & 3) * 32) >> 4),
                                    dks + (ks >> 2) * half16 + (ks & 3) * 2, idesc_s, ks > 0);
                        mma_commit(bar_s + g * 8);
                        if (!narrow) {
                            mma_commit(bar_empty + b * 8);
                            ++at;
                        }
                        alive = (narrow || wait(full_of(g, at), full_parity(at), a.status, item)) &&
                                wait(bar_p + g * 8, round & 1, a.status, item);
                        if (!alive) break;
                        b = buf_of(g, at);
                        ++at;
                        const uint64_t dvs = (narrow ? dv_one : dv) + uint64_t(b * (TILE >> 4));
                        if (t > 0) fence_copied();
                        fence_after_sync();
                        uint4 on[8];
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks) on[ks] = rows[ks];
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks)
                            if ((steps >> ks) & 1u)
                                mma_f16_ts_rows(o_col, s_col + ks * 8, dvs + uint64_t((ks * 16 * 128) >> 4), idesc_pv, on[ks]);
                        mma_commit(bar_empty + b * 8);
                        if (t + 1 == tiles) mma_commit(bar_o + g * 8);
                    }
                }
            }
        }
    } else if (warp == 15) {
        // ================================ O to global memory ================================
        if (elect_one()) {
            Where w = first;
            int n = 0;
            if (a.meta_stable) asm volatile("griddepcontrol.wait;\n" ::: "memory");
#pragma unroll 1
            for (int item = blockIdx.x; item < ta.n_items; item += stride, ++n, w = plus(w, step)) {
                if (!wait(bar_ob + (n % ITEMS) * 8, q_parity(n), a.status, item)) break;
                const int b = info[(n % ITEMS) * 2].w;
#pragma unroll
                for (int hf = 0; hf < DH; ++hf)
                    tma_store_4d(&tm_o, s_base + b * TILE + hf * HALF, hf * 64, tile_of(w) * ROWS, head_of(w), w.z);
                asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                arrive(bar_empty + b * 8);
            }
        }
    } else {
        // ================================ softmax ================================
        const int g = warp >> 2, r = tid & 127;           // my group and query row of its items
        const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
        const uint32_t tmem_s = tmem_base + g * G::COLS + lane_base, tmem_o = tmem_base + 2 * G::COLS + g * D + lane_base;
        const int sub = r / BM, j = r % BM;               // my block and row in it (sub is uniform in a warp)
        const float c2 = a.scale_log2;
        // mask words of my row: its own block's, and those from word w0 of its ancestor slots on (item and block may not exist)
        const uint32_t *mask = reinterpret_cast<const uint32_t *>(a.packed);
        const uint32_t blob_words = uint32_t(a.meta_stride >> 2), own0 = uint32_t(L.off_bmask >> 2) + j * NW,
                       ext0 = uint32_t(L.off_emask >> 2) + j * maw;
        auto own_words = [&](const Where &at, uint32_t (&w)[NW]) {
            const int b = tile_of(at) * SUB + sub;
            const bool ok = at.z < a.Z && b < a.nb;
            const uint32_t *from = mask + (uint32_t(at.z) * blob_words + own0 + uint32_t(b) * (BM * NW));
            if constexpr (NW == 4) {
                const uint4 v = ok ? __ldg(reinterpret_cast<const uint4 *>(from)) : make_uint4(0u, 0u, 0u, 0u);
                w[0] = v.x; w[1 % NW] = v.y; w[2 % NW] = v.z; w[3 % NW] = v.w;
            } else if constexpr (NW == 2) {
                const uint2 v = ok ? __ldg(reinterpret_cast<const uint2 *>(from)) : make_uint2(0u, 0u);
                w[0] = v.x; w[1 % NW] = v.y;
            } else {
                w[0] = ok ? __ldg(from) : 0u;
            }
        };
        auto ext_words = [&](const Where &at, int w0, uint32_t (&w)[EW]) {
            const int b = tile_of(at) * SUB + sub, left = at.z < a.Z && b < a.nb ? maw - w0 : 0;
            const uint32_t *from = mask + (uint32_t(at.z) * blob_words + ext0 + uint32_t(b) * uint32_t(BM * maw) + uint32_t(w0));
#pragma unroll
            for (int i = 0; i < EW; ++i) w[i] = i < left ? __ldg(from + i) : 0u;
        };
        uint32_t own[NW], ext[EW];
        Where at = first;
        own_words(at, own);
        ext_words(at, 0, ext);
        if (a.meta_stable) asm volatile("griddepcontrol.wait;\n" ::: "memory");

        bool alive = true;
        int round = 0, pairs = 0, n = g;                  // tiles, items with a second one (BOTH) so far; item number
#pragma unroll 1
        for (int item = blockIdx.x + g * stride; item < ta.n_items; item += 2 * stride, n += 2) {
            const Where at_next = plus(at, step);
            alive = __all_sync(0xffffffffu, wait(q_of(n), q_parity(n), a.status, item));
            if (!alive) break;
            const int4 in = info[(n % ITEMS) * 2];
            const int tiles = in.x;
            float m_ref = -INFINITY, l = 0.f;
            uint32_t zero[16];                            // my row of O, while S is on its way
#pragma unroll
            for (int c = 0; c < 16; ++c) zero[c] = 0u;
#pragma unroll 1
            for (int c0 = 0; c0 < D; c0 += 16) tmem_st16(tmem_o + c0, zero);
#pragma unroll 1
            for (int t = 0; t < tiles; ++t, ++round) {
                uint32_t word[NW];
#pragma unroll
                for (int i = 0; i < NW; ++i) word[i] = t == 0 ? own[i] : i < EW ? ext[i % EW] : 0u;
                // the words of the tile after next go out now: a loaded L2 answers late
                const bool last_tile = t + 1 == tiles;
                if (t == 0) own_words(at_next, own);
                if (t > 0 || last_tile) ext_words(last_tile ? at_next : at, last_tile ? 0 : t * NW, ext);
                const bool narrow = in.z != 0 && last_tile;
                const int segw = narrow ? NW / 2 : NW;    // my block's words in this tile; words past them are empty
                const int col_my = BOTH ? t * BM : sub * segw * 32;
                const uint32_t tmem_my = tmem_s + col_my;
                if (!BOTH || t == 0) {
                    alive = __all_sync(0xffffffffu, wait(bar_s + g * 8, (BOTH ? n >> 1 : round) & 1, a.status, item));
                    if (!alive) break;
                    fence_after_sync();
                }

                uint32_t live = 0;                        // bit i: some row of my warp has a bit in word i
                {
                    uint32_t on = 0;                      // lane k: rows of my warp with a column in step k of the tile
                    const int k = BOTH ? lane : lane - (col_my >> 4);
#pragma unroll
                    for (int i = 0; i < NW; ++i) {
                        const uint32_t lo = __ballot_sync(0xffffffffu, (word[i] & 0xffffu) != 0u), hi = __ballot_sync(0xffffffffu, word[i] > 0xffffu);
                        live |= uint32_t((lo | hi) != 0u) << i;
                        if (k == 2 * i) on = lo;
                        if (k == 2 * i + 1) on = hi;
                    }
                    if constexpr (BOTH) {
                        if (lane < (t == 0 ? 8 : 4)) reinterpret_cast<uint32_t *>(smem + G::OFF_ROWS)[(g * (G::COLS / 16) + t * 8 + lane) * 4 + (warp & 3)] = ~on;
                    } else if (lane < 8) {
                        reinterpret_cast<uint32_t *>(smem + G::OFF_ROWS)[(g * (G::COLS / 16) + lane) * 4 + (warp & 3)] = on;
                    }
                }
                float sum[2] = {0.f, 0.f}, mu = 0.f, mx = -INFINITY;
                // My live words, WT to a turn.  First round: the row's maximum, then the reference point.  Second round (or
                // at once, when one turn was all): probabilities, over S - word i of P covers columns 16 i .. of S,
                // below the words still to be read; words nobody uses are zeros.  One loop and one copy of its
                // code: what runs once per tile and does not stay in the instruction cache costs more than it saves
                // (two words to a turn at block_m 128: 1760 -> 1892 us on the forest of 65532 nodes; both words of
                // a row in one turn at block_m 64: 69.0 -> 67.5 us on the deep tree).
                constexpr int WT = NW == 2 ? 2 : 1;
                bool second = false;
                float alpha = 1.f;                        // what my row of O is to be scaled by
                if constexpr (BOTH) {
                    // A row that attends to nobody in its block but itself, as where the tree is numbered breadth first, needs no 32
                    // exponentials: where one word is all that a warp has, and one column of it all that a row has, the score is
                    // picked out (forest of 65532 nodes 1465 -> 1400 us).
                    uint32_t w = word[0];
#pragma unroll
                    for (int i = 1; i < NW; ++i) w |= word[i];
                    if (t == 0 && live != 0u && (live & (live - 1u)) == 0u && __ballot_sync(0xffffffffu, (w & (w - 1u)) != 0u) == 0u) {
                        const int wi = __ffs(live) - 1, at_c = __ffs(w) - 1;
                        uint32_t v[32], pk[16];
                        tmem_ld32(v, tmem_my + wi * 32);
                        tmem_ld_wait(v);
#pragma unroll
                        for (int half = 16; half > 0; half /= 2)
#pragma unroll
                            for (int c = 0; c < half; ++c) v[c] = (at_c & half) != 0 ? v[c + half] : v[c];
                        const float score = at_c < 0 ? -INFINITY : __uint_as_float(v[0]);
                        m_ref = fmaxf(m_ref, score);
                        const float p = fast_exp2(fmaf(score, c2, m_ref == -INFINITY ? 0.f : -(m_ref * c2)));
                        const uint32_t both = (at_c & 1) != 0 ? MT::pack(0.f, p) : MT::pack(p, 0.f);
#pragma unroll
                        for (int i = 0; i < 16; ++i) pk[i] = at_c >> 1 == i ? both : 0u;
                        tmem_st16(tmem_my + wi * 16, pk);
                        sum[0] = p;
                        live = 0u;
                    }
                }
#pragma unroll 1
                for (uint32_t rest = live; rest != 0u;) {
                    uint32_t s[WT][32];
                    int wi[WT];                           // the words' numbers; NW: none
#pragma unroll
                    for (int k = 0; k < WT; ++k) {
                        wi[k] = WT == 1 || rest != 0u ? __ffs(rest) - 1 : NW;
                        rest &= rest - 1;
                        if (WT == 1 || wi[k] < NW) tmem_ld32(s[k], tmem_my + wi[k] * 32);
                    }
                    float m = -INFINITY;
#pragma unroll
                    for (int k = 0; k < WT; ++k) {
                        if (WT > 1 && wi[k] >= NW) continue;
                        uint32_t w = word[0];
#pragma unroll
                        for (int i = 1; i < NW; ++i) w = wi[k] == i ? word[i] : w;
                        tmem_ld_wait(s[k]);
                        float m2[2] = {-INFINITY, -INFINITY};
#pragma unroll
                        for (int c = 0; c < 32; c += 2) {
                            s[k][c] = (w & (1u << c)) != 0u ? s[k][c] : 0xff800000u;
                            s[k][c + 1] = (w & (2u << c)) != 0u ? s[k][c + 1] : 0xff800000u;
                            m2[(c >> 1) & 1] = fmaxf(m2[(c >> 1) & 1], fmaxf(__uint_as_float(s[k][c]), __uint_as_float(s[k][c + 1])));
                        }
                        m = fmaxf(m, fmaxf(m2[0], m2[1]));
                    }
                    if (!second) {
                        mx = fmaxf(mx, m);
                        if (rest != 0u) continue;
                        const bool up = mx > m_ref;
                        if (BOTH ? up : __any_sync(0xffffffffu, up)) {
                            if (t > 0) alpha = up ? fast_exp2((m_ref - mx) * c2) : 1.f;
                            if (!BOTH && t > 0) {         // rescale my row of O (the stores are awaited with P's)
#pragma unroll 1
                                for (int c0 = 0; c0 < D; c0 += 16) {
                                    uint32_t o[16];
                                    tmem_ld16(o, tmem_o + c0);
#pragma unroll
                                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                                    tmem_st16(tmem_o + c0, o);
                                }
                                l *= alpha;
                            }
                            if (up) m_ref = mx;
                        }
                        mu = m_ref == -INFINITY ? 0.f : m_ref * c2;
                        second = true;
                        if (WT < NW && __popc(live) > WT) {       // more than a turn: once again from the first
                            rest = live;
                            continue;
                        }
                    }
#pragma unroll
                    for (int k = 0; k < WT; ++k) {
                        if (WT > 1 && wi[k] >= NW) continue;
                        uint32_t pk[16];
#pragma unroll
                        for (int c = 0; c < 32; c += 2) {
                            const float p0 = fast_exp2(fmaf(__uint_as_float(s[k][c]), c2, -mu));
                            const float p1 = fast_exp2(fmaf(__uint_as_float(s[k][c + 1]), c2, -mu));
                            sum[0] += p0;
                            sum[1] += p1;
                            pk[c >> 1] = MT::pack(p0, p1);
                        }
                        tmem_st16(tmem_s + (col_my >> 1) + wi[k] * 16, pk);
                    }
                }
                if (BOTH && t > 0) {                      // rescale it here, once the first tile's product has landed
                    alive = __all_sync(0xffffffffu, wait(bar_m + g * 8, pairs & 1, a.status, item));
                    if (!alive) break;
                    ++pairs;
                    fence_after_sync();
                    if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
                        for (int c0 = 0; c0 < D; c0 += 16) {
                            uint32_t o[16];
                            tmem_ld16(o, tmem_o + c0);
#pragma unroll
                            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                            tmem_st16(tmem_o + c0, o);
                        }
                        l *= alpha;
                    }
                }
                l += sum[0] + sum[1];
                tmem_st_wait();
                fence_before_sync();
                arrive(bar_p + g * 8);
            }
            if (!alive) break;

            // ---- O / l into the item's Q buffer (same swizzled layout), for warp 15 to store
            alive = __all_sync(0xffffffffu, wait(bar_o + g * 8, (n >> 1) & 1, a.status, item));
            if (!alive) break;
            fence_after_sync();
            const float inv = l > 0.f ? 1.f / l : 0.f;
            unsigned char *orow = smem + in.w * TILE + r * 128;
#pragma unroll 1
            for (int c0 = 0; c0 < D; c0 += 32) {
                uint32_t o[32];
                tmem_ld32(o, tmem_o + c0);
                tmem_ld_wait(o);
                unsigned char *to = orow + (c0 >> 6) * HALF;
                const int chunk0 = (c0 >> 3) & 7;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t v[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        v[i] = MT::pack(__uint_as_float(o[q * 8 + 2 * i]) * inv, __uint_as_float(o[q * 8 + 2 * i + 1]) * inv);
                    *reinterpret_cast<uint4 *>(to + (((chunk0 + q) ^ (r & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
                }
            }
            fence_before_sync();
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            arrive(bar_ob + (n % ITEMS) * 8);
            const int row = tile_of(at) * ROWS + r;
            if (a.lse != nullptr && row < a.n_q)
                a.lse[(size_t(at.z) * a.H + head_of(at)) * a.n_q + row] = m_ref * c2 + log2f(l);
            at = at_next;
        }
    }

    fence_before_sync();
    __syncthreads();
    if (warp == 9) tmem_free_all(tmem_base);
}

// ---- host side ---------------------------------------------------------------------------------

template <typename T, int D, int BM, tree_umma::Round ROUND>
cudaError_t launch_tree_umma_t(const AttnArgs &a, cudaStream_t stream) {
    using G = tree_umma::Geo<D>;
    constexpr bool bf16 = !std::is_same<T, __half>::value;
    const int H_kv = a.H / a.kv_group;
    alignas(64) CUtensorMap tq, tk, tv, to;
    if (!make_map(&tq, a.q, bf16, D, a.n_q, a.H, a.Z, a.qs_n, a.qs_h, a.qs_z, tree_umma::ROWS) ||
        !make_map(&tk, a.k, bf16, D, a.n_kv, H_kv, a.Z, a.ks_n, a.ks_h, a.ks_z, tree_umma::ROWS) ||
        !make_map(&tv, a.v, bf16, D, a.n_kv, H_kv, a.Z, a.vs_n, a.vs_h, a.vs_z, tree_umma::ROWS) ||
        !make_map(&to, a.o, bf16, D, a.n_q, a.H, a.Z, a.os_n, a.os_h, a.os_z, tree_umma::ROWS))
        return cudaErrorNotSupported;
    static DeviceOnce configured;
    const cudaError_t ce = configured.run([&] {
        return cudaFuncSetAttribute(tree_umma_kernel<T, D, BM, ROUND>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM_BYTES);
    });
    if (ce != cudaSuccess) return ce;
    TreeUmmaArgs ta = {};
    ta.row_tiles = (a.n_q + tree_umma::ROWS - 1) / tree_umma::ROWS;
    const long long items = (long long)ta.row_tiles * a.H * a.Z;
    // item numbers are ints, mask words are addressed with 32-bit offsets
    if (items > 0x3fffffff || size_t(a.Z) * a.meta_stride / 4 + packed_layout(a.nb, BM, a.ma).total / 4 > 0xfffffffeu)
        return cudaErrorNotSupported;
    ta.n_items = int(items);
    ta.heads_first = items <= 8LL * sm_count() ? 1 : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(std::min<long long>(items, sm_count())));
    cfg.blockDim = dim3(tree_umma::THREADS);
    cfg.dynamicSmemBytes = G::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, tree_umma_kernel<T, D, BM, ROUND>, a, ta, tq, tk, tv, to);
}

template <typename T, int D>
cudaError_t launch_tree_umma_d(const AttnArgs &a, cudaStream_t stream) {
    using tree_umma::Round;
    switch (a.bm) {
        case 32: return launch_tree_umma_t<T, D, 32, Round::TILE>(a, stream);
        case 64: return launch_tree_umma_t<T, D, 64, Round::TILE>(a, stream);
        case 128:
            if constexpr (D == 64)
                if (a.ma <= 64) return launch_tree_umma_t<T, D, 128, Round::BOTH>(a, stream);
            return launch_tree_umma_t<T, D, 128, Round::TILE>(a, stream);
    }
    return cudaErrorNotSupported;
}

}  // namespace fst
