// Attention behind a shared prefix on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// The prefix part of the reference kernel (fstattention.py:113-136) is plain dense attention: every query
// row attends to every prefix row.  A CTA has one or two query tiles of 128 rows and a run of column tiles;
// the column tiles of a query tile are the prefix in 128-row tiles, then the tree: one tile with the
// query tile's own K/V rows and, behind it, tiles of gathered ancestors, in which every block of the query tile has
// a segment of columns.  Tree tiles are masked by the rows' mask words and cost what a prefix tile costs; a 16-column
// step of their second product updates the rows that have a column in it and no others, so that a V that is not
// finite stays with those (32 heads of 256 rows behind 4096: 30.1 us with and without).
// Per query tile and column tile, a step:
//     S = Q K^T             tcgen05.mma  M=128 N=128 K=16 x D/16, both operands K-major in shared memory
//     P = softmax part      one thread per query row (TMEM lane = row, so no shuffles): a row of S in 128 registers,
//                           probabilities against a lazily moved reference point, P back to tensor memory
//     O += P V              tcgen05.mma  A = P in tensor memory, B = V (MN-major: rows of V are the K index)
// K/V tiles arrive by TMA (128-row x 64-column boxes, 128-byte swizzle; gathered rows by cp.async into the same
// layout) in a ring of stages.  Head dimension D is 64 or 128: one or two 64-column halves per Q / K / V tile.
//
// Shared-memory bandwidth is what a tile costs: at D 128 the two products read 96 KB of operands and the tile's
// K and V come in with 64 KB, against 1024 cycles of tensor work.  Hence P in tensor memory (writing it to and
// reading it from shared memory took another 64 KB), and hence two query tiles to a CTA where there are two
// that read the same K and V - neighbouring rows of a tree, or other heads of a grouped-query group: a
// K/V tile then comes in once for both.  Two softmax groups of four warps take a query tile each; with one
// query tile they take its column tiles in turn and their results are merged at the end.  Either way a
// group's barrier waits and tensor-memory latencies hide behind the other's exponentials.
//
// Twelve warps.  Warps 0-3 and 4-7 are the softmax groups; warp 8 loads K and V; one lane of warp 9 issues the
// products, the two groups' in turn: O += P V, then the group's next S (which overwrites P: tcgen05.mma
// of one thread run in order); warps 10 and 11 gather the K and the V rows of ancestors when warp 8 says that their stage
// is free.  All hand-offs are mbarriers (TMA completion, tcgen05.commit, or arrivals by the 128 threads of a group).
// A stage's fills are claimed in order by warp 8 alone, so no waiter is ever two phases behind or one ahead.
//
// Runs: the column tiles of a query tile are cut into up to eight runs, one CTA each, which form a
// cluster.  Every CTA leaves its rows, unnormalised, in its shared memory; each then merges its share of the rows
// out of all of them and writes the output.  There are no partial results in memory and no second kernel -
// except where clusters would leave SMs idle (prefix_plan): then every run leaves its rows in a workspace.
//
// With grouped-query attention a small tree's rows of several heads share a query tile (see
// prefix_heads_per_tile): the tile is loaded as one box per head and its rows go to their heads at the end.
//
// PAGED = true reads the prefix rows from a page pool through a block table (a KV cache): a
// tile is 128 / page_size pages and lane j of the loading warp requests page j.  The rows of a sequence's last page
// past its end hold whatever the cache holds, and a NaN or an infinity there times a probability of zero
// would be a NaN: 16-row steps of V past the end are left out, and where a step straddles it warp 11 clears the
// rows behind it before the product (eight
// sequences of up to 3001 rows, 8 K/V heads: 39.2 us without, 39.9 with it).
//
// Every wait is bounded in time (mbar_wait): on expiry the kernel records FST_DEV_TIMEOUT, stops
// issuing, frees its tensor memory and returns.

#include "fst_plan.h"
#include "fst_umma.cuh"

namespace fst {

namespace umma {

constexpr int QM = 128;                // query rows per tile (MMA M)
constexpr int KN = 128;                // K/V rows per tile (MMA N of the first product)

// Shared memory for head dimension D (64 or 128): a Q / K / V tile is 128 rows of D columns, D / 64 halves.
// One or two Q tiles, the rest of the tiles are the ring of K/V stages; then barriers.  At the end the
// groups' rows (fp32) and their statistics take the tiles' place.
template <int D>
struct Geo {
    static constexpr int TILE = (D / 64) * HALF;
    static constexpr int TILES = D == 128 ? 7 : 12;
    static constexpr int MAX_RING = TILES - 1;
    static constexpr int OFF_BAR = TILES * TILE;
    static constexpr int OFF_ROWS = OFF_BAR + 384;            // [tile parity][group][step][warp] rows with columns in a step of a tree tile
    static constexpr int SMEM_BYTES = OFF_ROWS + 512 + 1024;  // + 1 KB alignment slack
    static constexpr int OFF_STATS = 2 * QM * D * 4;          // [256] (exponent, sum) of the groups' rows, [256] of the CTA's
};
static_assert(Geo<128>::SMEM_BYTES <= 227 * 1024 && Geo<64>::SMEM_BYTES <= 227 * 1024, "one CTA's shared memory");
static_assert(Geo<128>::OFF_STATS + 4 * QM * 8 <= Geo<128>::OFF_BAR, "merge buffers fit");
static_assert(Geo<64>::OFF_STATS + 4 * QM * 8 <= Geo<64>::OFF_BAR, "merge buffers fit");
static_assert(1 + 3 * Geo<64>::MAX_RING + 9 <= 46, "barriers fit");

// the same word of shared memory in CTA `cta` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, int cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}
__device__ __forceinline__ float4 cluster_ld4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 cluster_ld2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}
// every thread of every CTA of the cluster; shared memory written before is visible after
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

}  // namespace umma

// Arguments of the prefix kernel beyond AttnArgs.
struct PrefixArgs {
    int n_runs;          // runs of column tiles
    int cluster;         // CTAs of a cluster: n_runs, or 1 where every run leaves a partial result of its own
    int pair;            // two query tiles to a CTA
    int q_tiles;         // query tiles of a head (or pack of heads)
    int kv_tiles;        // query tiles that read one K/V head
    int bm_shift;                        // block_m is 1 << bm_shift
    int pack, pack_shift;                // heads per query tile; a head's rows are 1 << pack_shift of the tile's
    // paged prefix: K/V rows live in pages of page_size rows; block_table[z][i] is the page
    // holding rows [i * page_size, (i + 1) * page_size) of batch element z, prefix_lens[z] its
    // number of prefix rows (AttnArgs::prefix is then the largest of them)
    const int32_t *block_table;
    const int32_t *prefix_lens;
    int table_stride, page_size, n_pages;
};

constexpr int PFX_SOFTMAX = 256;       // eight softmax warps: two groups of 128, one thread per query row each
constexpr int PFX_THREADS = PFX_SOFTMAX + 128;  // + loading, issuing and two gathering warps

// A query tile: its nodes [q0, q0 + rows) of heads h .. h + pack - 1 in blocks b0 .. b0 + n_blk - 1, every block
// with a segment of 1 << seg_shift columns in a gathered tile.
struct QueryTile {
    int h, q0, rows, b0, n_blk, seg_shift;
    __device__ __forceinline__ QueryTile(const AttnArgs &a, const PrefixArgs &pa, int head, int first) {
        h = head;
        q0 = first;
        rows = min(a.n_q - q0, 1 << pa.pack_shift);
        b0 = q0 >> pa.bm_shift;
        n_blk = (rows + a.bm - 1) >> pa.bm_shift;
        seg_shift = n_blk > 2 ? 5 : n_blk > 1 ? 6 : 7;
    }
};

template <typename T, int D, bool PAGED>
__global__ void __launch_bounds__(PFX_THREADS, 1)
prefix_umma_kernel(const AttnArgs a, const PrefixArgs pa, const __grid_constant__ CUtensorMap tm_q,
                   const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                   const __grid_constant__ CUtensorMap tm_kt, const __grid_constant__ CUtensorMap tm_vt) {
    using namespace umma;
    using MT = MmaTraits<T>;
    using G = Geo<D>;
    constexpr bool BF16 = !std::is_same<T, __half>::value;
    constexpr int DH = D / 64;                            // 64-column halves of a Q / K / V tile
    constexpr int TILE = G::TILE;

    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    extern __shared__ unsigned char smem_raw[];
    const uint32_t s_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *smem = smem_raw + (s_base - smem_u32(smem_raw));
    const int hk = blockIdx.y, z = blockIdx.z / pa.n_runs, run = blockIdx.z - z * pa.n_runs;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, qt = blockIdx.x;
    const int n_q = a.n_q;
    const int x0 = pa.pair ? blockIdx.x * 2 : blockIdx.x;
    const bool two = pa.pair && x0 + 1 < pa.kv_tiles;     // two query tiles ...
    const bool same = pa.q_tiles == 1;                    // ... of the same nodes, so that tree tiles are shared as well
    // the two query tiles; query(0) is the one where there is only one
    const int sub0 = x0 / pa.q_tiles, n0 = x0 - sub0 * pa.q_tiles, h0 = hk * a.kv_group + sub0 * pa.pack;
    const bool wraps = n0 + 1 == pa.q_tiles;              // the second one is the next heads' first
    auto query = [&](int g) { return QueryTile(a, pa, g && wraps ? h0 + pa.pack : h0, g ? (wraps ? 0 : n0 + 1) * QM : n0 * QM); };
    const int ring = G::TILES - (two ? 2 : 1);
    // Order of the loads.  skew: K of the next unit ahead of V.  K is done with after the first product and V a softmax later, so in
    // the order of use K waited for a stage behind an earlier V, was requested some 2500 cycles before its product and
    // came late for every fourth tile of a query tile by itself at D 128 (six stages; 32 heads of 256 rows behind
    // 4096: 27.0 -> 26.2 us).  Two query tiles, the longer ring of D 64 and runs spread over the GPU lose 1 to 3 % by it.
    const bool skew = !PAGED && D == 128 && !two && pa.cluster > 1;
    auto k_item = [&](int u) { return skew ? max(2 * u - 1, 0) : 2 * u; };
    auto v_item = [&](int u) { return 2 * u + (skew ? 2 : 1); };
    const uint32_t s_ring = s_base + (two ? 2 : 1) * TILE;

    // barriers: Q, full / empty / go (a gathered tile may be written) of every stage, S (landed), P (written), O (all
    // products done) of either group, V rows of a paged prefix's last tile (landed, to be cleared past the end)
    const uint32_t bar_q = s_base + G::OFF_BAR, bar_full = bar_q + 8, bar_empty = bar_full + G::MAX_RING * 8,
                   bar_go = bar_empty + G::MAX_RING * 8, bar_s = bar_go + G::MAX_RING * 8, bar_p = bar_s + 16, bar_o = bar_p + 32, bar_tail = bar_o + 16;    // P: [half][group]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + G::OFF_BAR + 376);

    if (warp == 8) {
        if (lane == 0) {
            mbar_init(bar_q, 1);
            mbar_init(bar_tail, 1);
            for (int i = 0; i < 3 * G::MAX_RING; ++i) mbar_init(bar_full + i * 8, 1);
            for (int i = 0; i < 2; ++i) {
                mbar_init(bar_s + i * 8, 1);
                mbar_init(bar_p + i * 8, PFX_SOFTMAX / 2);
                mbar_init(bar_p + 16 + i * 8, PFX_SOFTMAX / 2);
                mbar_init(bar_o + i * 8, 1);
            }
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        __syncwarp();
    } else if (warp == 9) {                               // tensor memory: S, O of either group (and P at D 64)
        tmem_alloc_all(smem_u32(tmem_slot));
        fence_before_sync();
    }
    // Launched with programmatic stream serialisation: wait for the grid ahead before the first access to memory.
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    // the loading warp does not wait for the others: barriers are its own work, its first loads leave at once
    if (warp == 8) asm volatile("bar.arrive 2, 384;\n" ::: "memory");
    else asm volatile("bar.sync 2, 384;\n" ::: "memory");

    // prefix rows of my batch element (paged: every batch element has its own count)
    const int prefix = PAGED ? max(0, min(__ldg(pa.prefix_lens + z), a.prefix)) : a.prefix;
    const PackedLayout L = packed_layout(a.nb, a.bm, a.ma);
    const unsigned char *blob = a.packed + size_t(z) * a.meta_stride;
    // ancestors of the tile's block s that lie outside it
    auto external = [&](const QueryTile &qt_, int s) -> int {
        return s < qt_.n_blk ? min(max(__ldg(reinterpret_cast<const int32_t *>(blob + L.off_count) + qt_.b0 + s), 0), a.ma) : 0;
    };
    auto gathered_tiles = [&](const QueryTile &qt_) -> int {
        const int longest = max(max(external(qt_, 0), external(qt_, 1)), max(external(qt_, 2), external(qt_, 3)));
        return (longest + (1 << qt_.seg_shift) - 1) >> qt_.seg_shift;
    };
    // My run of column tiles [T0, T0 + nt): tp prefix tiles, the own tile, gathered tiles.  The runs are cut as if
    // there were one gathered tile, so that no CTA waits for the counts before its first loads; nt_sure
    // tiles of the run are there whatever they say.
    const int tp = (prefix + KN - 1) / KN, per = (tp + 2 + pa.n_runs - 1) / pa.n_runs;
    const int T0 = run * per, T1 = run + 1 == pa.n_runs ? 0x3fffffff : T0 + per;
    const int nt_sure = max(0, min(T1, tp + 1) - T0);
    auto count_tiles = [&]() -> int {
        int g = gathered_tiles(query(0));
        if (two && !same) g = max(g, gathered_tiles(query(1)));
        return max(0, min(T1, tp + 1 + g) - T0);
    };
    // Steps j = 0, 1, ...: group j & 1 and column tile T0 + (two ? j >> 1 : j).  K/V tiles (units) are shared by
    // two steps each in the first 2 * shared steps (all of them when the two query tiles have the same nodes, else those
    // of the prefix); every other step has a unit of its own.
    // whether the prefix ends inside a 16-row step of V and whether that tile is in my run (it is shared if two is)
    const bool tail = PAGED && (prefix & 15) != 0 && T0 < tp && tp <= T1;
    auto n_shared = [&](int nt) -> int { return !two ? 0 : same ? nt : min(max(tp - T0, 0), nt); };
    const int nt_all = warp == 8 ? 0 : count_tiles();     // (the loading warp asks when it has nothing else to do)

    if (warp == 8) {
        // ====== loads: K and V of unit u are items k_item(u) and v_item(u) of the ring.  The whole warp for a paged prefix, one lane
        // otherwise.  Paged: a tile is KN / page_size pages, one pair of boxes each, and lane j takes page j - it
        // reads that page's number from the block table a tile before it requests the boxes, so the
        // table's latency is off the path, and a single thread is not left to issue sixteen copies one after
        // the other.  Pages past the end of my batch element's prefix repeat its last page. ======
        const bool lead = elect_one();
        if (PAGED || lead) {
            const int ps = PAGED ? pa.page_size : KN, npt = KN / ps;
            const int32_t *table = PAGED ? pa.block_table + size_t(z) * pa.table_stride : nullptr;
            const int last_page = PAGED ? max(prefix - 1, 0) / ps : 0;
            auto my_page = [&](int tile) -> int {
                return PAGED && lane < npt && tile < tp ? __ldg(table + min(tile * KN / ps + lane, last_page)) : 0;
            };
            int page = my_page(T0), page_v = 0;           // of the next K's tile, of the next V's
            bool known = false, alive = true;
            int nt = nt_sure, st = 0;
            uint32_t use = 0;                             // fills of the current stage before this one
            const int shared = n_shared(nt_sure);         // the same for the final count: see above
            int n_units = (two ? 2 : 1) * nt - shared, i0 = 0;
            auto unit_of = [&](int i) { return skew ? (i & 1 ? (i + 1) >> 1 : max(i - 2, 0) >> 1) : i >> 1; };
            auto v_next = [&](int i) { return skew ? i > 0 && (i & 1) == 0 : (i & 1) != 0; };
            auto load_q = [&]() {
                mbar_arrive_expect_tx(bar_q, (two ? 2 : 1) * TILE);
#pragma unroll 1
                for (int g = 0; g < (two ? 2 : 1); ++g) {
                    const QueryTile me = query(g);
#pragma unroll 1
                    for (int k = 0; k < pa.pack; ++k)
#pragma unroll
                        for (int hf = 0; hf < DH; ++hf)
                            tma_load_4d(s_base + g * TILE + hf * HALF + (k << pa.pack_shift) * 128, &tm_q, hf * 64, me.q0, me.h + k, z, bar_q);
                }
            };
            const int head_start = (two ? 2 : 4) + int(skew);         // everybody's first steps go ahead of the rest
            if constexpr (!PAGED && D == 128) {
                // Whole prefix tiles by themselves: with everything that the others need decided for every item one took some
                // 770 cycles, and a query tile's K and V together 1540 of the 1700 that its softmax takes.
                const int n_plain = min(max(tp - T0, 0), nt), limit = n_plain == 0 ? 0 : 2 * n_plain - int(skew);
                if (n_plain > 0) load_q();
#pragma unroll 1
                for (; i0 < limit; ++i0) {
                    const bool v = v_next(i0);
                    const uint32_t bar = bar_full + st * 8, dst = s_ring + st * TILE;
                    if (i0 == head_start) alive = mbar_wait(bar_full, 0, a.status, qt);
                    if (use > 0) alive = alive && wait(bar_empty + st * 8, (use - 1) & 1, a.status, qt);
                    if (!alive) break;
                    mbar_arrive_expect_tx(bar, TILE);
#pragma unroll
                    for (int hf = 0; hf < DH; ++hf) tma_load_4d(dst + hf * HALF, v ? &tm_vt : &tm_kt, hf * 64, (T0 + unit_of(i0)) * KN, hk, z, bar);
                    if (++st == ring) {
                        st = 0;
                        ++use;
                    }
                }
            }
#pragma unroll 1
            for (int i = i0; alive; ++i) {
                const bool is_v = v_next(i);
                const int u = unit_of(i);
                if (u >= n_units && !known) {             // only now ask how many gathered tiles there are
                    known = true;
                    nt = count_tiles();
                    n_units = (two ? 2 : 1) * nt - n_shared(nt);
                }
                if (u >= n_units && (is_v || !skew)) break;
                if (u < n_units) {
                    if (lead && i == 0) load_q();         // when there is anything to do: nobody would wait for it otherwise
                    const int x = u - shared, g = two && !same && x >= 0 ? x & 1 : 0;
                    const int tile = T0 + (two && !same && x >= 0 ? shared + (x >> 1) : u);
                    if (PAGED && !is_v) {
                        page_v = page;
                        if (tile + 1 < tp) page = my_page(tile + 1);
                    }
                    const int here = page_v;
                    const uint32_t dst = s_ring + st * TILE, bar = tail && is_v && tile + 1 == tp ? bar_tail : bar_full + st * 8;
                    if (i == head_start && T0 <= tp) {
                        if (lead) alive = mbar_wait(bar_full, 0, a.status, qt);
                        if (PAGED) alive = __all_sync(0xffffffffu, alive);
                        if (!alive) break;
                    }
                    if (use > 0) {
                        if (lead) alive = mbar_wait(bar_empty + st * 8, (use - 1) & 1, a.status, qt);
                        if (PAGED) alive = __all_sync(0xffffffffu, alive);
                        if (!alive) break;
                    }
                    if (tile > tp) {                      // gathered: the gathering warp's turn
                        if (lead) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar_go + st * 8) : "memory");
                    } else {
                        if (lead) mbar_arrive_expect_tx(bar, TILE);
                        if (PAGED) __syncwarp();
                        const bool pool = PAGED && tile < tp;
                        const CUtensorMap *map = pool ? (is_v ? &tm_v : &tm_k) : (is_v ? &tm_vt : &tm_kt);
                        if (pool ? lane < npt : lead) {
                            if (pool && unsigned(here) >= unsigned(pa.n_pages))   // the boxes then read as zeros
                                report(a.status, FST_DEV_INDEX_RANGE, z, tile * KN / ps + lane);
                            const int row = pool ? 0 : tile < tp ? tile * KN : (PAGED ? 0 : a.prefix) + query(g).q0;
                            const uint32_t to = dst + (pool ? lane * ps * 128 : 0);
#pragma unroll
                            for (int hf = 0; hf < DH; ++hf) tma_load_4d(to + hf * HALF, map, hf * 64, row, hk, pool ? here : z, bar);
                        }
                    }
                }
                if (++st == ring) {                       // (the place of a K that does not exist stays empty)
                    st = 0;
                    ++use;
                }
            }
        }
    } else if (warp == 9) {
        // ====== products: one lane issues O += P V of step j, then S of step j + 2 ======
        if (elect_one()) {
            fence_after_sync();
            const uint32_t tmem = *tmem_slot;
            const int nt = nt_all, shared = n_shared(nt), n_steps = (two ? 2 : 1) * nt;
            const uint32_t idesc_s = instr_desc(BF16, false, KN), idesc_pv = instr_desc(BF16, true, D);
            // descriptors of the tiles' first 16-wide step; a step further on adds its byte offset / 16
            const uint64_t dq = smem_desc(s_base, 16), dk = smem_desc(s_ring, 16), dv = smem_desc(s_ring, HALF);
            int k_st = 0, v_st = v_item(0), k_by = k_item(1);     // stages of the next K and the next V tile, items to the K after
            uint32_t k_ph = 0, v_ph = 0;
            auto next = [&](int &st, uint32_t &ph, int by) {
                st += by;
                if (st >= ring) {
                    st -= ring;
                    ph ^= 1u;
                }
            };
            bool alive = n_steps > 0 && mbar_wait(bar_q, 0, a.status, qt);
#pragma unroll 1
            for (int j = -2; j < n_steps && alive; ++j) {
                const int g = j & 1;
                const uint32_t tmem_s = tmem + g * 128, tmem_o = tmem + 256 + g * D, tmem_p = D == 128 ? tmem_s : tmem + 384 + g * 64;
                if (j >= 0) {
                    alive = mbar_wait(bar_full + v_st * 8, v_ph, a.status, qt) &&
                            mbar_wait(bar_p + g * 8, (j >> 1) & 1, a.status, qt);       // the first half of P is in tensor memory
                    if (!alive) break;
                    fence_after_sync();
                    // rows of a gathered tile past the lists' ends were never fetched, and those of the prefix's last
                    // tile past its end are not its own
                    const int tile = T0 + (two ? j >> 1 : j);
                    uint32_t live = 0xffu;
                    if (tile + 1 == tp) {
                        live = (1u << ((prefix - tile * KN + 15) >> 4)) - 1u;
                    } else if (tile > tp) {
                        const QueryTile me = query(two && !same ? g : 0);
                        const int slot0 = (tile - tp - 1) << me.seg_shift;
                        live = 0u;
#pragma unroll 1
                        for (int s = 0; s < me.n_blk; ++s) {
                            const int left = min(external(me, s) - slot0, 1 << me.seg_shift), steps = left > 0 ? (left + 15) >> 4 : 0;
                            live |= ((1u << steps) - 1u) << (s << me.seg_shift >> 4);
                        }
                    }
                    const uint64_t dvs = dv + uint64_t(v_st * (TILE >> 4));
                    auto steps = [&](auto &&product) {            // 16 rows of V each
#pragma unroll
                        for (int ks = 0; ks < KN / 16; ++ks) {
                            if (ks == KN / 32) {                  // the rest of P
                                alive = mbar_wait(bar_p + 16 + g * 8, (j >> 1) & 1, a.status, qt);
                                fence_after_sync();
                            }
                            if ((live >> ks) & 1u) product(ks, dvs + uint64_t((ks * 16 * 128) >> 4));
                        }
                    };
                    if (tile < tp) {
                        steps([&](int ks, uint64_t dvk) { mma_f16_ts(tmem_o, tmem_p + ks * 8, dvk, idesc_pv, true); });
                    } else {
                        const uint4 *rows = reinterpret_cast<const uint4 *>(smem + G::OFF_ROWS) + ((j >> 1 & 1) * 2 + g) * 8;
                        steps([&](int ks, uint64_t dvk) { mma_f16_ts_rows(tmem_o, tmem_p + ks * 8, dvk, idesc_pv, rows[ks]); });
                    }
                    if (j >= 2 * shared || g == 1) {      // the last to read this V
                        mma_commit(bar_empty + v_st * 8);
                        next(v_st, v_ph, 2);
                    }
                }
                const int j2 = j + 2;
                if (j2 >= n_steps) {
                    if (j >= 0) mma_commit(bar_o + g * 8);        // all of the group's products
                    continue;
                }
                alive = mbar_wait(bar_full + k_st * 8, k_ph, a.status, qt);
                if (!alive) break;
                fence_after_sync();
                const uint64_t dqs = dq + uint64_t((two ? g : 0) * (TILE >> 4)), dks = dk + uint64_t(k_st * (TILE >> 4));
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    const uint64_t koff = ((ks >> 2) * HALF + (ks & 3) * 32) >> 4;
                    mma_f16(tmem_s, dqs + koff, dks + koff, idesc_s, ks > 0);
                }
                mma_commit(bar_s + g * 8);
                if (j2 >= 2 * shared || g == 1) {         // the last to read this K
                    mma_commit(bar_empty + k_st * 8);
                    next(k_st, k_ph, k_by);
                    k_by = 2;
                }
            }
        }
    } else if (warp >= 10) {
        // ====== two gathering warps: ancestors' K rows (10) and V rows (11), whole steps of 16 rows at a time ======
        const int nt = nt_all, shared = n_shared(nt), n_units = (two ? 2 : 1) * nt - shared;
        const int plain = min(max(tp + 1 - T0, 0), nt), u0 = (two ? 2 : 1) * plain - min(shared, plain);
        const T *src = warp == 10 ? static_cast<const T *>(a.k) + z * a.ks_z + hk * a.ks_h
                                  : static_cast<const T *>(a.v) + z * a.vs_z + hk * a.vs_h;
        const int64_t row_stride = warp == 10 ? a.ks_n : a.vs_n;
        constexpr int CH = D / 8, RPP = 32 / CH;          // 16-byte chunks per row, rows per pass of the warp
        const int lr = lane / CH, lc = lane % CH;
        src += (PAGED ? 0 : a.prefix) * row_stride + lc * 8;
        auto item_of = [&](int u) { return warp == 10 ? k_item(u) : v_item(u); };
        // (stage and parity go along where the order is the plain one: 177 rows of 42 heads and 4 trees behind 401, where
        // they are on the path, 43.4 -> 42.9 us against a division and a count for each tile)
        int st = (2 * u0 + (warp - 10)) % ring, turn = warp - 10;     // stage; items since the first gathered one, mod ring
        uint32_t go_ph = 0;
        // skew: parity of a stage's turns so far, its earlier items that were gathered
        auto turn_of = [&](int item) -> uint32_t {
            uint32_t odd = 0;
#pragma unroll 1
            for (int i = item - ring; i >= k_item(u0); i -= ring) odd ^= uint32_t((i & 1) || i == 0 || i >= v_item(u0));
            return odd;
        };
        // The first pass, while the tensor cores are at the prefix, only asks for the rows to be brought into L2: a
        // unit's count, indices and rows are three memory latencies one after the other.
        const bool early = u0 > 0;
#pragma unroll 1
        for (int v = early ? 2 * u0 - n_units : u0; v <= n_units; ++v) {
            if (PAGED && v == u0 && tail && warp == 11) { // ahead of the gathered tiles: rows behind the prefix's end
                const int left = prefix - (tp - 1) * KN, rows = -left & 15, at = v_item(tp - 1 - T0) % ring;
                if (!__all_sync(0xffffffffu, mbar_wait(bar_tail, 0, a.status, qt))) break;
                for (int i = lane; i < rows * DH * 8; i += 32)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n"
                                 ::"r"(s_ring + at * TILE + (DH > 1 && (i & 8) ? HALF : 0) + (left + i / (DH * 8)) * 128 + (i & 7) * 16), "r"(0) : "memory");
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar_full + at * 8) : "memory");
            }
            if (v == n_units) break;
            const bool fetch = v >= u0;
            const int u = fetch ? v : v + n_units - u0, x = u - shared, tile = T0 + (two && !same ? shared + (x >> 1) : u);
            const QueryTile me = query(two && !same ? x & 1 : 0);
            const int seg = 1 << me.seg_shift, slot0 = (tile - tp - 1) << me.seg_shift;
            // a step's rows: lanes 0-15 those of an even step, lanes 16-31 those of the odd one behind it
            int node[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int row = k * 32 + lane, s = row >> me.seg_shift, slot = slot0 + (row & (seg - 1));
                node[k] = -1;
                if (s < me.n_blk && slot < external(me, s)) {
                    node[k] = __ldg(reinterpret_cast<const int32_t *>(blob + L.off_idx) + size_t(me.b0 + s) * a.ma + slot);
                    if (node[k] >= n_q) {
                        report(a.status, FST_DEV_INDEX_RANGE, me.b0 + s, slot);
                        node[k] = -1;
                    }
                }
            }
            if (!fetch) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (node[k] >= 0)
#pragma unroll
                        for (int hf = 0; hf < DH; ++hf)
                            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(src - lc * 8 + node[k] * row_stride + hf * 64));
                continue;
            }
            if (skew) {
                st = item_of(u) % ring;
                go_ph = turn_of(item_of(u));
            }
            if (!__all_sync(0xffffffffu, mbar_wait(bar_go + st * 8, go_ph, a.status, qt))) break;
            const uint32_t dst = s_ring + st * TILE + (lc >> 3) * HALF;
#pragma unroll 1
            for (int step = 0; step < QM / 16; ++step) {
                const int s = step * 16 >> me.seg_shift;
                if (slot0 + (step * 16 & (seg - 1)) >= external(me, s)) continue;      // nothing there: not used either
                const int mine = step < 4 ? (step < 2 ? node[0] : node[1]) : (step < 6 ? node[2] : node[3]);
#pragma unroll 4
                for (int i = 0; i < 16 / RPP; ++i) {
                    const int rr = i * RPP + lr, row = step * 16 + rr;
                    const int nd = __shfl_sync(0xffffffffu, mine, (step & 1) * 16 + rr);
                    cp_async16(dst + row * 128 + (((lc & 7) ^ (row & 7)) << 4), src + (nd < 0 ? 0 : nd) * row_stride, nd >= 0);
                }
            }
            cp_async_commit();
            cp_async_wait<0>();
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar_full + st * 8) : "memory");
            st += 2;
            if (st >= ring) st -= ring;
            turn += 2;
            if (turn >= ring) {
                turn -= ring;
                go_ph ^= 1u;
            }
        }
    } else {
        // ====== softmax: two groups of 128 threads, one thread per query row ======
        fence_after_sync();
        const uint32_t tmem = *tmem_slot;
        const int r = tid & 127, g = tid >> 7;            // my query row (TMEM lane r) and group
        const uint32_t lanes = uint32_t((warp & 3) * 32) << 16;
        const uint32_t tmem_s = tmem + g * 128 + lanes, tmem_o = tmem + 256 + g * D + lanes,
                       tmem_p = D == 128 ? tmem_s : tmem + 384 + g * 64 + lanes;
        const float c2 = a.scale_log2;
        float m_ref = -INFINITY, l = 0.f;                 // reference point of the exponent, row sum
        bool alive = true;

        // my node, its block in the query tile and row in the block: where its mask words are
        const QueryTile me = query(two ? g : 0);
        const int node = r & ((1 << pa.pack_shift) - 1), sub = node >> pa.bm_shift, jrow = node - sub * a.bm;
        const bool real = node < me.rows;
        const int seg = 1 << me.seg_shift;
        const uint32_t *own_words = reinterpret_cast<const uint32_t *>(blob + L.off_bmask) + (size_t(me.b0 + sub) * a.bm + jrow) * L.bw;
        const uint32_t *ext_words = reinterpret_cast<const uint32_t *>(blob + L.off_emask) + (size_t(me.b0 + sub) * a.bm + jrow) * L.maw;
        const int nt = nt_all, n_steps = (two ? 2 : 1) * nt;

        if (T1 > tp && real) {                            // on their way while the prefix is walked
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(own_words));
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(ext_words));
        }

        {
            uint32_t zero[16];                            // my row of O, while the first tiles are on their way
#pragma unroll
            for (int i = 0; i < 16; ++i) zero[i] = 0u;
#pragma unroll 1
            for (int c0 = 0; c0 < D; c0 += 16) tmem_st16(tmem_o + c0, zero);
        }
        int n = 0;                                        // tiles my group has taken
#pragma unroll 1
        for (int j = g; j < n_steps; j += 2, ++n) {
            const int tile = T0 + (two ? n : j);
            const bool full = (tile + 1) * KN <= prefix;
            uint32_t word[4];                             // columns of a masked tile that my row attends to
            if (tile < tp) {                              // the prefix's last tile may be partial
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int left = prefix - tile * KN - i * 32;
                    word[i] = left >= 32 ? 0xffffffffu : left > 0 ? (1u << left) - 1u : 0u;
                }
            } else {
                const bool own = tile == tp;
                const uint32_t *from = own ? own_words : ext_words;
                const int first = own ? 0 : (tile - tp - 1) << me.seg_shift >> 5, have = own ? L.bw : L.maw;
                const int at = (own ? sub * a.bm : sub << me.seg_shift) >> 5, nw = (own ? a.bm : seg) >> 5;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    word[i] = real && i >= at && i < at + nw && first + i - at < have ? __ldg(from + first + i - at) : 0u;
                // rows of my warp with a column in a step.  (S of my previous tile has landed, so the products of the one
                // before it, which read what is there, have been issued.)
                uint32_t *rows = reinterpret_cast<uint32_t *>(smem + G::OFF_ROWS) + ((n & 1) * 2 + g) * 32 + (warp & 3);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t lo = __ballot_sync(0xffffffffu, (word[i] & 0xffffu) != 0u), hi = __ballot_sync(0xffffffffu, word[i] > 0xffffu);
                    if (lane < 2) rows[(2 * i + lane) * 4] = lane == 0 ? lo : hi;
                }
            }
            // (S landing says that O += P V of my previous tile is done as well: it was issued before)
            alive = mbar_wait(bar_s + g * 8, n & 1, a.status, qt) && alive;
            fence_after_sync();
            uint32_t s[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(s[c], tmem_s + c * 32);
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld_wait(s[c]);
            if (!full) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if ((word[c] & (1u << i)) == 0u) s[c][i] = 0xff800000u;      // -inf
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};             // four independent chains
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int i = 0; i < 32; i += 2)
                    mx4[(i >> 1) & 3] = fmaxf(mx4[(i >> 1) & 3], fmaxf(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])));
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            // the reference moves when a row has outgrown it by more than 2^8 (always on the first live tile)
            const bool up = (mx - m_ref) * c2 > 8.f;      // true from -inf
            if (__any_sync(0xffffffffu, up)) {
                if (n > 0) {                              // rescale my row of O in tensor memory
                    const float alpha = up ? fast_exp2((m_ref - mx) * c2) : 1.f;
#pragma unroll 1
                    for (int c0 = 0; c0 < D; c0 += 8) {
                        uint32_t o[8];
                        tmem_ld8(o, tmem_o + c0);
#pragma unroll
                        for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st8(tmem_o + c0, o);
                    }
                    l *= alpha;
                }
                if (up) m_ref = mx;
            }
            const float mu = m_ref == -INFINITY ? 0.f : m_ref * c2;
            const uint64_t scale2 = pair(c2, c2), shift2 = pair(-mu, -mu);
            uint64_t l2[2] = {0, 0};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t packed[16];
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const uint64_t x = fma2(pair(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), scale2, shift2);
                    float p0, p1;
                    unpair(x, p0, p1);
                    p0 = fast_exp2(p0);
                    p1 = fast_exp2(p1);
                    l2[(i >> 1) & 1] = add2(l2[(i >> 1) & 1], pair(p0, p1));
                    packed[i >> 1] = MT::pack(p0, p1);
                }
                tmem_st16(tmem_p + c * 16, packed);
                if (c & 1) {                              // half of P: its products may begin
                    tmem_st_wait();
                    fence_before_sync();
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar_p + (c >> 1) * 16 + g * 8) : "memory");
                }
            }
            float la, lb;
            unpair(add2(l2[0], l2[1]), la, lb);
            l += la + lb;
        }

        // ---- rows of O, unnormalised, and their (exponent, sum) into shared memory, once every product of either
        // group is done with the operands there; 16-byte chunks swizzled.  Two groups with one query tile
        // merge here: either reads both accumulators, for every other 32 columns.
        if (n > 0) alive = mbar_wait(bar_o + g * 8, 0, a.status, qt) && alive;
        fence_after_sync();
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        float2 *stats = reinterpret_cast<float2 *>(smem + G::OFF_STATS);
        stats[tid] = make_float2(n > 0 && alive && m_ref != -INFINITY ? m_ref * c2 : -INFINITY, l);
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        const float2 st0 = stats[two ? tid : r], st1 = two ? make_float2(-INFINITY, 0.f) : stats[QM + r];
        const float mu = fmaxf(st0.x, st1.x);
        const float w0 = st0.x == -INFINITY ? 0.f : fast_exp2(st0.x - mu), w1 = st1.x == -INFINITY ? 0.f : fast_exp2(st1.x - mu);
        if (two || g == 0) stats[2 * QM + tid] = make_float2(mu, st0.y * w0 + st1.y * w1);
        float *srow = reinterpret_cast<float *>(smem) + (two ? tid : r) * D;
        const uint32_t tmem_first = two ? tmem_o : tmem + 256 + lanes;
#pragma unroll 1
        for (int c0 = two ? 0 : g * 32; c0 < D; c0 += two ? 32 : 64) {
            uint32_t o[32], o1[32];
            tmem_ld32(o, tmem_first + c0);
            if (!two) tmem_ld32(o1, tmem_first + D + c0);
            tmem_ld_wait(o);
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = w0 == 0.f ? 0u : __float_as_uint(__uint_as_float(o[i]) * w0);   // without a column: never written
            if (!two) {
                tmem_ld_wait(o1);
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (w1 != 0.f) o[i] = __float_as_uint(fmaf(__uint_as_float(o1[i]), w1, __uint_as_float(o[i])));
            }
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const int chunk = (c0 + i) >> 2;
                *reinterpret_cast<uint4 *>(srow + ((chunk ^ (r & 7)) << 2)) = make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
            }
        }
    }

    // ---- merge: a row lies in every CTA of the cluster.  Every CTA takes an equal share of the rows.  Shared memory of
    // another CTA reads at some 12 bytes per cycle, which is why prefix_plan prefers few runs.
    const QueryTile tile_a = query(0), tile_b = query(two);
    fence_before_sync();
    __syncwarp();
    if (pa.cluster > 1) cluster_sync();
    else __syncthreads();
    if (warp == 9) {
        fence_after_sync();
        tmem_free_all(*tmem_slot);
    }
    const int rows_all = two ? 2 * QM : QM, share = (rows_all + pa.cluster - 1) / pa.cluster;
    const bool partial = pa.cluster < pa.n_runs;          // rows in fp32 for the merge kernel, slot by slot
    const int row_lo = partial ? 0 : run * share, row_hi = min(rows_all, row_lo + share);
    // a lane has a 64-byte piece of a row: four chunks of 16 bytes, LPR lanes a row
    constexpr int LPR = D / 16, RPW = 32 / LPR;
    const int c = lane % LPR;
#pragma unroll 1
    for (int row = row_lo + warp * RPW + lane / LPR; row < row_hi; row += PFX_THREADS / 32 * RPW) {
        float4 acc[4] = {};
        float mu = -INFINITY, l = 0.f;
#pragma unroll 1
        for (int s = 0; s < pa.cluster; ++s) {
            const uint32_t base = cluster_addr(s_base, s);
            const float2 st = cluster_ld2(base + G::OFF_STATS + (2 * QM + row) * 8);
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = cluster_ld4(base + row * D * 4 + (((k * LPR + c) ^ (row & 7)) << 4));
            const float top = fmaxf(mu, st.x), to = top == -INFINITY ? 0.f : top;
            const float w_old = fast_exp2(mu - to), w = fast_exp2(st.x - to);
            mu = top;
            l = l * w_old + st.y * w;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc[k].x = acc[k].x * w_old + v[k].x * w;
                acc[k].y = acc[k].y * w_old + v[k].y * w;
                acc[k].z = acc[k].z * w_old + v[k].z * w;
                acc[k].w = acc[k].w * w_old + v[k].w * w;
            }
        }
        const bool first = row < QM;
        const int node = row & ((1 << pa.pack_shift) - 1), gr = (first ? tile_a.q0 : tile_b.q0) + node;
        const int h = (first ? tile_a.h : tile_b.h) + ((row & 127) >> pa.pack_shift);
        if (node >= (first ? tile_a.rows : tile_b.rows)) continue;
        const float inv = l == 0.f ? 0.f : 1.f / l;       // (a NaN stays one: no maximum shows it, but the sum does)
        const float lse = l == 0.f ? -INFINITY : mu + log2f(l);
        if (partial) {
            const size_t slot_row = ((size_t(run) * a.Z + z) * a.H + h) * n_q + gr;
            float4 *to = reinterpret_cast<float4 *>(a.part_o + slot_row * D);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                to[k * LPR + c] = make_float4(acc[k].x * inv, acc[k].y * inv, acc[k].z * inv, acc[k].w * inv);
            if (c == 0) a.part_lse[slot_row] = lse;
            continue;
        }
        uint2 *to = reinterpret_cast<uint2 *>(static_cast<T *>(a.o) + z * a.os_z + h * a.os_h + gr * a.os_n);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            to[k * LPR + c] = make_uint2(MT::pack(acc[k].x * inv, acc[k].y * inv), MT::pack(acc[k].z * inv, acc[k].w * inv));
        if (a.lse != nullptr && c == 0) a.lse[(size_t(z) * a.H + h) * n_q + gr] = lse;
    }
    if (pa.cluster == 1) return;
    __syncwarp();
    cluster_sync();                                       // nobody leaves while its rows are being read
}

// rank-4 map over a page pool (columns, rows of a page, K/V heads, pages) with 64-column x page boxes
static bool make_map_pool(CUtensorMap *map, bool bf16, int D, const PagedArgs &pg, int H_kv, const void *pool) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[4] = {cuuint64_t(D), cuuint64_t(pg.page_size), cuuint64_t(H_kv), cuuint64_t(pg.n_pages)};
    const cuuint64_t strides[3] = {cuuint64_t(pg.stride_row) * 2, cuuint64_t(pg.stride_head) * 2,
                                   cuuint64_t(pg.stride_page) * 2};
    const cuuint32_t box[4] = {64, cuuint32_t(pg.page_size), 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
              const_cast<void *>(pool), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename T, int D, bool PAGED>
static cudaError_t launch_prefix_t(const AttnArgs &a, const PagedArgs *pg, int n_runs, cudaStream_t stream) {
    constexpr bool bf16 = !std::is_same<T, __half>::value;
    const int H_kv = a.H / a.kv_group;
    alignas(64) CUtensorMap tq, tk, tv, tkt, tvt;
    const int pack = prefix_heads_per_tile(a.H, H_kv, a.n_q);
    if (!make_map(&tq, a.q, bf16, D, a.n_q, a.H, a.Z, a.qs_n, a.qs_h, a.qs_z, umma::QM / pack) ||
        !make_map(&tkt, a.k, bf16, D, a.n_kv, H_kv, a.Z, a.ks_n, a.ks_h, a.ks_z, umma::KN) ||
        !make_map(&tvt, a.v, bf16, D, a.n_kv, H_kv, a.Z, a.vs_n, a.vs_h, a.vs_z, umma::KN))
        return cudaErrorNotSupported;
    if (!PAGED) {
        tk = tkt;
        tv = tvt;
    } else if (!make_map_pool(&tk, bf16, D, *pg, H_kv, pg->k_pool) || !make_map_pool(&tv, bf16, D, *pg, H_kv, pg->v_pool)) {
        return cudaErrorNotSupported;
    }
    static DeviceOnce configured;
    const cudaError_t ce = configured.run([&] {
        return cudaFuncSetAttribute(prefix_umma_kernel<T, D, PAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    umma::Geo<D>::SMEM_BYTES);
    });
    if (ce != cudaSuccess) return ce;
    if ((long long)a.Z * n_runs > 65535) return cudaErrorInvalidValue;
    const PrefixPlan plan = prefix_plan(a.Z, a.H, H_kv, a.n_q, a.prefix, sm_count(), a.part_o != nullptr, n_runs, PAGED ? pg->page_size : 128);
    PrefixArgs pa = {};
    pa.n_runs = plan.runs;
    pa.cluster = plan.spread ? 1 : plan.runs;
    pa.pair = plan.pair;
    pa.q_tiles = (a.n_q + umma::QM - 1) / umma::QM;
    pa.kv_tiles = a.kv_group / pack * pa.q_tiles;
    pa.bm_shift = a.bm == 32 ? 5 : a.bm == 64 ? 6 : 7;
    pa.pack = pack;
    pa.pack_shift = 7;
    for (int p = pack; p > 1; p /= 2) --pa.pack_shift;
    if (PAGED) {
        pa.block_table = pg->block_table;
        pa.prefix_lens = pg->prefix_lens;
        pa.table_stride = pg->table_stride;
        pa.page_size = pg->page_size;
        pa.n_pages = pg->n_pages;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pa.pair ? (pa.kv_tiles + 1) / 2 : pa.kv_tiles, H_kv, a.Z * pa.n_runs);
    cfg.blockDim = dim3(PFX_THREADS);
    cfg.dynamicSmemBytes = umma::Geo<D>::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = unsigned(pa.cluster);
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, prefix_umma_kernel<T, D, PAGED>, a, pa, tq, tk, tv, tkt, tvt);
    if (e != cudaSuccess || !plan.spread) return e;
    AttnArgs merge = a;
    merge.part_slots = pa.n_runs;
    return launch_combine(merge, bf16 ? FST_BF16 : FST_F16, stream);
}

template <bool PAGED>
static cudaError_t launch_prefix_any(const AttnArgs &a, const PagedArgs *pg, int dtype, int n_runs, cudaStream_t stream) {
    if ((a.D != 64 && a.D != 128) || a.prefix <= 0 || n_runs < 1 || a.bm < 32) return cudaErrorNotSupported;
    if (dtype == FST_F16)
        return a.D == 128 ? launch_prefix_t<__half, 128, PAGED>(a, pg, n_runs, stream)
                          : launch_prefix_t<__half, 64, PAGED>(a, pg, n_runs, stream);
    if (dtype == FST_BF16)
        return a.D == 128 ? launch_prefix_t<__nv_bfloat16, 128, PAGED>(a, pg, n_runs, stream)
                          : launch_prefix_t<__nv_bfloat16, 64, PAGED>(a, pg, n_runs, stream);
    return cudaErrorNotSupported;
}

// The whole call - prefix and tree - in n_runs runs of column tiles (without room for partial results, part_o, at most
// kMaxClusterRuns).
cudaError_t launch_prefix_umma(const AttnArgs &a, int dtype, int n_runs, cudaStream_t stream) {
    return launch_prefix_any<false>(a, nullptr, dtype, n_runs, stream);
}

// The same with the prefix rows in a page pool; a.k / a.v hold the tree's rows only.
cudaError_t launch_prefix_umma_paged(const AttnArgs &a, const PagedArgs &pg, int dtype, int n_runs, cudaStream_t stream) {
    if (pg.page_size != 16 && pg.page_size != 32 && pg.page_size != 64 && pg.page_size != 128)
        return cudaErrorNotSupported;
    return launch_prefix_any<true>(a, &pg, dtype, n_runs, stream);
}

}  // namespace fst
