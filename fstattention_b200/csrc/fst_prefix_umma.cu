// Attention behind a shared prefix on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// The prefix part of the reference kernel (fstattention.py:113-136) is plain dense attention: every query
// row attends to every prefix row.  One CTA per (128 query rows, head, batch element, run of column tiles);
// the column tiles of a query tile are the prefix in 128-row tiles, then the tree: one tile with the
// query tile's own K/V rows and, behind it, tiles of gathered ancestors, in which every block of the query tile has
// a segment of columns.  Tree tiles are masked by the rows' mask words and cost what a prefix tile costs;
// run beside this kernel as a launch of its own on a second stream, the tree part took a fork, a join, a
// further partial result and, at small sizes, most of the call.  Per tile t
//     S(t) = Q K(t)^T       tcgen05.mma  M=128 N=128 K=16 x D/16, both operands K-major in shared memory
//     P(t) = softmax part   one thread per query row (TMEM lane = row, so no shuffles): tcgen05.ld
//                           of S, probabilities against a lazily moved reference point, P written
//                           to shared memory in the 128-byte-swizzled K-major layout
//     O_g += P(t) V(t)      tcgen05.mma  A = P, B = V (MN-major: rows of V are the K index)
// Tensor memory holds two S buffers and two accumulators O_0, O_1 (4 x 128 columns).  K/V tiles
// arrive by TMA (128-row x 64-column boxes, 128-byte swizzle; gathered rows by cp.async into the same
// layout) into two stages each.  Head dimension D is 64 or 128: one or two 64-column halves per Q / K / V tile.
//
// Twelve warps.  Warps 0-3 and 4-7 are two softmax groups; group g takes the tiles with t & 1 == g
// and keeps its own reference point, row sums, P buffer and accumulator O_g, so the groups never
// wait for one another and one group's barrier waits and tensor-memory latencies hide behind the
// other's exponentials.  Warp 8 loads K and its lane 0 issues S(t); warp 9 loads V and its lane 0
// issues O_g += P V; warps 10 and 11 gather the K and the V rows of ancestors when 8 and 9 say that their stage is
// free.  All hand-offs are mbarriers (TMA completion, tcgen05.commit, or arrivals by
// the 128 threads of a group); every barrier indexed by t & 1 completes once per two tiles, so a
// waiter can never fall two phases behind.  At the end the groups' results are merged through
// shared memory and written: as the output itself when there is one run, else as one partial result per
// run (normalised rows in fp32 plus base-2 log-sum-exp) that combine_splits_kernel merges.
//
// With grouped-query attention a small tree's rows of several heads share a query tile (see
// prefix_heads_per_tile): the tile is loaded as one box per head and its rows go to their heads at the end.
//
// PAGED = true reads the prefix rows from a page pool through a block table (a KV cache): a
// tile is 128 / page_size pages and lane j of the loading warp requests page j.
//
// Every wait is bounded in time (mbar_wait): on expiry the kernel records FST_DEV_TIMEOUT, stops
// issuing, frees its tensor memory and returns.

#include "fst_plan.h"
#include "fst_umma.cuh"

namespace fst {

namespace umma {

constexpr int QM = 128;                // query rows per CTA (MMA M)
constexpr int KN = 128;                // K/V rows per tile (MMA N of the first product)
constexpr int TILE_P = 2 * HALF;       // bytes of a P tile (128 x 128 fp16)

// Shared-memory map for head dimension D (64 or 128): a Q / K / V tile is 128 rows of D columns,
// D / 64 halves.  Q | P x 2 (double buffered) | K x 2 stages | V x 2 stages | barriers.
template <int D>
struct Geo {
    static constexpr int TILE = (D / 64) * HALF;
    static constexpr int OFF_Q = 0;
    static constexpr int OFF_P = OFF_Q + TILE;
    static constexpr int OFF_K = OFF_P + 2 * TILE_P;
    static constexpr int OFF_V = OFF_K + 2 * TILE;
    static constexpr int OFF_BAR = OFF_V + 2 * TILE;
    static constexpr int SMEM_BYTES = OFF_BAR + 160 + 1024;   // + barriers, TMEM address, 1 KB alignment slack
};

}  // namespace umma

// Arguments of the prefix kernel beyond AttnArgs.
struct PrefixArgs {
    int n_runs;          // runs of column tiles (CTAs per query tile, head, batch element)
    // paged prefix: K/V rows live in pages of page_size rows; block_table[z][i] is the page
    // holding rows [i * page_size, (i + 1) * page_size) of batch element z, prefix_lens[z] its
    // number of prefix rows (AttnArgs::prefix is then the largest of them)
    const int32_t *block_table;
    const int32_t *prefix_lens;
    int table_stride, page_size, n_pages;
    int pack, pack_shift;                // heads per query tile; a head's rows are 1 << pack_shift of the tile's
};

constexpr int PFX_SOFTMAX = 256;       // eight softmax warps: two groups of 128, one thread per query row each
constexpr int PFX_THREADS = PFX_SOFTMAX + 128;  // + two issuing and two gathering warps

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
    constexpr int TILE = G::TILE, OFF_Q = G::OFF_Q, OFF_P = G::OFF_P, OFF_K = G::OFF_K, OFF_V = G::OFF_V,
                  OFF_BAR = G::OFF_BAR;

    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");   // the merge kernel may take its place
    extern __shared__ unsigned char smem_raw[];
    const uint32_t s_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *smem = smem_raw + (s_base - smem_u32(smem_raw));
    const int qt = blockIdx.x, h = blockIdx.y * pa.pack, hk = h / a.kv_group;   // query tile, (first) head, K/V head
    const int z = blockIdx.z / pa.n_runs, run = blockIdx.z - z * pa.n_runs;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int n_q = a.n_q;
    // prefix rows of my batch element (paged: every batch element has its own count)
    const int prefix = PAGED ? max(0, min(__ldg(pa.prefix_lens + z), a.prefix)) : a.prefix;

    const int lane = tid & 31;

    // The query tile's nodes [q0, q0 + rows_t) in blocks b0 .. b0 + n_blk - 1, every block with a segment of
    // seg columns in a gathered tile.  external(s): ancestors of block s outside it.
    const int q0 = qt * QM, rows_t = min(n_q - q0, 1 << pa.pack_shift), b0 = q0 / a.bm, n_blk = (rows_t + a.bm - 1) / a.bm;
    const int seg_shift = n_blk > 2 ? 5 : n_blk > 1 ? 6 : 7, seg = 1 << seg_shift;
    const PackedLayout L = packed_layout(a.nb, a.bm, a.ma);
    const unsigned char *blob = a.packed + size_t(z) * a.meta_stride;
    auto external = [&](int s) -> int {
        return s < n_blk ? min(max(__ldg(reinterpret_cast<const int32_t *>(blob + L.off_count) + b0 + s), 0), a.ma) : 0;
    };
    int longest = max(max(external(0), external(1)), max(external(2), external(3)));
    // My run of column tiles [T0, T0 + nt): tp prefix tiles, the own tile, gathered tiles.  The runs are cut as if
    // there were one gathered tile, so that no CTA waits for the counts before its first loads; nt_sure
    // tiles of the run are there whatever they say.
    const int tp = (prefix + KN - 1) / KN, per = (tp + 2 + pa.n_runs - 1) / pa.n_runs;
    const int T0 = run * per, T1 = run + 1 == pa.n_runs ? 0x7fffffff : T0 + per;
    const int nt_sure = max(0, min(T1, tp + 1) - T0);

    // barriers: Q, K[2], V[2] (TMA), S[2] (S product landed in its buffer), O[2] (O += P V done, per P buffer),
    // P[2] (all softmax threads are through with S(t) and have written P(t)).  Every barrier that is
    // indexed by t & 1 completes once per two tiles, so a waiter can never fall two phases behind.
    const uint32_t bar_q = s_base + OFF_BAR, bar_k = bar_q + 8, bar_v = bar_q + 24, bar_s = bar_q + 40,
                   bar_o = bar_q + 56, bar_p = bar_q + 72, bar_go = bar_q + 88;   // go[K][2], go[V][2]: a gathered tile's stage is free
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + OFF_BAR + 144);

    // Loads are issued by whole warps (8: K, 9: V).  Contiguous prefix: lane 0 requests the two
    // boxes of a tile.  Paged: a tile is KN / page_size pages, one pair of boxes each, and lane j
    // takes page j - it reads that page's number from the block table (my_page) a tile before
    // it requests the boxes, so the table's latency is off the path, and a single thread is
    // not left to issue sixteen copies one after the other.  Pages past the end of my batch
    // element's prefix repeat its last page: finite values under columns the softmax masks.
    const int ps = PAGED ? pa.page_size : KN, npt = KN / ps;
    const int32_t *table = PAGED ? pa.block_table + size_t(z) * pa.table_stride : nullptr;
    const int last_page = PAGED ? max(prefix - 1, 0) / ps : 0;
    auto my_page = [&](int t) -> int {
        if (!PAGED || lane >= npt) return 0;
        return __ldg(table + min((T0 + t) * KN / ps + lane, last_page));
    };
    auto warp_load = [&](uint32_t dst, const CUtensorMap *map, const CUtensorMap *map_tree, uint32_t bar, uint32_t go, int t, int page) {
        const int tile = T0 + t;
        if (tile > tp) {                                     // gathered: the gathering warp's turn
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(go) : "memory");
            return;
        }
        if (lane == 0) mbar_arrive_expect_tx(bar, TILE);
        if (tile == tp) {                                 // the query tile's own rows
            if (lane == 0) {
#pragma unroll
                for (int hf = 0; hf < DH; ++hf)
                    tma_load_4d(dst + hf * HALF, map_tree, hf * 64, (PAGED ? 0 : a.prefix) + q0, hk, z, bar);
            }
            return;
        }
        if (PAGED) __syncwarp();                          // (contiguous: only lane 0 ever comes here)
        if (PAGED) {
            if (lane < npt) {
                if (unsigned(page) >= unsigned(pa.n_pages))       // the boxes then read as zeros
                    report(a.status, FST_DEV_INDEX_RANGE, z, tile * KN / ps + lane);
#pragma unroll
                for (int hf = 0; hf < DH; ++hf)
                    tma_load_4d(dst + lane * ps * 128 + hf * HALF, map, hf * 64, 0, hk, page, bar);
            }
        } else if (lane == 0) {
#pragma unroll
            for (int hf = 0; hf < DH; ++hf) tma_load_4d(dst + hf * HALF, map, hf * 64, tile * KN, hk, z, bar);
        }
    };
    auto load_q = [&]() {
        if (lane != 0) return;
        mbar_arrive_expect_tx(bar_q, TILE);
        for (int i = 0; i < pa.pack; ++i)
#pragma unroll
            for (int hf = 0; hf < DH; ++hf)
                tma_load_4d(s_base + OFF_Q + hf * HALF + (i << pa.pack_shift) * 128, &tm_q, hf * 64, q0, h + i, z, bar_q);
    };
    auto load_k = [&](int t, int page) {
        warp_load(s_base + OFF_K + (t & 1) * TILE, &tm_k, &tm_kt, bar_k + (t & 1) * 8, bar_go + (t & 1) * 8, t, page);
    };
    auto load_v = [&](int t, int page) {
        warp_load(s_base + OFF_V + (t & 1) * TILE, &tm_v, &tm_vt, bar_v + (t & 1) * 8, bar_go + 16 + (t & 1) * 8, t, page);
    };
    // Warp 8 sets the barriers up and sends the first loads off before the CTA-wide sync, so that
    // they are under way while warp 9 allocates tensor memory.
    if (warp == 8) {
        if (lane == 0) {
            mbar_init(bar_q, 1);
            for (int i = 0; i < 2; ++i) {
                mbar_init(bar_k + i * 8, 1);
                mbar_init(bar_v + i * 8, 1);
                mbar_init(bar_s + i * 8, 1);
                mbar_init(bar_o + i * 8, 1);
                mbar_init(bar_p + i * 8, PFX_SOFTMAX / 2);
                mbar_init(bar_go + i * 8, 1);
                mbar_init(bar_go + 16 + i * 8, 1);
            }
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        __syncwarp();
        if (PAGED || lane == 0) {
            if (nt_sure > 0) load_q();
            const int page0 = T0 < tp ? my_page(0) : 0, page1 = T0 + 1 < tp ? my_page(1) : 0;
            if (nt_sure > 0) {
                load_k(0, page0);
                load_v(0, page0);
            }
            if (nt_sure > 1) {
                load_k(1, page1);
                load_v(1, page1);
            }
        }
    }
    if (warp == 9) {                                      // tensor memory: two S buffers and two accumulators, 128 columns each
        umma::tmem_alloc_all(smem_u32(tmem_slot));
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_s0 = tmem_base, tmem_o = tmem_base + 256;   // S(t) at tmem_s0 + (t & 1) * 128, O_g at tmem_o + g * 128

    const int nt = max(0, min(T1, tp + 1 + ((longest + seg - 1) >> seg_shift)) - T0);

    if (warp >= 10) {
        // ====== two gathering warps: ancestors' K rows (10) and V rows (11), whole steps of 16 rows at a time ======
        const T *src = warp == 10 ? static_cast<const T *>(a.k) + z * a.ks_z + hk * a.ks_h
                                  : static_cast<const T *>(a.v) + z * a.vs_z + hk * a.vs_h;
        const int64_t row_stride = warp == 10 ? a.ks_n : a.vs_n;
        constexpr int CH = D / 8, RPP = 32 / CH;          // 16-byte chunks per row, rows per pass of the warp
        const int lr = lane / CH, lc = lane % CH;
        src += (PAGED ? 0 : a.prefix) * row_stride + lc * 8;
        uint32_t turn = 0;                                // parity of the next hand-over of each stage
#pragma unroll 1
        for (int t = max(0, tp + 1 - T0); t < nt; ++t) {
            const int st = t & 1, slot0 = (T0 + t - tp - 1) << seg_shift;
            // a step's rows: lanes 0-15 those of an even step, lanes 16-31 those of the odd one behind it
            int node[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int row = k * 32 + lane, s = row >> seg_shift, slot = slot0 + (row & (seg - 1));
                node[k] = -1;
                if (s < n_blk && slot < external(s)) {
                    node[k] = __ldg(reinterpret_cast<const int32_t *>(blob + L.off_idx) + size_t(b0 + s) * a.ma + slot);
                    if (node[k] >= n_q) {
                        report(a.status, FST_DEV_INDEX_RANGE, b0 + s, slot);
                        node[k] = -1;
                    }
                }
            }
            const uint32_t go = bar_go + (warp == 10 ? 0 : 16) + st * 8;
            if (!__all_sync(0xffffffffu, mbar_wait(go, (turn >> st) & 1, a.status, qt))) break;
            turn ^= 1u << st;
            const uint32_t dst = s_base + (warp == 10 ? OFF_K : OFF_V) + st * TILE + (lc >> 3) * HALF;
#pragma unroll 1
            for (int step = 0; step < QM / 16; ++step) {
                const int s = step * 16 >> seg_shift;
                if (slot0 + (step * 16 & (seg - 1)) >= external(s)) continue;      // nothing there: not used either
                const int mine = step < 4 ? (step < 2 ? node[0] : node[1]) : (step < 6 ? node[2] : node[3]);
#pragma unroll
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
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"((warp == 10 ? bar_k : bar_v) + st * 8) : "memory");
        }
    } else if (warp >= 8) {
        // ====== two issuing warps: 8 loads K and issues S = Q K^T, 9 loads V and issues O += P V ======
        // Lane 0 waits and issues the products; the whole warp takes part in the loads.
        const uint32_t idesc_s = instr_desc(BF16, false, KN), idesc_pv = instr_desc(BF16, true, D);
        bool alive = true;
        if (warp == 8 && nt > 0 && (PAGED || lane == 0)) {     // contiguous: lane 0 alone
            // descriptors of the tiles' first 16-wide step; a step further on adds its byte offset / 16
            const uint64_t dq = smem_desc(s_base + OFF_Q, 16), dk = smem_desc(s_base + OFF_K, 16);
            int page = T0 + 2 < tp ? my_page(2) : 0;      // my page of the tile to be requested next
            if (nt_sure == 0) load_q();
            for (int t = nt_sure; t < min(nt, 2); ++t) load_k(t, 0);
            if (lane == 0) alive = mbar_wait(bar_q, 0, a.status, qt) && alive;
#pragma unroll 1
            for (int t = 0; t < nt; ++t) {                // S(t) = Q K(t)^T into S buffer t & 1
                const int st = t & 1;
                if (lane == 0 && alive) {
                    // the buffer is free when the softmax warps are through with tile t-2
                    if (t > 1) alive = mbar_wait(bar_p + st * 8, ((t >> 1) - 1) & 1, a.status, qt) && alive;
                    alive = mbar_wait(bar_k + st * 8, (t >> 1) & 1, a.status, qt) && alive;
                    if (alive) {
                        umma::fence_after_sync();
                        const uint64_t dks = dk + uint64_t(st * (TILE >> 4));
#pragma unroll
                        for (int ks = 0; ks < D / 16; ++ks) {
                            const uint64_t koff = ((ks >> 2) * HALF + (ks & 3) * 32) >> 4;
                            mma_f16(tmem_s0 + st * 128, dq + koff, dks + koff, idesc_s, ks > 0);
                        }
                        mma_commit(bar_s + st * 8);
                        // K stage st is free as soon as S(t) has been formed
                        if (t + 2 < nt) alive = mbar_wait(bar_s + st * 8, (t >> 1) & 1, a.status, qt) && alive;
                    }
                }
                if (PAGED) alive = __shfl_sync(0xffffffffu, alive, 0);
                if (!alive) break;
                if (t + 2 < nt) {
                    load_k(t + 2, page);
                    if (T0 + t + 3 < tp) page = my_page(t + 3);
                }
            }
        } else if (warp == 9 && nt > 0 && (PAGED || lane == 0)) {
            const uint64_t dp = smem_desc(s_base + OFF_P, 16), dv = smem_desc(s_base + OFF_V, HALF);
            int page = T0 + 2 < tp ? my_page(2) : 0;
            for (int t = nt_sure; t < min(nt, 2); ++t) load_v(t, 0);
            const int ext[4] = {external(0), external(1), external(2), external(3)};
#pragma unroll 1
            for (int t = 0; t < nt; ++t) {                // O_g += P(t) V(t), g = t & 1
                const int st = t & 1;
                if (lane == 0 && alive) {
                    alive = mbar_wait(bar_p + st * 8, (t >> 1) & 1, a.status, qt) && alive;   // P(t) is in shared memory
                    alive = mbar_wait(bar_v + st * 8, (t >> 1) & 1, a.status, qt) && alive;
                    if (alive) {
                        umma::fence_after_sync();
                        // rows of a gathered tile past the lists' ends were never fetched
                        uint32_t live = 0xffu;
                        if (T0 + t > tp) {
                            const int slot0 = (T0 + t - tp - 1) << seg_shift;
                            live = 0u;
#pragma unroll
                            for (int s = 0; s < 4; ++s) {
                                const int left = min(ext[s] - slot0, seg), steps = left > 0 ? (left + 15) >> 4 : 0;
                                live |= ((1u << steps) - 1u) << (s << seg_shift >> 4);
                            }
                        }
                        bool more = t > 1;
                        const uint64_t dps = dp + uint64_t(st * (TILE_P >> 4)), dvs = dv + uint64_t(st * (TILE >> 4));
#pragma unroll
                        for (int ks = 0; ks < KN / 16; ++ks) {    // 16 prefix rows per step
                            const uint64_t aoff = ((ks >> 2) * HALF + (ks & 3) * 32) >> 4;
                            if (!((live >> ks) & 1u)) continue;
                            mma_f16(tmem_o + st * 128, dps + aoff, dvs + uint64_t((ks * 16 * 128) >> 4), idesc_pv, more);
                            more = true;
                        }
                        mma_commit(bar_o + st * 8);
                        // V stage st is free once that product has read it
                        if (t + 2 < nt) alive = mbar_wait(bar_o + st * 8, (t >> 1) & 1, a.status, qt) && alive;
                    }
                }
                if (PAGED) alive = __shfl_sync(0xffffffffu, alive, 0);
                if (!alive) break;
                if (t + 2 < nt) {
                    load_v(t + 2, page);
                    if (T0 + t + 3 < tp) page = my_page(t + 3);
                }
            }
        }
    } else {
        // ============ softmax: two groups of 128 threads, one thread per query row, alternating tiles ============
        // Group g owns the tiles with t & 1 == g: S buffer g, P buffer g and the accumulator O_g,
        // with its own reference point and row sum, so the groups never wait for one another and
        // one group's waits and tensor-memory latencies hide behind the other's exponentials.
        const int r = tid & 127, g = tid >> 7;            // my query row (TMEM lane r) and group
        const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
        const uint32_t tmem_s = tmem_s0 + g * 128, tmem_og = tmem_o + g * 128;
        unsigned char *prow = smem + OFF_P + g * TILE_P + r * 128; // my row of P buffer g
        const float c2 = a.scale_log2;
        float m_ref = -INFINITY, l = 0.f;                 // reference point of the exponent, row sum
        bool alive = true;
        float mx = -INFINITY, l_tile = 0.f, mu = 0.f;     // results / parameter of a sweep

        // my node, its block in the query tile and row in the block: where its mask words are
        const int node = r & ((1 << pa.pack_shift) - 1), sub = node / a.bm, j = node - sub * a.bm;
        const bool real = node < rows_t;
        const uint32_t *own_words = reinterpret_cast<const uint32_t *>(blob + L.off_bmask) + (size_t(b0 + sub) * a.bm + j) * L.bw;
        const uint32_t *ext_words = reinterpret_cast<const uint32_t *>(blob + L.off_emask) + (size_t(b0 + sub) * a.bm + j) * L.maw;
        uint32_t word[4];                                 // columns of a masked tile that my row attends to
        auto tile_words = [&](int tile) {
            if (tile < tp) {                                 // the prefix's last, partial tile
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int left = prefix - tile * KN - i * 32;
                    word[i] = left >= 32 ? 0xffffffffu : left > 0 ? (1u << left) - 1u : 0u;
                }
                return;
            }
            const uint32_t *from = tile == tp ? own_words : ext_words;
            const int first = tile == tp ? 0 : (tile - tp - 1) << seg_shift >> 5, have = tile == tp ? L.bw : L.maw;
            const int at = (tile == tp ? sub * a.bm : sub << seg_shift) >> 5, n = (tile == tp ? a.bm : seg) >> 5;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                word[i] = real && i >= at && i < at + n && first + i - at < have ? __ldg(from + first + i - at) : 0u;
        };

        // One sweep over my row of S: row maximum, and (WRITE) probabilities against the reference
        // point into my row of P plus their sum.  MASK: columns without a bit in word are -inf.  S is read 32
        // columns at a time, the next load in flight while the current one is processed.
        auto sweep = [&](auto write_c, auto mask_c) {
            constexpr bool WRITE = decltype(write_c)::value, MASK = decltype(mask_c)::value;
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, l4[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t ra[32], rb[32];
            tmem_ld32(ra, tmem_s + lane_base);
            tmem_ld_wait(ra);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t (&cur)[32] = (c & 1) ? rb : ra;
                uint32_t (&nxt)[32] = (c & 1) ? ra : rb;
                if (c < 3) tmem_ld32(nxt, tmem_s + lane_base + (c + 1) * 32);
                uint32_t packed[16];
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    float s0 = __uint_as_float(cur[i]), s1 = __uint_as_float(cur[i + 1]);
                    if (MASK) {
                        s0 = (word[c] & (1u << i)) != 0u ? s0 : -INFINITY;
                        s1 = (word[c] & (2u << i)) != 0u ? s1 : -INFINITY;
                    }
                    mx4[(i >> 1) & 3] = fmaxf(mx4[(i >> 1) & 3], fmaxf(s0, s1));   // four independent chains
                    if (WRITE) {
                        const float p0 = fast_exp2(fmaf(s0, c2, -mu)), p1 = fast_exp2(fmaf(s1, c2, -mu));
                        l4[(i >> 1) & 3] += p0 + p1;
                        packed[i >> 1] = MT::pack(p0, p1);
                    }
                }
                if (WRITE) {
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {      // four 16-byte chunks of my row, swizzled
                        const int chunk = c * 4 + q4;
                        *reinterpret_cast<uint4 *>(prow + (chunk >> 3) * HALF + (((chunk & 7) ^ (r & 7)) << 4)) =
                            make_uint4(packed[q4 * 4], packed[q4 * 4 + 1], packed[q4 * 4 + 2], packed[q4 * 4 + 3]);
                    }
                }
                if (c < 3) tmem_ld_wait(nxt);
            }
            mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            l_tile = (l4[0] + l4[1]) + (l4[2] + l4[3]);
        };
        const std::true_type yes{};
        const std::false_type no{};

        int n_mine = 0;                                   // tiles my group has taken
#pragma unroll 1
        for (int t = g; t < nt; t += 2, ++n_mine) {
            const bool full = (T0 + t + 1) * KN <= prefix;
            if (!full) tile_words(T0 + t);
            alive = mbar_wait(bar_s + g * 8, n_mine & 1, a.status, qt) && alive;
            // P buffer g and O_g belong to the tensor core until O_g += P V of my previous tile is done
            if (n_mine > 0) alive = mbar_wait(bar_o + g * 8, (n_mine - 1) & 1, a.status, qt) && alive;
            umma::fence_after_sync();

            // Probabilities are formed against the current reference point while the row maximum
            // is tracked (one pass over S).  Only if a row of my warp has outgrown its reference
            // by more than 2^8 (always on the first tile) is the reference moved, O_g rescaled,
            // and the tile done again.
            if (n_mine == 0) {
                // first tile: the maximum of the first 32 columns is reference enough to start
                // with (should a later column outgrow it by 2^8 the tile is redone below)
                uint32_t f[32];
                tmem_ld32(f, tmem_s + lane_base);
                tmem_ld_wait(f);
                mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (full || (word[0] & (1u << i)) != 0u) mx = fmaxf(mx, __uint_as_float(f[i]));
            }
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass) {
                if (pass == 1 || n_mine == 0) {
                    const bool up = (mx - m_ref) * c2 > 8.f;          // true from -inf
                    if (n_mine > 0) {                     // rescale my row of O_g in tensor memory
                        const float alpha = up ? fast_exp2((m_ref - mx) * c2) : 1.f;
#pragma unroll 1
                        for (int c0 = 0; c0 < D; c0 += 32) {
                            uint32_t o[32];
                            tmem_ld32(o, tmem_og + lane_base + c0);
                            tmem_ld_wait(o);
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                            tmem_st32(tmem_og + lane_base + c0, o);
                        }
                        l *= alpha;
                    }
                    if (up) m_ref = mx;
                    mu = m_ref == -INFINITY ? 0.f : m_ref * c2;
                }
                if (full) sweep(yes, no);
                else sweep(yes, yes);
                if (!__any_sync(0xffffffffu, (mx - m_ref) * c2 > 8.f)) break;
            }
            l += l_tile;
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // P visible to the tensor core
            umma::fence_before_sync();
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar_p + g * 8) : "memory");
        }

        // ---- epilogue: merge the two groups' results; O / l and the log-sum-exp of every row go to
        // this run's partial-result slot.  Each thread puts its unnormalised row of O_g into shared
        // memory (the K and V stages, free once every product is done; the (exponent, sum) pairs
        // go to the P buffers); then each warp merges and writes whole rows, 512 contiguous bytes
        // per store instruction.
        if (n_mine > 0) alive = mbar_wait(bar_o + g * 8, (n_mine - 1) & 1, a.status, qt) && alive;
        umma::fence_after_sync();
        asm volatile("bar.sync 1, 256;\n" ::: "memory");  // every product of either group is done
        float2 *stats = reinterpret_cast<float2 *>(smem + OFF_P);            // [2][128]
        float *stage = reinterpret_cast<float *>(smem + OFF_K);              // [2][128][128], 16-byte chunks swizzled
        const float my_mu = (n_mine > 0 && alive && m_ref != -INFINITY) ? m_ref * c2 : -INFINITY;
        stats[g * 128 + r] = make_float2(my_mu, l);
        {
            float *srow = stage + (g * 128 + r) * D;
#pragma unroll 1
            for (int c0 = 0; c0 < D; c0 += 32) {
                uint32_t o[32];
                if (n_mine > 0) {
                    tmem_ld32(o, tmem_og + lane_base + c0);
                    tmem_ld_wait(o);
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = 0u;
                }
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const int chunk = (c0 + i) >> 2;
                    *reinterpret_cast<uint4 *>(srow + ((chunk ^ (r & 7)) << 2)) = make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
                }
            }
        }
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        const size_t slot = size_t(run);
        const bool whole = pa.n_runs == 1;                // this is the output already
        constexpr int RPW = QM / (PFX_SOFTMAX / 32);      // 16 rows per warp: rows warp * 16 ..
        // lanes 0..15 work out the two groups' weights for one row each; they are handed round by shuffle
        float f0 = 0.f, f1 = 0.f;
        {
            const int rr = warp * RPW + (lane & (RPW - 1));
            const float2 s0 = stats[rr], s1 = stats[128 + rr];
            const float mu_all = fmaxf(s0.x, s1.x);
            const float w0 = s0.x == -INFINITY ? 0.f : fast_exp2(s0.x - mu_all);
            const float w1 = s1.x == -INFINITY ? 0.f : fast_exp2(s1.x - mu_all);
            const float l_all = s0.y * w0 + s1.y * w1;
            const float inv = l_all > 0.f ? 1.f / l_all : 0.f;
            f0 = w0 * inv;
            f1 = w1 * inv;
            const int grow = qt * QM + (rr & ((1 << pa.pack_shift) - 1)), hr = h + (rr >> pa.pack_shift);
            if (lane < RPW && grow < n_q && (!whole || a.lse != nullptr))
                (whole ? a.lse : a.part_lse)[((slot * a.Z + z) * a.H + hr) * n_q + grow] =
                    l_all > 0.f ? mu_all + log2f(l_all) : -INFINITY;
        }
#pragma unroll 4
        for (int i = 0; i < RPW; ++i) {
            const int rr = warp * RPW + i, grow = qt * QM + (rr & ((1 << pa.pack_shift) - 1)), hr = h + (rr >> pa.pack_shift);
            const float g0 = __shfl_sync(0xffffffffu, f0, i), g1 = __shfl_sync(0xffffffffu, f1, i);
            if (lane >= D / 4) continue;                  // a row is D / 4 chunks of four floats
            const int sw = (lane ^ (rr & 7)) << 2;
            const float4 v0 = *reinterpret_cast<const float4 *>(stage + rr * D + sw);
            const float4 v1 = *reinterpret_cast<const float4 *>(stage + (128 + rr) * D + sw);
            if (grow >= n_q) continue;
            if (whole) {
                T *to = static_cast<T *>(a.o) + z * a.os_z + hr * a.os_h + grow * a.os_n;
                reinterpret_cast<uint2 *>(to)[lane] = make_uint2(MT::pack(v0.x * g0 + v1.x * g1, v0.y * g0 + v1.y * g1),
                                                                 MT::pack(v0.z * g0 + v1.z * g1, v0.w * g0 + v1.w * g1));
            } else {
                const size_t prow_g = ((slot * a.Z + z) * a.H + hr) * n_q + grow;
                reinterpret_cast<float4 *>(a.part_o + prow_g * D)[lane] =
                    make_float4(v0.x * g0 + v1.x * g1, v0.y * g0 + v1.y * g1, v0.z * g0 + v1.z * g1, v0.w * g0 + v1.w * g1);
            }
        }
    }

    umma::fence_before_sync();
    __syncthreads();
    if (warp == 9) umma::tmem_free_all(tmem_base);
}

// rank-4 map with 64-column x 128-row boxes (kept in the calling thread's table of maps)
static bool make_map_rows128(CUtensorMap *map, const void *base, bool bf16, int D, int rows, int H, int Z,
                             int64_t stride_n, int64_t stride_h, int64_t stride_z) {
    return make_map(map, base, bf16, D, rows, H, Z, stride_n, stride_h, stride_z, 128);
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
        !make_map_rows128(&tkt, a.k, bf16, D, a.n_kv, H_kv, a.Z, a.ks_n, a.ks_h, a.ks_z) ||
        !make_map_rows128(&tvt, a.v, bf16, D, a.n_kv, H_kv, a.Z, a.vs_n, a.vs_h, a.vs_z))
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
    PrefixArgs pa{n_runs, nullptr, nullptr, 0, 0, 0, pack, 7};
    for (int p = pack; p > 1; p /= 2) --pa.pack_shift;
    if (PAGED) {
        pa.block_table = pg->block_table;
        pa.prefix_lens = pg->prefix_lens;
        pa.table_stride = pg->table_stride;
        pa.page_size = pg->page_size;
        pa.n_pages = pg->n_pages;
    }
    dim3 grid((a.n_q + umma::QM - 1) / umma::QM, a.H / pack, a.Z * n_runs);
    prefix_umma_kernel<T, D, PAGED><<<grid, PFX_THREADS, umma::Geo<D>::SMEM_BYTES, stream>>>(a, pa, tq, tk, tv, tkt, tvt);
    return cudaGetLastError();
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

// The whole call - prefix and tree - in n_runs runs of column tiles: the output when there is one, else partial
// results 0 .. n_runs - 1.
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
