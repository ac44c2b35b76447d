// Tree precompute: parent array -> per-block ancestor list, row-by-ancestor mask, leaf list.
//
// Semantics follow the reference's create_fst_attention_kernel_inputs (utils.py:104-129):
//   A_b   = ascending unique strict ancestors of the rows of block b          (utils.py:119)
//   mask  = [row j][slot a] : A_b[a] is an ancestor of row j, or is row j     (utils.py:124-127)
//   leaf  = rows of the block that are not in A_b, rows past the last node
//           included                                                           (utils.py:121-122)
// The reference gets there with unique / isin over a lineage matrix in Python loops; here one
// CTA per (tree, block) marks ancestors by walking parent links (byte flags in shared memory,
// plain stores: many walkers hit the same few nodes and atomics on one word would serialise),
// packs the flags into a bitmap, ranks the set bits with a popcount prefix scan (which yields
// the ascending order of torch.unique without sorting) and walks each row's chain once more to
// set its mask bits.
// Integer work only; the reference-format outputs are bit-identical to the reference's.
//
// The packed form written for the attention kernels splits A_b in two: ancestors outside the
// block's own rows ("external", gathered row by row) and ancestors inside it, which the kernel
// reads from the block's contiguous K/V rows through a row-by-row bit mask that also carries
// the self bit (the reference's leaf path, utils.py:121-122, and its self-through-mask case,
// utils.py:124-127, become the diagonal of that mask).
//
// Also here: the converter from reference-format metadata tensors to the packed form.

#include <algorithm>
#include <atomic>
#include <climits>

#include "fst_common.cuh"

namespace fst {

constexpr int PRE_THREADS = 256;
constexpr int PRE_WARPS = PRE_THREADS / 32;

// four bits as four bool bytes
__device__ __forceinline__ uint32_t bool_bytes(uint32_t bits) { return ((bits & 0xfu) * 0x00204081u) & 0x01010101u; }

constexpr int kWideNodes = 8192;       // larger trees are not staged
constexpr int SET_MOST = 128;          // rows of a block, and its ancestors
constexpr int SET_SLOTS = 1024;
struct AncestorSet {
    uint4 bits[SET_MOST];              // masks of the slots
    uint4 row[SET_MOST];               // and of the block's rows
    int key[SET_SLOTS];                // node at a place of the hash table, -1: none
    int node[SET_MOST];                // in the order of their places, INT_MAX behind the last
    int sorted[SET_MOST];              // by slot
    uint32_t blk[SET_MOST * (SET_MOST / 32)];
    int16_t up[SET_SLOTS];             // place of the parent, -1: a root
    int16_t slot[SET_SLOTS];           // slot of the node at that place
    int16_t place[SET_MOST];           // their places
    int16_t jump[SET_MOST], self[SET_MOST];    // of a slot: an ancestor's slot; of a row: its own slot, -1: nobody's ancestor
    int warp[PRE_WARPS];               // taken places of a warp's share
    int full;                          // too many nodes for the table
};

// One block's metadata by way of a hash set of its ancestors; false, with nothing written, when there are more than max_ancestors.
//   * a row climbs until it meets a node that is in the set, and links every node to its parent's place on the way;
//   * a node's slot is the number of smaller ones: everybody compares;
//   * the slots' masks, a uint4 each, by pointer doubling over the links; a row's mask is its parent's.
template <typename Parent>
__device__ __forceinline__ bool precompute_set(AncestorSet &set, const Parent &par, int b, int n_nodes, int bm, int ma,
                                               unsigned char *blob, const PackedLayout &L, int64_t *o_idx, uint8_t *o_mask, int64_t *o_leaf) {
    const int tid = threadIdx.x, row0 = b * bm, maw = L.maw, bw = L.bw;
    for (int i = tid; i < SET_SLOTS / 4; i += PRE_THREADS) reinterpret_cast<int4 *>(set.key)[i] = make_int4(-1, -1, -1, -1);
    if (tid < SET_MOST) {
        set.node[tid] = INT_MAX;
        set.self[tid] = -1;
        reinterpret_cast<uint4 *>(set.blk)[tid] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (tid == 0) set.full = 0;
    __syncthreads();

    int first = -1;                                       // place of my row's parent
    if (tid < bm) {
        int x = row0 + tid < n_nodes ? par(row0 + tid) : -1, below = -1;
        while (x >= 0) {
            const int next = par(x);                      // under way while x is looked up
            int at = int((uint32_t(x) * 0x9E3779B1u) >> 22), was, tries = 0;
            while ((was = atomicCAS(&set.key[at], -1, x)) != -1 && was != x && ++tries < 2 * SET_MOST) at = (at + 1) & (SET_SLOTS - 1);
            if (tries >= 2 * SET_MOST) {                  // no set of SET_MOST nodes has such a run of taken places
                set.full = 1;
                break;
            }
            if (below < 0) first = at;
            else set.up[below] = int16_t(at);
            if (was == x) break;                          // somebody else goes on from here
            if (next < 0) set.up[at] = -1;
            below = at;
            x = next;
        }
    }
    __syncthreads();
    // the nodes and their places, in the order of the places: four to a thread (counting them in the climb would make the
    // counter a link of a deep tree's chain)
    static_assert(SET_SLOTS == 4 * PRE_THREADS, "four places to a thread");
    const int4 mine4 = reinterpret_cast<const int4 *>(set.key)[tid];
    const int own = int(mine4.x >= 0) + int(mine4.y >= 0) + int(mine4.z >= 0) + int(mine4.w >= 0);
    int before = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, before, o);
        if ((tid & 31) >= o) before += v;
    }
    if ((tid & 31) == 31) set.warp[tid >> 5] = before;
    __syncthreads();
    int n = 0;
    before -= own;
#pragma unroll
    for (int w = 0; w < PRE_WARPS; ++w) {
        before += w < tid >> 5 ? set.warp[w] : 0;
        n += set.warp[w];
    }
    if (n > ma || set.full) return false;
    const int four[4] = {mine4.x, mine4.y, mine4.z, mine4.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (four[i] >= 0) {
            set.place[before] = int16_t(tid * 4 + i);
            set.node[before++] = four[i];
        }
    __syncthreads();

    // slots: thread pairs share a node, half of the comparisons each
    const int k = tid >> 1, mine = set.node[k];
    int rank = 0;
#pragma unroll 4
    for (int i = tid & 1; i < (n + 3) >> 2; i += 2) {
        const int4 v = reinterpret_cast<const int4 *>(set.node)[i];
        rank += int(v.x < mine) + int(v.y < mine) + int(v.z < mine) + int(v.w < mine);
    }
    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
    const bool have = (tid & 1) == 0 && k < n;
    const int at = have ? set.place[k] : 0;
    if (have) {
        set.slot[at] = int16_t(rank);
        set.sorted[rank] = mine;
        if (mine >= row0) set.self[mine - row0] = int16_t(rank);
    }
    const int n_ext = __syncthreads_count(have && mine < row0);
    if (have) {
        const int p = set.up[at];
        set.jump[rank] = p < 0 ? int16_t(-1) : set.slot[p];
        const uint32_t bit = 1u << (rank & 31);
        const int w = rank >> 5;
        set.bits[rank] = make_uint4(w == 0 ? bit : 0u, w == 1 ? bit : 0u, w == 2 ? bit : 0u, w == 3 ? bit : 0u);
    }
    const int above = first < 0 ? -1 : set.slot[first];   // slot of my row's parent
    if (tid < ma) {
        const int node = tid < n ? set.sorted[tid] : -1;
        if (o_idx) o_idx[tid] = node;
        if (blob) reinterpret_cast<int32_t *>(blob + L.off_idx)[size_t(b) * ma + tid] = tid < n_ext ? node : -1;
    }
    if (tid == 0 && blob) reinterpret_cast<int32_t *>(blob + L.off_count)[b] = n_ext;
    __syncthreads();
    for (;;) {
        uint4 got = make_uint4(0u, 0u, 0u, 0u);
        int to = tid < n ? set.jump[tid] : -1;
        const bool any = to >= 0;
        if (any) {
            got = set.bits[to];
            to = set.jump[to];
        }
        if (!__syncthreads_or(any)) break;
        if (any) {
            uint4 m = set.bits[tid];
            m.x |= got.x; m.y |= got.y; m.z |= got.z; m.w |= got.w;
            set.bits[tid] = m;
            set.jump[tid] = int16_t(to);
        }
        __syncthreads();
    }
    if (tid < bm) {
        const int j = tid, self = set.self[j];
        uint4 m = above >= 0 ? set.bits[above] : make_uint4(0u, 0u, 0u, 0u);
        if (self >= 0) {
            const uint32_t bit = 1u << (self & 31);
            m.x |= self >> 5 == 0 ? bit : 0u; m.y |= self >> 5 == 1 ? bit : 0u; m.z |= self >> 5 == 2 ? bit : 0u; m.w |= self >> 5 == 3 ? bit : 0u;
        }
        set.row[j] = m;
        uint32_t *blk = set.blk + j * bw;
        blk[j >> 5] = 1u << (j & 31);                     // every row attends to itself, and to its ancestors in the block
        const uint32_t word[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const int below = n_ext - w * 32;             // slots of this word that are outside
            for (uint32_t in = below >= 32 ? 0u : below > 0 ? word[w] & ~((1u << below) - 1u) : word[w]; in != 0u; in &= in - 1u) {
                const int c = set.sorted[w * 32 + __ffs(in) - 1] - row0;
                blk[c >> 5] |= 1u << (c & 31);
            }
        }
        if (o_leaf) o_leaf[j] = self >= 0 ? int64_t(-1) : int64_t(row0 + j);
    }
    __syncthreads();
    const uint32_t *row = reinterpret_cast<const uint32_t *>(set.row);
    if (blob) {
        uint32_t *p_emask = reinterpret_cast<uint32_t *>(blob + L.off_emask) + size_t(b) * bm * maw;
        uint32_t *p_bmask = reinterpret_cast<uint32_t *>(blob + L.off_bmask) + size_t(b) * bm * bw;
        for (int i = tid; i < bm * maw; i += PRE_THREADS) {
            const int j = maw == 4 ? i >> 2 : i / maw, w = i - j * maw, outside = n_ext - w * 32;
            p_emask[i] = row[j * 4 + w] & (outside >= 32 ? 0xffffffffu : outside > 0 ? (1u << outside) - 1u : 0u);
        }
        for (int i = tid; i < bm * bw; i += PRE_THREADS) p_bmask[i] = set.blk[i];
    }
    if (o_mask) {
        if ((ma & 15) == 0 && (reinterpret_cast<uintptr_t>(o_mask) & 15) == 0) {     // sixteen bool bytes per store
            const int pieces = ma / 16, step = PRE_THREADS / pieces, j0 = tid / pieces, at16 = (tid - j0 * pieces) * 16;
            if (j0 < step)
                for (int j = j0; j < bm; j += step) {
                    const uint32_t half = row[j * 4 + (at16 >> 5)] >> (at16 & 31);
                    reinterpret_cast<uint4 *>(o_mask)[j * pieces + (at16 >> 4)] =
                        make_uint4(bool_bytes(half), bool_bytes(half >> 4), bool_bytes(half >> 8), bool_bytes(half >> 12));
                }
        } else {
            for (int i = tid; i < bm * ma; i += PRE_THREADS) {
                const int j = i / ma, c = i - j * ma;
                o_mask[i] = (row[j * 4 + (c >> 5)] >> (c & 31)) & 1u;
            }
        }
    }
    return true;
}

// BYTE_FLAGS: ancestors are first marked as one byte per node and packed into the bitmap by
// ballots (the fast path: plain stores never serialise).  Without it the walkers set bitmap bits
// with atomicOr directly; that needs 1/9 of the shared memory and is what lets trees of a
// hundred thousand nodes and more fit (a CTA keeps a bitmap of every node below its last row).
template <bool BYTE_FLAGS, bool SET>
__global__ void __launch_bounds__(PRE_THREADS)
precompute_kernel(const int32_t *__restrict__ parent_all, int n_nodes, int bm, int ma, int par_cap, int depth_cap,
                  int64_t *__restrict__ anc_idx_all, uint8_t *__restrict__ anc_mask_all,
                  int64_t *__restrict__ leaf_idx_all, unsigned char *__restrict__ packed_all,
                  size_t packed_stride, int32_t *status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int b = blockIdx.x, tree = blockIdx.y, nb = gridDim.x;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int row0 = b * bm;
    const int row_end = row0 + bm;                       // may run past the last node
    const int n_here = min(row_end, n_nodes);            // nodes that exist below row_end
    const int W = (row_end + 31) >> 5;                   // bitmap words, phantom rows included
    const int maw = (ma + 31) >> 5;

    uint32_t *bitmap = reinterpret_cast<uint32_t *>(smem_raw);
    int *rank = reinterpret_cast<int *>(bitmap + W);     // set bits in words below w
    const int bw = (bm + 31) >> 5;
    uint32_t *rowmask = reinterpret_cast<uint32_t *>(rank + W);      // [bm][maw] over all of A_b
    uint32_t *blkmask = rowmask + size_t(bm) * maw;                   // [bm][bw] over block rows
    int *warp_tot = reinterpret_cast<int *>(blkmask + size_t(bm) * bw);
    unsigned char *flag = reinterpret_cast<unsigned char *>(warp_tot + 40);   // [W*32] node is an ancestor
    int *chain = reinterpret_cast<int *>(flag + (BYTE_FLAGS ? size_t(W) * 32 : 0));   // [depth_cap][bm] ancestors of row j
    int *depth = chain + size_t(depth_cap) * bm;                      // [bm] recorded chain length
    // SET: the parents of all nodes below the block's end, then the set; everything above takes their place if it does not do
    int *s_par = SET ? reinterpret_cast<int *>(smem_raw) : depth + bm;

    const int32_t *parent = parent_all + size_t(tree) * n_nodes;
    const int cap = min(par_cap, n_here);
    // parents are checked once, here: a malformed entry is reported and treated as a root, so
    // every walk below ends
    auto checked = [&](int x, int p) -> int {
        if (p >= x || p < -1) {
            report(status, FST_DEV_MALFORMED_TREE, x, p);
            p = -1;
        }
        return p;
    };
    for (int i0 = tid; i0 < cap; i0 += 8 * PRE_THREADS) {    // eight loads in flight per thread
        int v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + u * PRE_THREADS;
            v[u] = i < cap ? __ldg(parent + i) : -1;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + u * PRE_THREADS;
            if (i < cap) s_par[i] = checked(i, v[u]);
        }
    }
    if constexpr (SET) {
        AncestorSet &set = *reinterpret_cast<AncestorSet *>(smem_raw + ((size_t(cap) * 4 + 15) & ~size_t(15)));
        const PackedLayout L = packed_layout(nb, bm, ma);
        const size_t blk = size_t(tree) * nb + b;
        __syncthreads();
        if (precompute_set(set, [&](int x) { return s_par[x]; }, b, n_nodes, bm, ma, packed_all ? packed_all + size_t(tree) * packed_stride : nullptr, L,
                           anc_idx_all ? anc_idx_all + blk * ma : nullptr, anc_mask_all ? anc_mask_all + blk * size_t(bm) * ma : nullptr,
                           leaf_idx_all ? leaf_idx_all + blk * bm : nullptr))
            return;
        // more ancestors than the bound: again, with room for as many as there are
        s_par = depth + bm;
        __syncthreads();
        for (int i = tid; i < cap; i += PRE_THREADS) s_par[i] = checked(i, __ldg(parent + i));
    }
    if (BYTE_FLAGS) {
        for (int i = tid; i < W * 8; i += PRE_THREADS) reinterpret_cast<uint32_t *>(flag)[i] = 0u;
    } else {
        for (int i = tid; i < W; i += PRE_THREADS) bitmap[i] = 0u;
    }
    for (int i = tid; i < bm * maw; i += PRE_THREADS) rowmask[i] = 0u;
    for (int i = tid; i < bm * bw; i += PRE_THREADS) blkmask[i] = 0u;
    __syncthreads();

    const bool all_staged = cap >= n_here;
    auto par = [&](int x) -> int {
        if (all_staged || x < cap) return s_par[x];
        return checked(x, __ldg(parent + x));
    };

    // 1. every row climbs to its root, recording the chain (its lineage) and flagging each node
    //    as an ancestor.  Flags are bytes written with plain stores: many rows hit the same few
    //    nodes and atomics on one word would serialise.  The loop body is kept minimal because
    //    its length times the depth of the tree is the critical path of this kernel.
    int too_deep = 0;
    for (int j = tid; j < bm; j += PRE_THREADS) {
        const int k = row0 + j;
        int n = 0;
        if (k < n_nodes) {
            int a = par(k);
            while (a >= 0) {
                if (n < depth_cap) chain[n * bm + j] = a;
                if (BYTE_FLAGS) flag[a] = 1;
                else atomicOr(&bitmap[a >> 5], 1u << (a & 31));
                ++n;
                a = par(a);
            }
        }
        depth[j] = n;
        too_deep |= n > depth_cap;
    }
    const bool walk_masks = __syncthreads_or(too_deep) != 0;          // also: flags complete
    // flags -> bitmap, one warp per word
    if (BYTE_FLAGS) {
        for (int w = wid; w < W; w += PRE_WARPS) {
            const uint32_t word = __ballot_sync(0xffffffffu, flag[w * 32 + lane] != 0);
            if (lane == 0) bitmap[w] = word;
        }
        __syncthreads();
    }

    // 2. exclusive popcount scan over the bitmap words -> rank[w]
    const int per = (W + PRE_THREADS - 1) / PRE_THREADS;
    const int w0 = min(W, tid * per), w1 = min(W, w0 + per);
    int mine = 0;
    for (int w = w0; w < w1; ++w) mine += __popc(bitmap[w]);
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const int v = lane < PRE_WARPS ? warp_tot[lane] : 0;
        int iv = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, iv, o);
            if (lane >= o) iv += u;
        }
        warp_tot[lane] = iv - v;
        if (lane == 31) warp_tot[32] = iv;
    }
    __syncthreads();
    {
        int base = warp_tot[wid] + inc - mine;
        for (int w = w0; w < w1; ++w) {
            rank[w] = base;
            base += __popc(bitmap[w]);
        }
    }
    const int n_anc = warp_tot[32];
    const int n_keep = min(n_anc, ma);
    if (n_anc > ma && tid == 0) report(status, FST_DEV_ANCESTOR_OVERFLOW, tree * 65536 + b, n_anc);
    __syncthreads();
    // external ancestors are the ones below row0; they come first in ascending order
    const int n_ext = min(ma, rank[row0 >> 5] + __popc(bitmap[row0 >> 5] & ((1u << (row0 & 31)) - 1u)));

    const PackedLayout L = packed_layout(nb, bm, ma);
    unsigned char *blob = packed_all ? packed_all + size_t(tree) * packed_stride : nullptr;
    int32_t *p_count = blob ? reinterpret_cast<int32_t *>(blob + L.off_count) : nullptr;
    int32_t *p_idx = blob ? reinterpret_cast<int32_t *>(blob + L.off_idx) + size_t(b) * ma : nullptr;
    uint32_t *p_emask = blob ? reinterpret_cast<uint32_t *>(blob + L.off_emask) + size_t(b) * bm * maw
                             : nullptr;
    uint32_t *p_bmask = blob ? reinterpret_cast<uint32_t *>(blob + L.off_bmask) + size_t(b) * bm * bw
                             : nullptr;
    const size_t blk = size_t(tree) * nb + b;
    int64_t *o_idx = anc_idx_all ? anc_idx_all + blk * ma : nullptr;
    uint8_t *o_mask = anc_mask_all ? anc_mask_all + blk * size_t(bm) * ma : nullptr;
    int64_t *o_leaf = leaf_idx_all ? leaf_idx_all + blk * bm : nullptr;

    // 3. ascending ancestor list: slot = rank of the bit; one warp per word, one lane per node
    for (int w = wid; w < W; w += PRE_WARPS) {
        const uint32_t bits = bitmap[w];
        if ((bits >> lane) & 1u) {
            const int pos = rank[w] + __popc(bits & ((1u << lane) - 1u));
            if (pos < ma) {
                const int node = w * 32 + lane;
                if (p_idx && node < row0) p_idx[pos] = node;
                if (o_idx) o_idx[pos] = node;
            }
        }
    }
    if (p_idx)
        for (int a = n_ext + tid; a < ma; a += PRE_THREADS) p_idx[a] = -1;
    if (o_idx)
        for (int a = n_keep + tid; a < ma; a += PRE_THREADS) o_idx[a] = -1;
    if (tid == 0 && p_count) p_count[b] = n_ext;

    // 4. mask rows: bit (row, slot of node) for the row itself, when it is somebody's ancestor
    //    here, and for every node of its chain; plus the same in block-column space.
    if (!walk_masks) {
        // one work item per recorded (row, chain step), spread over all threads
        for (int j = tid; j < bm; j += PRE_THREADS) {
            const int k = row0 + j;
            atomicOr(&blkmask[j * bw + (j >> 5)], 1u << (j & 31));     // every row attends to itself
            if (k < n_nodes && ((bitmap[k >> 5] >> (k & 31)) & 1u)) {
                const int pos = rank[k >> 5] + __popc(bitmap[k >> 5] & ((1u << (k & 31)) - 1u));
                if (pos < ma) atomicOr(&rowmask[j * maw + (pos >> 5)], 1u << (pos & 31));
            }
        }
        int dmax = 0;
        for (int j = lane; j < bm; j += 32) dmax = max(dmax, depth[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dmax = max(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        for (int i = tid; i < dmax * bm; i += PRE_THREADS) {
            const int sidx = i / bm, j = i - sidx * bm;
            if (sidx < depth[j]) {
                const int x = chain[i];
                const uint32_t word = bitmap[x >> 5];
                const int pos = rank[x >> 5] + __popc(word & ((1u << (x & 31)) - 1u));
                if (pos < ma) atomicOr(&rowmask[j * maw + (pos >> 5)], 1u << (pos & 31));
                if (x >= row0) atomicOr(&blkmask[j * bw + ((x - row0) >> 5)], 1u << ((x - row0) & 31));
            }
        }
    } else {
        // a chain longer than the recording space: walk every row's chain again
        for (int j = tid; j < bm; j += PRE_THREADS) {
            const int k = row0 + j;
            blkmask[j * bw + (j >> 5)] |= 1u << (j & 31);
            if (k < n_nodes) {
                int x = k;
                while (x >= 0) {
                    const uint32_t word = bitmap[x >> 5];
                    const uint32_t bit = 1u << (x & 31);
                    const int up = par(x);
                    if (word & bit) {
                        const int pos = rank[x >> 5] + __popc(word & (bit - 1u));
                        if (pos < ma) rowmask[j * maw + (pos >> 5)] |= 1u << (pos & 31);
                        if (x >= row0) blkmask[j * bw + ((x - row0) >> 5)] |= 1u << ((x - row0) & 31);
                    }
                    x = up;
                }
            }
        }
    }
    __syncthreads();

    if (p_emask) {
        for (int i = tid; i < bm * maw; i += PRE_THREADS) {
            const int w = i % maw, lo = w * 32;           // keep the bits of external slots only
            const uint32_t keep = n_ext >= lo + 32 ? 0xffffffffu : (n_ext > lo ? (1u << (n_ext - lo)) - 1u : 0u);
            p_emask[i] = rowmask[i] & keep;
        }
        for (int i = tid; i < bm * bw; i += PRE_THREADS) p_bmask[i] = blkmask[i];
    }
    if (o_mask) {
        if ((ma & 3) == 0) {                             // four bool bytes per store
            uint32_t *o32 = reinterpret_cast<uint32_t *>(o_mask);
            const int n4 = bm * ma / 4;
            for (int i = tid; i < n4; i += PRE_THREADS) {
                const int e = i * 4, j = e / ma, a = e - j * ma;
                const uint32_t nib = (rowmask[j * maw + (a >> 5)] >> (a & 31)) & 0xFu;
                o32[i] = (nib & 1u) | ((nib & 2u) << 7) | ((nib & 4u) << 14) | ((nib & 8u) << 21);
            }
        } else {
            for (int i = tid; i < bm * ma; i += PRE_THREADS) {
                const int j = i / ma, a = i - j * ma;
                o_mask[i] = (rowmask[j * maw + (a >> 5)] >> (a & 31)) & 1u;
            }
        }
    }

    // 5. leaves: block rows that are not in the ancestor set (rows past the last node too)
    if (o_leaf)
        for (int j = tid; j < bm; j += PRE_THREADS) {
            const int k = row0 + j;
            const bool leaf = !((bitmap[k >> 5] >> (k & 31)) & 1u);
            o_leaf[j] = leaf ? int64_t(k) : int64_t(-1);
        }
}

// The same for large trees.  precompute_kernel keeps the parents of every node below the block's last row
// in shared memory, so a block of a 131068-node tree reads half a megabyte to follow fifteen links per
// row, one CTA to an SM.  Here
//   * the rows climb through L2 (the parent array fits it many times over) and stop at the first node that
//     another row has been to; a bitmap of the nodes below the block is the only thing that grows with
//     the tree, and everything that walks it skips its empty words 32 at a time;
//   * the mask is inherited instead of climbed for again: a slot's row is its parent slot's row and its own
//     bit, by pointer doubling over the (at most max_ancestors) slots, and a block row's mask is its
//     parent's;
// so that a CTA's time is one climb and its shared memory lets seven share an SM.  131068 nodes, block_m 128, with
// the reference-format tensors: 161 us with precompute_kernel.
//
// With seven CTAs to an SM what counts is how many instructions a block takes, and a bitmap of 131068 nodes
// is 4096 words to clear and to walk twice for some seventy ancestors (28.7 us; its list took 5.6 us of a CTA's 20, one lane
// writing the neighbours that share a word).  Blocks and bounds of at most 128 therefore keep their ancestors in
// a hash set (precompute_set): 16.4 us, of which the climb, one dependent L2 read for each of fifteen levels, is the
// largest part.  A block with more ancestors than the bound is left to the bitmap, which counts them.
constexpr int WIDE_THREADS = PRE_THREADS, WIDE_WARPS = WIDE_THREADS / 32;

// 32-bit words of shared memory: bitmap and 16-bit ranks of Wp words, masks of slots or rows, block masks,
// parent and own slot of every row, and of every slot its node and parent slot
__host__ __device__ inline size_t wide_smem_words(size_t Wp, int bm, int ma, bool inherit) {
    const size_t maw = (ma + 31) / 32, bw = (bm + 31) / 32;
    return Wp + Wp / 2 + size_t(inherit && ma > bm ? ma : bm) * maw + size_t(bm) * bw + size_t(bm) * 2 + (inherit ? size_t(ma) * 2 : 0);
}

// (apart by SET: the set's code beside the bitmap's took registers from it, 12 to 20 % of a build with a bound of 512)
template <bool SET>
__global__ void __launch_bounds__(WIDE_THREADS, 7)
precompute_wide_kernel(const int32_t *__restrict__ parent_all, int n_nodes, int bm, int ma, int inherit_ok,
                       int64_t *__restrict__ anc_idx_all, uint8_t *__restrict__ anc_mask_all,
                       int64_t *__restrict__ leaf_idx_all, unsigned char *__restrict__ packed_all,
                       size_t packed_stride, int32_t *status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_warp[WIDE_WARPS], s_ext[WIDE_WARPS];
    const int b = blockIdx.x, tree = blockIdx.y, nb = gridDim.x;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int row0 = b * bm, maw = (ma + 31) >> 5, bw = (bm + 31) >> 5;
    // bitmap words, phantom rows included; every warp scans a run of whole 32-word groups
    const int per_warp = (((row0 + bm + 31) >> 5) + 32 * WIDE_WARPS - 1) / (32 * WIDE_WARPS) * 32, W = per_warp * WIDE_WARPS;

    uint32_t *bitmap = reinterpret_cast<uint32_t *>(smem_raw);       // [W]
    uint16_t *rank = reinterpret_cast<uint16_t *>(bitmap + W);       // [W] set bits below word w (only where w has any)
    uint32_t *bits = bitmap + W + W / 2;                             // inherited: [slot][maw], else [row][maw]
    uint32_t *blkmask = bits + size_t(inherit_ok && ma > bm ? ma : bm) * maw;   // [bm][bw] over block rows
    int *up = reinterpret_cast<int *>(blkmask + size_t(bm) * bw);    // [bm] parent of row j, then its slot
    int *self = up + bm;                                             // [bm] slot of row j itself, -1: nobody's ancestor
    int *node_of = self + bm, *jump = node_of + ma;                  // [ma] (inherited only)

    const int32_t *parent = parent_all + size_t(tree) * n_nodes;
    auto par = [&](int x) -> int {                        // a malformed entry is reported and treated as a root
        const int p = __ldg(parent + x);
        if (p >= x || p < -1) {
            report(status, FST_DEV_MALFORMED_TREE, x, p);
            return -1;
        }
        return p;
    };
    if constexpr (SET) {
        const size_t blk = size_t(tree) * nb + b;
        if (precompute_set(*reinterpret_cast<AncestorSet *>(smem_raw), par, b, n_nodes, bm, ma,
                           packed_all ? packed_all + size_t(tree) * packed_stride : nullptr, packed_layout(nb, bm, ma),
                           anc_idx_all ? anc_idx_all + blk * ma : nullptr, anc_mask_all ? anc_mask_all + blk * size_t(bm) * ma : nullptr,
                           leaf_idx_all ? leaf_idx_all + blk * bm : nullptr))
            return;
        __syncthreads();                                  // more ancestors than the bound: the bitmap takes the set's place
    }
    for (int i = tid; i < W / 4; i += WIDE_THREADS) reinterpret_cast<uint4 *>(bitmap)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int i = tid; i < bm * bw; i += WIDE_THREADS) blkmask[i] = 0u;
    __syncthreads();

    // 1. every row climbs until it meets a marked node
    for (int j = tid; j < bm; j += WIDE_THREADS) {
        int x = row0 + j < n_nodes ? par(row0 + j) : -1;
        up[j] = x;
        while (x >= 0) {
            const int next = par(x);                      // under way while x is marked
            const uint32_t bit = 1u << (x & 31);
            if (atomicOr(&bitmap[x >> 5], bit) & bit) break;
            x = next;
        }
    }
    __syncthreads();

    // 2. ranks: set bits before every word that has some
    int mine = 0;
    for (int i = 0; i < per_warp; i += 32) mine += __popc(bitmap[wid * per_warp + i + lane]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane == 0) s_warp[wid] = mine;
    __syncthreads();
    int base = 0, n_anc = 0;
#pragma unroll
    for (int w = 0; w < WIDE_WARPS; ++w) {
        if (w < wid) base += s_warp[w];
        n_anc += s_warp[w];
    }
    const int n_keep = min(n_anc, ma);
    const bool inherit = inherit_ok && n_anc <= ma;
    if (n_anc > ma && tid == 0) report(status, FST_DEV_ANCESTOR_OVERFLOW, tree * 65536 + b, n_anc);

    const PackedLayout L = packed_layout(nb, bm, ma);
    unsigned char *blob = packed_all ? packed_all + size_t(tree) * packed_stride : nullptr;
    const size_t blk = size_t(tree) * nb + b;
    int64_t *o_idx = anc_idx_all ? anc_idx_all + blk * ma : nullptr;
    int32_t *p_idx = blob ? reinterpret_cast<int32_t *>(blob + L.off_idx) + size_t(b) * ma : nullptr;

    // 3. ascending ancestor list, a lane per word
    int ext = 0;                                          // listed nodes below the block
    for (int i = 0; i < per_warp; i += 32) {
        const int w = wid * per_warp + i + lane;
        uint32_t word = bitmap[w];
        if (__ballot_sync(0xffffffffu, word != 0u) == 0u) continue;
        const int own = __popc(word);
        int before = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += v;
        }
        const int group = __shfl_sync(0xffffffffu, before, 31);
        int pos = base + before - own;
        rank[w] = uint16_t(min(pos, 0xffff));
        for (; word != 0u; word &= word - 1u, ++pos) {
            const int node = w * 32 + __ffs(word) - 1;
            if (node < row0) ++ext;
            if (pos < ma) {
                if (p_idx && node < row0) p_idx[pos] = node;
                if (o_idx) o_idx[pos] = node;
                if (inherit) node_of[pos] = node;
            }
        }
        base += group;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ext += __shfl_xor_sync(0xffffffffu, ext, o);
    if (lane == 0) s_ext[wid] = ext;
    if (!inherit)
        for (int i = tid; i < bm * maw; i += WIDE_THREADS) bits[i] = 0u;
    __syncthreads();
    int n_ext = 0;
#pragma unroll
    for (int w = 0; w < WIDE_WARPS; ++w) n_ext += s_ext[w];
    n_ext = min(n_ext, ma);
    if (p_idx)
        for (int i = n_ext + tid; i < ma; i += WIDE_THREADS) p_idx[i] = -1;
    if (o_idx)
        for (int i = n_keep + tid; i < ma; i += WIDE_THREADS) o_idx[i] = -1;
    if (tid == 0 && blob) reinterpret_cast<int32_t *>(blob + L.off_count)[b] = n_ext;

    // 4. masks.  Slot of a node, -1 when it is nobody's ancestor here
    auto slot_of = [&](int x) -> int {
        const uint32_t word = bitmap[x >> 5], bit = 1u << (x & 31);
        return word & bit ? int(rank[x >> 5]) + __popc(word & (bit - 1u)) : -1;
    };
    if (inherit) {
        for (int s = tid; s < n_keep; s += WIDE_THREADS) {
            const int p = par(node_of[s]);
            jump[s] = p < 0 ? -1 : slot_of(p);
            for (int w = 0; w < maw; ++w) bits[s * maw + w] = w == (s >> 5) ? 1u << (s & 31) : 0u;
        }
        for (int j = tid; j < bm; j += WIDE_THREADS) {
            const int p = up[j];
            up[j] = p < 0 ? -1 : slot_of(p);
            self[j] = row0 + j < n_nodes ? slot_of(row0 + j) : -1;
        }
        __syncthreads();
        constexpr int PER = 2;                            // (slot, word) pairs per thread: 128 slots of 4 words
        const int pairs = n_keep * maw;
        for (;;) {
            bool any = false;
            uint32_t got[PER];
            int far[PER];
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = tid + k * WIDE_THREADS;
                got[k] = 0u;
                far[k] = -1;
                if (i < pairs) {
                    const int s = i / maw, w = i - s * maw, to = jump[s];
                    if (to >= 0) {
                        got[k] = bits[to * maw + w];
                        far[k] = jump[to];
                        any = true;
                    }
                } else {
                    break;
                }
            }
            if (!__syncthreads_or(any)) break;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = tid + k * WIDE_THREADS;
                if (i >= pairs) break;
                bits[i] |= got[k];
                if (i % maw == 0) jump[i / maw] = far[k];
            }
            __syncthreads();
        }
    } else {                                              // too many ancestors, or too wide a mask: climb again
        for (int j = tid; j < bm; j += WIDE_THREADS)
            for (int x = row0 + j < n_nodes ? row0 + j : -1; x >= 0;) {
                const int next = par(x), pos = slot_of(x);    // the next load is under way meanwhile
                if (pos >= 0 && pos < ma) bits[j * maw + (pos >> 5)] |= 1u << (pos & 31);
                if (pos >= 0 && x >= row0) blkmask[j * bw + ((x - row0) >> 5)] |= 1u << ((x - row0) & 31);
                x = next;
            }
        __syncthreads();
    }
    auto row_word = [&](int j, int w) -> uint32_t {       // word w of row j's mask over all of A_b
        if (!inherit) return bits[j * maw + w];
        const uint32_t above = up[j] >= 0 ? bits[up[j] * maw + w] : 0u;
        return above | (self[j] >= 0 && (self[j] >> 5) == w ? 1u << (self[j] & 31) : 0u);
    };
    for (int j = tid; j < bm; j += WIDE_THREADS) {
        blkmask[j * bw + (j >> 5)] |= 1u << (j & 31);     // every row attends to itself
        if (inherit)                                      // and to its ancestors inside the block
            for (int s = n_ext; s < n_keep; ++s)
                if ((row_word(j, s >> 5) >> (s & 31)) & 1u) {
                    const int c = node_of[s] - row0;
                    blkmask[j * bw + (c >> 5)] |= 1u << (c & 31);
                }
    }

    if (blob) {
        uint32_t *p_emask = reinterpret_cast<uint32_t *>(blob + L.off_emask) + size_t(b) * bm * maw;
        for (int i = tid; i < bm * maw; i += WIDE_THREADS) {
            const int j = i / maw, w = i - j * maw, lo = w * 32;      // keep the bits of external slots only
            const uint32_t keep = n_ext >= lo + 32 ? 0xffffffffu : (n_ext > lo ? (1u << (n_ext - lo)) - 1u : 0u);
            p_emask[i] = row_word(j, w) & keep;
        }
    }
    if (anc_mask_all) {
        uint8_t *o_mask = anc_mask_all + blk * size_t(bm) * ma;
        if ((ma & 15) == 0 && (reinterpret_cast<uintptr_t>(o_mask) & 15) == 0) {   // sixteen bool bytes per store
            const int pieces = ma / 16;
            for (int i = tid; i < bm * pieces; i += WIDE_THREADS) {
                const int j = i / pieces, at = (i - j * pieces) * 16;
                const uint32_t half = row_word(j, at >> 5) >> (at & 31);
                reinterpret_cast<uint4 *>(o_mask)[i] = make_uint4(bool_bytes(half), bool_bytes(half >> 4), bool_bytes(half >> 8), bool_bytes(half >> 12));
            }
        } else {
            for (int i = tid; i < bm * ma; i += WIDE_THREADS) {
                const int j = i / ma, at = i - j * ma;
                o_mask[i] = (row_word(j, at >> 5) >> (at & 31)) & 1u;
            }
        }
    }
    // 5. leaves: block rows that are not in the ancestor set (rows past the last node too)
    if (leaf_idx_all)
        for (int j = tid; j < bm; j += WIDE_THREADS) {
            const int k = row0 + j;
            leaf_idx_all[blk * bm + j] = ((bitmap[k >> 5] >> (k & 31)) & 1u) ? int64_t(-1) : int64_t(k);
        }
    __syncthreads();
    if (blob) {
        uint32_t *p_bmask = reinterpret_cast<uint32_t *>(blob + L.off_bmask) + size_t(b) * bm * bw;
        for (int i = tid; i < bm * bw; i += WIDE_THREADS) p_bmask[i] = blkmask[i];
    }
}

// -------------------------------------------------------------------------------------------
// reference-format tensors -> packed blob
// -------------------------------------------------------------------------------------------
constexpr int PACK_THREADS = 512;
constexpr int PACK_WORDS = 64;         // mask words of a row held in shared memory, half for each mask

__global__ void __launch_bounds__(PACK_THREADS)
pack_kernel(const int64_t *__restrict__ anc_idx_all, const uint8_t *__restrict__ anc_mask_all,
            const int64_t *__restrict__ leaf_idx_all, int bm, int ma, int64_t index_base,
            unsigned char *__restrict__ packed_all, size_t packed_stride, int32_t *status, int wide_words) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int b = blockIdx.x, tree = blockIdx.y, nb = gridDim.x;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int maw = (ma + 31) >> 5, bw = (bm + 31) >> 5;
    // slot -> external position (>= 0), or -1 - column for an ancestor inside the block, or
    // INT_MIN for padding
    int *slot_map = reinterpret_cast<int *>(smem_raw);               // [ma]
    uint32_t *s_wide = reinterpret_cast<uint32_t *>(slot_map + ma);  // [wide_words] the block's two masks
    __shared__ uint32_t s_bits[PACK_THREADS / 32][PACK_WORDS];
    __shared__ int s_warp[PACK_THREADS / 32];
    __shared__ int s_base;
    if (tid == 0) s_base = 0;
    __syncthreads();

    const PackedLayout L = packed_layout(nb, bm, ma);
    unsigned char *blob = packed_all + size_t(tree) * packed_stride;
    int32_t *p_count = reinterpret_cast<int32_t *>(blob + L.off_count);
    int32_t *p_idx = reinterpret_cast<int32_t *>(blob + L.off_idx) + size_t(b) * ma;
    uint32_t *p_emask = reinterpret_cast<uint32_t *>(blob + L.off_emask) + size_t(b) * bm * maw;
    uint32_t *p_bmask = reinterpret_cast<uint32_t *>(blob + L.off_bmask) + size_t(b) * bm * bw;
    const size_t blk = size_t(tree) * nb + b;
    const int64_t *g_idx = anc_idx_all + blk * ma;
    const uint8_t *g_mask = anc_mask_all + blk * size_t(bm) * ma;
    const int64_t *g_leaf = leaf_idx_all + blk * bm;
    const int64_t row0 = int64_t(b) * bm;

    // The mask's bytes are asked for first, sixteen at a time: nothing but their use depends on the slot
    // map (row after row, a warp each, with loads behind the map, took 8.4 us at 64 x 64).
    constexpr int AHEAD = 2;
    const bool wide = wide_words > 0;                     // both masks of the block fit shared memory
    const int pieces = ma / 16, n_pieces = bm * pieces;
    uint4 bytes[AHEAD];
    if (wide) {
        const uint4 *src = reinterpret_cast<const uint4 *>(g_mask);
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            const int i = tid + k * PACK_THREADS;
            bytes[k] = i < n_pieces ? __ldg(src + i) : make_uint4(0u, 0u, 0u, 0u);
        }
        for (int i = tid; i < wide_words; i += PACK_THREADS) s_wide[i] = 0u;
    }
    const int64_t my_leaf = tid < bm ? __ldg(g_leaf + tid) : -1;

    // external slots keep their order; an exclusive scan of the "is external" flags places them
    for (int a0 = 0; a0 < ma; a0 += PACK_THREADS) {
        const int a = a0 + tid;
        bool ext = false;
        int node = -1;
        int code = INT_MIN;
        if (a < ma) {
            const int64_t v = g_idx[a];
            const int64_t rel = v - index_base;
            if (v >= 0 && rel >= 0) {
                if (rel > 0x7fffffffLL) {
                    report(status, FST_DEV_INDEX_RANGE, tree * 65536 + b, a);
                } else if (rel >= row0 && rel < row0 + bm) {
                    code = -1 - int(rel - row0);
                } else {
                    ext = true;
                    node = int(rel);
                }
            }
        }
        const uint32_t votes = __ballot_sync(0xffffffffu, ext);
        if (lane == 0) s_warp[wid] = __popc(votes);
        __syncthreads();
        int pos = s_base + __popc(votes & ((1u << lane) - 1u));
        for (int w = 0; w < wid; ++w) pos += s_warp[w];
        if (ext) {
            code = pos;
            p_idx[pos] = node;
        }
        if (a < ma) slot_map[a] = code;
        __syncthreads();
        if (tid == 0) {
            int add = 0;
            for (int w = 0; w < PACK_THREADS / 32; ++w) add += s_warp[w];
            s_base += add;
        }
        __syncthreads();
    }
    const int n_ext = s_base;
    for (int a = n_ext + tid; a < ma; a += PACK_THREADS) p_idx[a] = -1;
    if (tid == 0) p_count[b] = n_ext;

    if (wide) {
        uint32_t *e = s_wide, *m = s_wide + size_t(bm) * maw;
        for (int j = tid; j < bm; j += PACK_THREADS) {
            const int64_t leaf = j == tid ? my_leaf : __ldg(g_leaf + j);
            if (leaf < 0 || leaf < index_base) continue;
            if (leaf - index_base != row0 + j) report(status, FST_DEV_INDEX_RANGE, tree * 65536 + b, -1 - j);
            atomicOr(&m[j * bw + (j >> 5)], 1u << (j & 31));
        }
        auto scatter = [&](int i, const uint4 &v) {
            const int j = i / pieces, a0 = (i - j * pieces) * 16;
            const uint32_t part[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int q = 0; q < 4; ++q)
                for (uint32_t rest = part[q]; rest != 0u;) {
                    const int k = (__ffs(rest) - 1) >> 3;     // the next byte that is not zero
                    rest &= ~(0xffu << (8 * k));
                    const int code = slot_map[a0 + q * 4 + k];
                    if (code >= 0) atomicOr(&e[j * maw + (code >> 5)], 1u << (code & 31));
                    else if (code != INT_MIN) atomicOr(&m[j * bw + ((-1 - code) >> 5)], 1u << ((-1 - code) & 31));
                }
        };
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (tid + k * PACK_THREADS < n_pieces) scatter(tid + k * PACK_THREADS, bytes[k]);
        for (int i = tid + AHEAD * PACK_THREADS; i < n_pieces; i += PACK_THREADS)
            scatter(i, __ldg(reinterpret_cast<const uint4 *>(g_mask) + i));
        __syncthreads();
        for (int i = tid; i < bm * maw; i += PACK_THREADS) p_emask[i] = e[i];
        for (int i = tid; i < bm * bw; i += PACK_THREADS) p_bmask[i] = m[i];
        return;
    }
    // Scatter the mask bytes into the two bit masks: a warp per row, a lane per byte, and the few bits
    // that are set go through shared memory (one thread per row, byte after byte, took 8 us at
    // 64 x 64; the loads of a whole row are now one access).
    uint32_t *er = s_bits[wid];
    uint32_t *br = er + PACK_WORDS / 2;
    const bool small = maw <= PACK_WORDS / 2 && bw <= PACK_WORDS / 2;
    for (int j = wid; j < bm; j += PACK_THREADS / 32) {
        uint32_t *e_out = p_emask + size_t(j) * maw, *b_out = p_bmask + size_t(j) * bw;
        uint32_t *e = small ? er : e_out, *m = small ? br : b_out;   // very wide masks: straight to memory
        for (int w = lane; w < maw; w += 32) e[w] = 0u;
        for (int w = lane; w < bw; w += 32) m[w] = 0u;
        __syncwarp();
        const int64_t leaf = g_leaf[j];
        const bool is_leaf = leaf >= 0 && leaf >= index_base;
        if (lane == 0 && is_leaf) {
            if (leaf - index_base != row0 + j) report(status, FST_DEV_INDEX_RANGE, tree * 65536 + b, -1 - j);
            atomicOr(&m[j >> 5], 1u << (j & 31));
        }
        const uint8_t *src = g_mask + size_t(j) * ma;
        for (int a = lane; a < ma; a += 32) {
            if (!src[a]) continue;
            const int code = slot_map[a];
            if (code >= 0) atomicOr(&e[code >> 5], 1u << (code & 31));
            else if (code != INT_MIN) atomicOr(&m[(-1 - code) >> 5], 1u << ((-1 - code) & 31));
        }
        __syncwarp();
        if (small) {
            for (int w = lane; w < maw; w += 32) e_out[w] = e[w];
            for (int w = lane; w < bw; w += 32) b_out[w] = m[w];
            __syncwarp();
        }
    }
}

// largest dynamic shared memory enabled so far, per device and kernel variant
static std::atomic<size_t> g_pre_smem_set[3][kMaxDevices];
static std::atomic<size_t> g_pack_smem_set[kMaxDevices];
static std::atomic<size_t> g_wide_smem_set[2][kMaxDevices];

cudaError_t launch_precompute(const int32_t *parent, int n_trees, int n_nodes, int bm, int ma,
                              int64_t *anc_idx, uint8_t *anc_mask, int64_t *leaf_idx,
                              void *packed, size_t packed_stride, int32_t *status,
                              cudaStream_t stream) {
    const int nb = (n_nodes + bm - 1) / bm;
    const int maw = (ma + 31) / 32;
    const size_t W = (size_t(nb) * bm + 31) / 32;
    const size_t budget = 200 * 1024;
    // bitmap + ranks + the two row masks + scan scratch + chain lengths
    const size_t base = (2 * W + size_t(bm) * maw + size_t(bm) * ((bm + 31) / 32) + 40 + size_t(bm)) * 4;
    // recording space for the rows' chains: as deep as 48 KB allows, at most 1024 levels
    int depth_cap = int((48 * 1024) / (size_t(bm) * 4));
    if (depth_cap > 1024) depth_cap = 1024;
    // Blocks and bounds of up to 128 start with the ancestor set; what is left to the flags then is a tree that is
    // refused, which need not be quick: its rows are climbed twice, and the space goes to more CTAs on an SM.
    // Us per build, flags / set, with the reference-format tensors: 256 nodes 6.5 / 5.7, 1020 7.5 / 6.0, 64 of them 17.1 / 12.4,
    // 16 x 8192 61.6 / 28.9, 4096 deep ones (depth 96) 15.3 / 14.5, four of 8000 32.6 / 18.7.
    const bool few = bm <= SET_MOST && ma <= SET_MOST, set = few && n_nodes <= kWideNodes;
    if (depth_cap < 1 || set) depth_cap = 1;
    // Byte flags (one byte per node below the last row) while they leave room to stage a good
    // part of the parent array; beyond that the walkers set bitmap bits with atomics.
    bool byte_flags = base + W * 32 + size_t(depth_cap) * bm * 4 + 16 * 1024 <= budget;
    size_t fixed = base + (byte_flags ? W * 32 : 0) + size_t(depth_cap) * bm * 4;
    while (fixed + 1024 > budget && depth_cap > 1) {     // a tight budget: record shallower chains
        depth_cap = depth_cap / 2;                         // (deeper rows are walked a second time)
        fixed = base + size_t(depth_cap) * bm * 4;
    }
    const bool fits = fixed + 1024 <= budget;
    const size_t cap = fits ? (budget - fixed) / 4 : 0;
    const int par_cap = int(cap < size_t(n_nodes) ? cap : size_t(n_nodes));
    const size_t smem = std::max(fixed + size_t(par_cap) * 4, set ? ((size_t(n_nodes) * 4 + 15) & ~size_t(15)) + sizeof(AncestorSet) : 0);
    // Large trees: when a block's share of the parent array outgrows what one pass of the CTA stages in the
    // time a climb through L2 takes (see precompute_wide_kernel).  A bound of more than 128 ancestors, and more
    // than two to a row, is for deep trees, which that kernel climbs twice through L2 (its masks are not
    // inherited): where the staging kernel needs a single wave it stays (9400 nodes, block_m 64: depth 100 25 us
    // against 35, depth 500 118 against 130, parents drawn from the 256 nodes before 26 against 43; in two waves
    // 46 against 35 and 229 against 129; with a bound of 128 a tree of depth 15 takes 17 against 12.6, of depth 64
    // 21.2 against 22.8).
    const int slot = current_device_slot();
    if (slot < 0) return cudaErrorInvalidDevice;
    const bool one_wave = fits && size_t(nb) * n_trees <= sm_count() * (228 * 1024 / (smem + 1024));
    if (n_nodes > kWideNodes && !(one_wave && ma > std::max(128, 2 * bm))) {
        const size_t Ww = (W + 32 * WIDE_WARPS - 1) / (32 * WIDE_WARPS) * (32 * WIDE_WARPS);
        const bool inherit = ma <= 128 && !few;           // masks of all slots: 2 KB, two words per thread
        const size_t wide_smem = std::max(wide_smem_words(Ww, bm, ma, inherit) * 4, few ? sizeof(AncestorSet) : 0);
        if (wide_smem <= budget) {
            auto kernel = few ? precompute_wide_kernel<true> : precompute_wide_kernel<false>;
            std::atomic<size_t> &enabled = g_wide_smem_set[few ? 1 : 0][slot];
            if (wide_smem > 48 * 1024 && wide_smem > enabled.load(std::memory_order_acquire)) {
                cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(wide_smem));
                if (e != cudaSuccess) return e;
                enabled.store(wide_smem, std::memory_order_release);
            }
            kernel<<<dim3(nb, n_trees), WIDE_THREADS, wide_smem, stream>>>(
                parent, n_nodes, bm, ma, inherit ? 1 : 0, anc_idx, anc_mask, leaf_idx, static_cast<unsigned char *>(packed),
                packed_stride, status);
            return cudaGetLastError();
        }
    }
    if (!fits) return cudaErrorInvalidConfiguration;
    auto kernel = set ? precompute_kernel<true, true> : byte_flags ? precompute_kernel<true, false> : precompute_kernel<false, false>;
    std::atomic<size_t> &enabled = g_pre_smem_set[set ? 2 : byte_flags ? 1 : 0][slot];
    if (smem > 48 * 1024 && smem > enabled.load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
        enabled.store(smem, std::memory_order_release);
    }
    dim3 grid(nb, n_trees);
    kernel<<<grid, PRE_THREADS, smem, stream>>>(
        parent, n_nodes, bm, ma, par_cap, depth_cap, anc_idx, anc_mask, leaf_idx,
        static_cast<unsigned char *>(packed), packed_stride, status);
    return cudaGetLastError();
}

cudaError_t launch_pack(const int64_t *anc_idx, const uint8_t *anc_mask, const int64_t *leaf_idx,
                        int n_trees, int nb, int bm, int ma, int64_t index_base, void *packed,
                        size_t packed_stride, int32_t *status, cudaStream_t stream) {
    const size_t words = size_t(bm) * ((ma + 31) / 32 + (bm + 31) / 32);
    const bool wide = words <= 8192 && ma % 16 == 0 && (reinterpret_cast<uintptr_t>(anc_mask) & 15) == 0;
    const size_t smem = size_t(ma) * 4 + (wide ? words * 4 : 0);
    const int slot = current_device_slot();
    if (slot < 0) return cudaErrorInvalidDevice;
    if (smem > 48 * 1024 && smem > g_pack_smem_set[slot].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(pack_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
        g_pack_smem_set[slot].store(smem, std::memory_order_release);
    }
    dim3 grid(nb, n_trees);
    pack_kernel<<<grid, PACK_THREADS, smem, stream>>>(
        anc_idx, anc_mask, leaf_idx, bm, ma, index_base, static_cast<unsigned char *>(packed),
        packed_stride, status, wide ? int(words) : 0);
    return cudaGetLastError();
}

}  // namespace fst
