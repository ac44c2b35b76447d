// Tree construction on the device: from the top-k candidate scores of the speculation heads to
// a parent array, without a host round trip.
//
// The reference only builds a fixed synthetic forest on the CPU (create_tree, utils.py:27-77):
// topk roots, level sizes size[l] = topk * int(size[l-1] * left_weight_factor), node r of a level
// hanging under node r / topk of the level above - a "left-weighted" tree in which only the
// first part of every level is expanded.  Its README (README.md:17) names the use: Medusa-style
// trees, the cartesian products of every head's top-k candidates.  This kernel is that
// construction driven by scores: head l gives topk candidate scores (log-probabilities, any
// order), a node's score is the sum along its path, and of every level the
// int(size * left_weight_factor) best nodes are expanded, best first, each into the topk
// candidates of the next head.  With equal scores "best" falls back to position and the result
// is exactly create_tree's forest.  Node numbering is level by level, so parents precede their
// children and fst_dfs_order / fst_precompute can take the array as it is.
//
// One CTA per tree.  A level is at most LEVEL_CAP nodes, in shared memory.  The order is total (ties broken by
// position, the one a stable sort would give), and a node's place in it is the count of the nodes that beat it.
// No pairs are compared for that: a level was written parent by parent, best parent first, so the nodes that
// took candidate k of the head are a descending list for every k, those of a list that beat a given node
// are its first ones, and a binary search per list counts them.  The thread that ranked a node writes
// its children: a level costs one barrier and a chain of log2(parents) shared-memory reads.  Counting all
// pairs took 10.2 us for four trees of 1020 nodes (depth 7, top 4) and grew with the square of a level.

#include "fst_common.cuh"

namespace fst {

constexpr int BUILD_THREADS = 512;
constexpr int LEVEL_CAP = 4096;
constexpr int HEAD_CAP = 1024;         // candidate scores kept in shared memory

struct LevelPlan {
    int n_levels;                       // depth + 1
    int size[kMaxTreeLevels];           // nodes of level l
    int start[kMaxTreeLevels + 1];      // first node of level l; start[n_levels] = node count
    // how level l is ranked: its nodes are topk lists of len[l]; half[l] is the largest power of two that is no
    // longer, and 1 << share[l] threads of a warp divide a node's lists among themselves
    int len[kMaxTreeLevels], half[kMaxTreeLevels], share[kMaxTreeLevels];
};

__global__ void __launch_bounds__(BUILD_THREADS)
build_tree_topk_kernel(const float *__restrict__ scores_all, int topk, LevelPlan plan, int max_nodes,
                       int32_t *__restrict__ parent_all, int32_t *__restrict__ choice_all,
                       float *__restrict__ node_score_all) {
    __shared__ float levels[2][LEVEL_CAP];                // path scores of the previous / the new level
    __shared__ float heads[HEAD_CAP];
    const int tree = blockIdx.x, tid = threadIdx.x;
    const float *scores = scores_all + size_t(tree) * plan.n_levels * topk;
    // all heads' scores at once: fetched level by level, each level would wait a memory latency for its topk numbers
    if (plan.n_levels * topk <= HEAD_CAP) {
        for (int i = tid; i < plan.n_levels * topk; i += BUILD_THREADS) heads[i] = scores[i];
        scores = heads;
        __syncthreads();
    }
    int32_t *parent = parent_all + size_t(tree) * max_nodes;
    int32_t *choice = choice_all ? choice_all + size_t(tree) * max_nodes : nullptr;
    float *node_score = node_score_all ? node_score_all + size_t(tree) * max_nodes : nullptr;

    for (int i = tid; i < plan.size[0]; i += BUILD_THREADS) {
        const float s = scores[i];
        levels[0][i] = s;
        if (i < max_nodes) {
            parent[i] = -1;
            if (choice) choice[i] = i;
            if (node_score) node_score[i] = s;
        }
    }
    // rows past the last node of the forest (a caller with fixed-size tensors): isolated roots
    for (int i = plan.start[plan.n_levels] + tid; i < max_nodes; i += BUILD_THREADS) {
        parent[i] = -1;
        if (choice) choice[i] = -1;
        if (node_score) node_score[i] = -INFINITY;
    }
    __syncthreads();
    // level l - 1 is topk descending lists: list k is entries k, k + topk, ...  (of the roots: one entry each)
#pragma unroll 1
    for (int l = 1; l < plan.n_levels; ++l) {
        const int prev = plan.size[l - 1], len = plan.len[l - 1], half = plan.half[l - 1], shift = plan.share[l - 1];
        const int here = plan.size[l], first = plan.start[l], from = plan.start[l - 1];
        const float *c = levels[(l - 1) & 1], *head = scores + l * topk;
        float *nxt = levels[l & 1];
        const int part = tid & ((1 << shift) - 1);
#pragma unroll 1
        for (int i0 = (tid & ~31) >> shift; i0 < prev; i0 += BUILD_THREADS >> shift) {     // whole warps
            const int i = i0 + ((tid & 31) >> shift);
            const float mine = i < prev ? c[i] : 0.f;
            int rank = 0;                                 // nodes that beat mine
#pragma unroll 2
            for (int k = part; k < topk; k += 1 << shift) {
                int n = 0;                                // of list k
                for (int step = half; step > 0; step >>= 1) {
                    const int at = min(n + step - 1, len - 1) * topk + k;
                    const float s = c[at];
                    const bool beats = s > mine || (s == mine && at < i);
                    n += n + step <= len && beats ? step : 0;
                }
                rank += n;
            }
            for (int o = (1 << shift) >> 1; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
            rank *= topk;                                 // my first child in the new level
            if (i >= prev || rank >= here) continue;      // not expanded
            for (int k = part; k < topk; k += 1 << shift) {
                const float s = mine + head[k];
                const int node = first + rank + k;
                nxt[rank + k] = s;
                if (node < max_nodes) {
                    parent[node] = from + i;
                    if (choice) choice[node] = l * topk + k;
                    if (node_score) node_score[node] = s;
                }
            }
        }
        __syncthreads();
    }
}

// Level sizes of the forest (the reference's recurrence, utils.py:46-52, in the same double
// arithmetic Python uses).  Returns the node count, or -1 when a level outgrows the kernel.
static long long plan_levels(int depth, int topk, double left_weight_factor, LevelPlan *plan) {
    if (depth < 0 || depth + 1 > kMaxTreeLevels || topk < 1) return -1;
    long long total = 0;
    long long sz = topk;
    for (int l = 0; l <= depth; ++l) {
        if (l > 0) sz = (long long)topk * (long long)(double(sz) * left_weight_factor);
        if (sz < 0 || sz > LEVEL_CAP) return -1;
        if (plan) {
            plan->size[l] = int(sz);
            plan->start[l] = int(total);
        }
        total += sz;
    }
    if (plan) {
        for (int l = 0; l <= depth; ++l) {
            const int n = plan->size[l];
            plan->len[l] = n / topk;
            plan->half[l] = 1;
            while (plan->half[l] * 2 <= plan->len[l]) plan->half[l] *= 2;
            plan->share[l] = 0;
            for (int t = 2; t <= 32 && t <= topk && n * t <= BUILD_THREADS; t *= 2) ++plan->share[l];
        }
        plan->n_levels = depth + 1;
        plan->start[depth + 1] = int(total);
    }
    return total;
}

long long tree_topk_nodes(int depth, int topk, double left_weight_factor) {
    return plan_levels(depth, topk, left_weight_factor, nullptr);
}

cudaError_t launch_build_tree_topk(const float *scores, int n_trees, int depth, int topk,
                                   double left_weight_factor, int max_nodes, int32_t *parent, int32_t *choice,
                                   float *node_score, cudaStream_t stream) {
    LevelPlan plan;
    const long long total = plan_levels(depth, topk, left_weight_factor, &plan);
    if (total < 0) return cudaErrorInvalidConfiguration;
    build_tree_topk_kernel<<<n_trees, BUILD_THREADS, 0, stream>>>(scores, topk, plan, max_nodes, parent, choice,
                                                                  node_score);
    return cudaGetLastError();
}

}  // namespace fst
