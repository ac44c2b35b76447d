// Depth-first renumbering of a tree on the device.
//
// The reference leaves node ordering as a TODO (README.md:19-20): its precompute
// (utils.py:104-129) takes whatever numbering the caller has, and with a breadth-first numbering
// a 64-row block of a deep tree has ancestors all over the tree.  Numbered depth first (pre-order,
// children in their old relative order) a block is a few root-to-leaf paths and gathers a
// fraction of the rows.  This kernel computes that numbering from a parent array that is already
// on the GPU, so a decoder that builds its tree on the device never goes back to the host:
//     order[i]      = old index of the node that becomes node i
//     new_parent[i] = its parent in the new numbering (still < i, or -1)
// One CTA per tree, everything in shared memory, integer arithmetic only.  Every step takes a number of
// rounds that is the logarithm of the depth, or the depth, never the number of nodes:
//   1. depth[i]: pointer doubling;
//   2. size[a], nodes in the subtree of a: one level at a time from the deepest up, each node adding
//      its own total to its parent;
//   3. off[i], sizes of the siblings of i with a smaller index (roots are siblings of one another): every
//      node walks its parent's list of children; where a node has too many children for that, one
//      warp sweeps the nodes in index order instead, 32 at a time, with a running sum per parent;
//   4. pos[i] = sum over i and its ancestors a of (off[a] + 1), less one: pointer doubling again;
//   5. scatter.
// (Every node climbing to its root with an atomic at every step, and the sweep for every tree, took 19.8 us
// for four trees of 1020 nodes; this takes 6.)
// A malformed parent (parent[i] >= i or < -1) is reported through the status record and the
// outputs are left untouched.

#include "fst_common.cuh"

namespace fst {

constexpr int REORDER_THREADS = 1024;
constexpr int REORDER_MAX_NODES = 8192;                   // six int arrays of that many nodes in shared memory
constexpr int REORDER_SIBLINGS = 48;                      // longest list of children that is walked

// PER: nodes per thread
template <int PER>
__global__ void __launch_bounds__(REORDER_THREADS)
dfs_order_kernel(const int32_t *__restrict__ parent, int n, int32_t *__restrict__ order,
                 int32_t *__restrict__ new_parent, int32_t *status) {
    extern __shared__ int32_t rs[];
    int32_t *par = rs;                                    // [n]
    int32_t *size = par + n;                              // [n]   subtree sizes
    int32_t *jump = size + n;                             // [n]   doubling: an ancestor, 2^round levels up
    int32_t *val = jump + n;                              // [n]   doubling: sum up to (not including) that ancestor
    int32_t *head = val + n;                              // [n+1] first child in the list; slot n = the roots
    int32_t *next = head + n + 1;                         // [n]   next sibling in the list
    __shared__ int bad, deepest, crowd;
    const int tree = blockIdx.x, tid = threadIdx.x;
    const int32_t *src = parent + size_t(tree) * n;
    if (tid == 0) bad = deepest = crowd = 0;
    __syncthreads();
    int32_t p0[PER];                                      // loads of all my nodes under way at once
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = tid + k * REORDER_THREADS;
        p0[k] = i < n ? __ldg(src + i) : -1;
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = tid + k * REORDER_THREADS;
        if (i >= n) break;
        const int32_t p = p0[k];
        if (p >= i || p < -1) {
            report(status, FST_DEV_MALFORMED_TREE, i, int(p));
            bad = 1;
        }
        par[i] = jump[i] = p;
        size[i] = 1;
        val[i] = 1;
        head[i] = -1;
    }
    if (tid == 0) head[n] = -1;
    __syncthreads();
    if (bad) return;                                      // everything below relies on parent[i] < i

    // val[i] becomes the sum of the first values of i and all its ancestors
    auto doubling = [&]() {
        for (;;) {
            int32_t j[PER], v[PER];
            bool any = false;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = tid + k * REORDER_THREADS;
                j[k] = i < n ? jump[i] : -1;
                v[k] = 0;
                if (j[k] >= 0) {
                    v[k] = val[j[k]];
                    j[k] = jump[j[k]];
                    any = true;
                }
            }
            if (!__syncthreads_or(any)) return;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int i = tid + k * REORDER_THREADS;
                if (i < n) {
                    val[i] += v[k];
                    jump[i] = j[k];
                }
            }
            __syncthreads();
        }
    };
    doubling();                                           // val: depth + 1

    int32_t depth[PER];
    int mine = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = tid + k * REORDER_THREADS;
        depth[k] = i < n ? val[i] - 1 : 0;
        mine = max(mine, depth[k]);
        // the children's lists, in whatever order the exchanges come
        if (i < n) next[i] = atomicExch(&head[par[i] < 0 ? n : par[i]], i);
    }
    atomicMax(&deepest, int(__reduce_max_sync(0xffffffffu, unsigned(mine))));
    __syncthreads();
    for (int level = deepest; level > 0; --level) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int i = tid + k * REORDER_THREADS;
            if (depth[k] == level && i < n) atomicAdd(&size[par[i]], size[i]);
        }
        __syncthreads();
    }

    // sizes of earlier siblings
    bool long_list = false;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = tid + k * REORDER_THREADS;
        if (i >= n) break;
        int32_t before = 0;
        int steps = 0;
        for (int c = head[par[i] < 0 ? n : par[i]]; c >= 0 && steps <= REORDER_SIBLINGS; c = next[c], ++steps)
            if (c < i) before += size[c];
        long_list = long_list || steps > REORDER_SIBLINGS;
        val[i] = before + 1;
        jump[i] = par[i];
    }
    if (long_list) crowd = 1;
    __syncthreads();
    if (crowd) {                                          // somebody has more children than a walk is good for
        for (int i = tid; i <= n; i += REORDER_THREADS) head[i] = 0;  // running sum per parent
        __syncthreads();
        if (tid < 32) {
            const int lane = tid;
            for (int base = 0; base < n; base += 32) {
                const int i = base + lane;
                const int32_t p = i < n ? par[i] : -2;    // -2 matches no real parent
                const int32_t sz = i < n ? size[i] : 0;
                int32_t before = 0, total = 0;
                bool first = true;                        // lowest lane of its sibling group
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const int32_t pj = __shfl_sync(0xffffffffu, p, j), sj = __shfl_sync(0xffffffffu, sz, j);
                    if (pj == p) {
                        total += sj;
                        if (j < lane) {
                            before += sj;
                            first = false;
                        }
                    }
                }
                const int slot = p < 0 ? n : p;
                if (i < n) val[i] = head[slot] + before + 1;
                __syncwarp();
                if (i < n && first) head[slot] += total;
                __syncwarp();
            }
        }
        __syncthreads();
    }
    doubling();                                           // val: final position + 1

    int32_t *ord = order + size_t(tree) * n, *npar = new_parent + size_t(tree) * n;
    for (int i = tid; i < n; i += REORDER_THREADS) {
        const int32_t at = val[i] - 1, p = par[i];
        ord[at] = i;
        npar[at] = p < 0 ? -1 : val[p] - 1;
    }
}

template <int PER>
static cudaError_t launch_dfs_order_per(const int32_t *parent, int n_trees, int n_nodes, int32_t *order,
                                        int32_t *new_parent, int32_t *status, cudaStream_t stream) {
    const size_t smem = (size_t(n_nodes) * 6 + 1) * sizeof(int32_t);
    static DeviceOnce configured;
    const cudaError_t e = configured.run([&] {
        return cudaFuncSetAttribute(dfs_order_kernel<PER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    int((size_t(PER) * REORDER_THREADS * 6 + 1) * sizeof(int32_t)));
    });
    if (e != cudaSuccess) return e;
    dfs_order_kernel<PER><<<n_trees, REORDER_THREADS, smem, stream>>>(parent, n_nodes, order, new_parent, status);
    return cudaGetLastError();
}

cudaError_t launch_dfs_order(const int32_t *parent, int n_trees, int n_nodes, int32_t *order,
                             int32_t *new_parent, int32_t *status, cudaStream_t stream) {
    if (n_nodes > REORDER_MAX_NODES) return cudaErrorInvalidValue;
    const int per = (n_nodes + REORDER_THREADS - 1) / REORDER_THREADS;
    auto launch = per <= 1 ? launch_dfs_order_per<1> : per <= 2 ? launch_dfs_order_per<2>
                : per <= 4 ? launch_dfs_order_per<4> : launch_dfs_order_per<REORDER_MAX_NODES / REORDER_THREADS>;
    return launch(parent, n_trees, n_nodes, order, new_parent, status, stream);
}

}  // namespace fst
