// Tree attention, fp32-arithmetic kernel for every dtype and head_dim in {16,32,64,128}.
//
// Computes what the reference's _fwd_kernel computes (fstattention.py:21-151): for each query
// row of a block, softmax over {its ancestors outside the block, from the block's gathered
// list} + {itself and its ancestors inside the block} + {every shared-prefix row}, times V.
// Online softmax in base 2 (scores are scaled by sm_scale*log2(e) like fstattention.py:59).  All
// arithmetic is fp32, so fp32 inputs keep fp32 accuracy; this is the kernel for fp32 tensors,
// small head dimensions and odd block sizes.  The tensor-core kernels cover fp16/bf16 at D=64/128.
//
// What bounds it is latency: a row attends to a handful of keys.  So every row has a warp of its
// own, only keys whose mask bit is set are touched (the warp first compacts the row's mask words
// into a list), a key's row is read by D / 4 lanes with one wide load each - coalesced, and at
// D < 128 several keys side by side, each group of lanes with its own running softmax, merged at
// the end - and a batch of keys' K and V loads is in flight at once.  31-node tree, 4 heads, D 64,
// fp32: 38.7 us with one key per lane and four rows per warp one after another, 5 us now.

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <initializer_list>

#include "fst_common.cuh"

namespace fst {

constexpr int SIMT_WARPS = 8;          // rows per CTA
constexpr int SIMT_LIST = 128;         // keys a warp lists before it works them off

template <typename T> __device__ inline float to_float(T x);
template <> __device__ inline float to_float<float>(float x) { return x; }
template <> __device__ inline float to_float<__half>(__half x) { return __half2float(x); }
template <> __device__ inline float to_float<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T> __device__ inline T from_float(float x);
template <> __device__ inline float from_float<float>(float x) { return x; }
template <> __device__ inline __half from_float<__half>(float x) { return __float2half_rn(x); }
template <> __device__ inline __nv_bfloat16 from_float<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// four consecutive elements of a row as floats; VEC: the address is aligned to all four of them
template <typename T, bool VEC>
__device__ __forceinline__ float4 load4(const T *p) {
    if constexpr (!VEC) {
        return make_float4(to_float(p[0]), to_float(p[1]), to_float(p[2]), to_float(p[3]));
    } else if constexpr (sizeof(T) == 4) {
        return *reinterpret_cast<const float4 *>(p);
    } else {
        const uint2 raw = *reinterpret_cast<const uint2 *>(p);
        const T *e = reinterpret_cast<const T *>(&raw);
        return make_float4(to_float(e[0]), to_float(e[1]), to_float(e[2]), to_float(e[3]));
    }
}

template <typename T, int D, bool VEC>
__global__ void __launch_bounds__(SIMT_WARPS * 32)
attn_simt_kernel(const AttnArgs a) {
    constexpr int LPK = D / 4;                        // lanes per key
    constexpr int G = 32 / LPK;                       // keys side by side
    constexpr int U = D == 128 ? 8 : 4;               // keys in flight per group
    __shared__ int s_list[SIMT_WARPS][SIMT_LIST];
    const int h = blockIdx.y, z = blockIdx.z;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int grp = lane / LPK, d0 = (lane % LPK) * 4;
    const int row = blockIdx.x * SIMT_WARPS + wid;
    if (row >= a.n_q) return;                         // warps are on their own from here on
    const int b = row / a.bm, j = row - b * a.bm;

    const PackedLayout L = packed_layout(a.nb, a.bm, a.ma);
    const unsigned char *blob = a.packed + size_t(z) * a.meta_stride;
    const int count = min(max(reinterpret_cast<const int32_t *>(blob + L.off_count)[b], 0), a.ma);
    const int32_t *idx = reinterpret_cast<const int32_t *>(blob + L.off_idx) + size_t(b) * a.ma;
    const uint32_t *emask = reinterpret_cast<const uint32_t *>(blob + L.off_emask) + (size_t(b) * a.bm + j) * L.maw;
    const uint32_t *bmask = reinterpret_cast<const uint32_t *>(blob + L.off_bmask) + (size_t(b) * a.bm + j) * L.bw;

    const int hk = h / a.kv_group;                    // my K/V head
    const T *kp = static_cast<const T *>(a.k) + z * a.ks_z + hk * a.ks_h + d0;
    const T *vp = static_cast<const T *>(a.v) + z * a.vs_z + hk * a.vs_h + d0;
    const float4 q = load4<T, VEC>(static_cast<const T *>(a.q) + z * a.qs_z + h * a.qs_h + row * a.qs_n + d0);

    float m = -INFINITY, l = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    // one step of my group's online softmax over up to U keys (K/V rows; -1: none)
    auto absorb = [&](const long long (&key)[U]) {
        float4 kr[U], vr[U];
        float s[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            kr[u] = vr[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (key[u] >= 0) {
                kr[u] = load4<T, VEC>(kp + key[u] * a.ks_n);
                vr[u] = load4<T, VEC>(vp + key[u] * a.vs_n);
            }
        }
        float mn = m;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float dot = q.x * kr[u].x;
            dot = fmaf(q.y, kr[u].y, dot);
            dot = fmaf(q.z, kr[u].z, dot);
            dot = fmaf(q.w, kr[u].w, dot);
#pragma unroll
            for (int o = LPK / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            s[u] = key[u] >= 0 ? dot * a.scale_log2 : -INFINITY;
            mn = fmaxf(mn, s[u]);
        }
        // No key so far, or none with a score above -inf: weights of zero - but a NaN score, which no maximum shows,
        // is a NaN weight, and the row's result is NaN.
        const float base = mn == -INFINITY ? 0.f : mn;
        const float alpha = exp2f(m - base);
        l *= alpha;
        acc.x *= alpha; acc.y *= alpha; acc.z *= alpha; acc.w *= alpha;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float p = exp2f(s[u] - base);
            l += p;
            acc.x = fmaf(p, vr[u].x, acc.x); acc.y = fmaf(p, vr[u].y, acc.y);
            acc.z = fmaf(p, vr[u].z, acc.z); acc.w = fmaf(p, vr[u].w, acc.w);
        }
        m = mn;
    };

    // the row's keys, compacted 32 mask bits at a time and worked off when the list fills up
    int listed = 0;
    int *list = s_list[wid];
    auto flush = [&]() {
        __syncwarp();
        for (int i0 = 0; i0 < listed; i0 += G * U) {
            long long key[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * G + grp;
                key[u] = i < listed ? (long long)a.prefix + list[i] : -1LL;
            }
            absorb(key);
            __syncwarp();
        }
        listed = 0;
    };
    auto append = [&](bool on, int node) {
        const uint32_t votes = __ballot_sync(0xffffffffu, on);
        if (listed + __popc(votes) > SIMT_LIST) flush();
        if (on) list[listed + __popc(votes & ((1u << lane) - 1u))] = node;
        listed += __popc(votes);
    };
    for (int c0 = 0; c0 < a.bm; c0 += 32) {           // the row itself and ancestors in the block
        const int c = c0 + lane, node = b * a.bm + c;
        append(c < a.bm && ((bmask[c0 >> 5] >> lane) & 1u) && node < a.n_q, node);
    }
    for (int a0 = 0; a0 < count; a0 += 32) {          // external ancestors, gated by mask bits
        const int s = a0 + lane;
        const int node = s < count ? idx[s] : -1;
        bool on = s < count && ((emask[a0 >> 5] >> lane) & 1u);
        if (on && (node < 0 || node >= a.n_q)) {
            report(a.status, FST_DEV_INDEX_RANGE, b, s);
            on = false;
        }
        append(on, node);
    }
    flush();
    for (int p0 = 0; p0 < a.prefix; p0 += G * U) {    // shared prefix, dense
        long long key[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int p = p0 + u * G + grp;
            key[u] = p < a.prefix ? (long long)p : -1LL;
        }
        absorb(key);
        __syncwarp();
    }

    // merge the groups
#pragma unroll
    for (int o = LPK; o < 32; o <<= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
        const float4 c2 = make_float4(__shfl_xor_sync(0xffffffffu, acc.x, o), __shfl_xor_sync(0xffffffffu, acc.y, o),
                                      __shfl_xor_sync(0xffffffffu, acc.z, o), __shfl_xor_sync(0xffffffffu, acc.w, o));
        const float mn = fmaxf(m, m2);
        const float w = m == -INFINITY ? 0.f : exp2f(m - mn), w2 = m2 == -INFINITY ? 0.f : exp2f(m2 - mn);
        l = l * w + l2 * w2;
        acc.x = acc.x * w + c2.x * w2; acc.y = acc.y * w + c2.y * w2;
        acc.z = acc.z * w + c2.z * w2; acc.w = acc.w * w + c2.w * w2;
        m = mn;
    }
    const float inv = l > 0.f ? 1.f / l : 0.f;
    if (grp == 0) {
        T *op = static_cast<T *>(a.o) + z * a.os_z + h * a.os_h + row * a.os_n + d0;
        if constexpr (VEC && sizeof(T) == 4) {
            *reinterpret_cast<float4 *>(op) = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
        } else {
            op[0] = from_float<T>(acc.x * inv);
            op[1] = from_float<T>(acc.y * inv);
            op[2] = from_float<T>(acc.z * inv);
            op[3] = from_float<T>(acc.w * inv);
        }
    }
    if (a.lse && lane == 0)
        a.lse[(size_t(z) * a.H + h) * a.n_q + row] = m + log2f(l);
}

template <typename T, int D>
static cudaError_t launch_simt_d(const AttnArgs &a, cudaStream_t stream) {
    // four elements per load where every row and head starts on such a boundary, else one by one
    const uintptr_t piece = 4 * sizeof(T);
    bool vec = true;
    for (const void *p : {a.q, a.k, a.v, (const void *)a.o}) vec = vec && reinterpret_cast<uintptr_t>(p) % piece == 0;
    for (int64_t s : {a.qs_z, a.qs_h, a.qs_n, a.ks_z, a.ks_h, a.ks_n, a.vs_z, a.vs_h, a.vs_n, a.os_z, a.os_h, a.os_n})
        vec = vec && s % 4 == 0;
    dim3 grid((a.n_q + SIMT_WARPS - 1) / SIMT_WARPS, a.H, a.Z), block(SIMT_WARPS * 32);
    if (vec) attn_simt_kernel<T, D, true><<<grid, block, 0, stream>>>(a);
    else attn_simt_kernel<T, D, false><<<grid, block, 0, stream>>>(a);
    return cudaGetLastError();
}

template <typename T>
static cudaError_t launch_simt_t(const AttnArgs &a, cudaStream_t stream) {
    switch (a.D) {
        case 16: return launch_simt_d<T, 16>(a, stream);
        case 32: return launch_simt_d<T, 32>(a, stream);
        case 64: return launch_simt_d<T, 64>(a, stream);
        case 128: return launch_simt_d<T, 128>(a, stream);
        default: return cudaErrorNotSupported;
    }
}

cudaError_t launch_attention_simt(const AttnArgs &a, int dtype, cudaStream_t stream) {
    switch (dtype) {
        case FST_F16: return launch_simt_t<__half>(a, stream);
        case FST_BF16: return launch_simt_t<__nv_bfloat16>(a, stream);
        case FST_F32: return launch_simt_t<float>(a, stream);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace fst
