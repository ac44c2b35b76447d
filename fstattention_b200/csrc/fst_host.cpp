// Host path of the Python package: tensors in, library calls out.
//
// A decoder calls fst_attention once per layer and the attention of a small tree takes about 5 us
// on the GPU, so what a call costs on the host decides the step time of eager programs: reading
// shapes, strides and pointers through Python attributes, building two dozen ctypes arguments and
// allocating through the dispatcher took 12-15 us per call.  Here the same checks and the same
// library calls (include/fstattn_b200.h) are made from C++ on the tensors' own fields.
//
// Everything follows torch's rules: outputs and workspaces come from torch's caching allocator on
// the current stream, launches go to the current stream of q's device, errors are Python
// exceptions.  Nothing here computes anything.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <atomic>
#include <cmath>
#include <mutex>
#include <optional>
#include <vector>

#include "fst_plan.h"
#include "fstattn_b200.h"

namespace {

struct PyError {};                                        // a Python exception is set

[[noreturn]] void raise(PyObject *type, const char *what) {
    PyErr_SetString(type, what);
    throw PyError{};
}
void check_status(int rc, const char *what) {
    if (rc == FST_OK) return;
    PyErr_Format(PyExc_RuntimeError, "%s: %s (status %d)", what, fst_status_string(rc), rc);
    throw PyError{};
}

// ---- argument access -------------------------------------------------------------------------
const at::Tensor &tensor(PyObject *o) {
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "a torch.Tensor is expected");
    return THPVariable_Unpack(o);
}
long long integer(PyObject *o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PyError{};
    return v;
}
double real(PyObject *o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PyError{};
    return v;
}

at::Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Device &dev) {
    return at::detail::empty_cuda(size, type, dev, std::nullopt);
}

// Tensors that outlive the call and are written in place later - metadata, whose versions say whether anybody has, and status
// records - are ordinary ones also when the call is made under torch.inference_mode().
struct OrdinaryTensors {
    c10::InferenceMode off{false};
};

// Attention launches on a device share one status record (the first problem seen stays until it
// is cleared).  Records live as long as the process.
at::Tensor *const *status_slots() {
    static at::Tensor *slots[64] = {};
    return slots;
}
at::Tensor *status_of(const at::Device &dev, bool create) {
    static std::mutex mutex;
    at::Tensor **slots = const_cast<at::Tensor **>(status_slots());
    const int i = dev.index();
    if (i < 0 || i >= 64) raise(PyExc_RuntimeError, "device index out of range");
    std::lock_guard<std::mutex> lock(mutex);
    if (slots[i] == nullptr && create) {
        const OrdinaryTensors guard;
        slots[i] = new at::Tensor(at::zeros({4}, at::TensorOptions().dtype(at::kInt).device(dev)));
    }
    return slots[i];
}

int sm_count(int device) {
    constexpr int kB200 = 148;
    static std::atomic<int> cached[64];
    if (device < 0) return kB200;                         // the tensor is on the host
    int n = cached[device & 63].load(std::memory_order_acquire);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) {
            cudaGetLastError();                           // or torch would report it after its next launch
            n = kB200;
        }
        cached[device & 63].store(n, std::memory_order_release);
    }
    return n;
}

// ---- the runs a shared prefix is cut into -------------------------------------------------------
// Only the tensor-core kernels split.  With head_dim 64 or 128, a positive scale and as many prefix rows as
// prefix_umma_pays asks for, the call goes to the tcgen05 kernel (fst_plan.h says in how many runs).  Otherwise
// the tree kernel walks the prefix itself: split to about four CTAs per SM, or, where the tcgen05 kernel is
// ruled out by the scale alone, in runs of 256 rows to about one CTA per SM and 128 query rows (8 heads of
// 127 rows behind 4096: 21.8 us, 125 unsplit).
struct Splits {
    int runs;
    bool workspace;
    bool umma = false;                                    // the tcgen05 prefix kernel takes the call
};
Splits pick_splits(const std::optional<long long> &asked, at::ScalarType type, int64_t Z, int64_t H, int64_t H_kv, int64_t n_q,
                   int64_t D, int64_t prefix, int64_t block_m, double scale, int kernel, int device) {
    if ((type != at::kHalf && type != at::kBFloat16) || (D != 64 && D != 128) ||
        (block_m != 32 && block_m != 64 && block_m != 128) || kernel == FST_KERNEL_SIMT || kernel == FST_KERNEL_MMA ||
        prefix <= 0)
        return {1, false};
    const int64_t cap = 65535 / std::max<int64_t>(Z, 1);
    const auto clamp = [&](int64_t v) { return int(std::max<int64_t>(1, std::min(v, cap))); };
    if (kernel == FST_KERNEL_AUTO && scale <= 0.0 && prefix >= 256) {
        const int64_t tiles = Z * H * ((n_q + 127) / 128);
        const int runs = clamp(asked ? *asked : std::min(sm_count(device) / std::max<int64_t>(tiles, 1), prefix / 256));
        return {runs, runs > 1};
    }
    if (kernel == FST_KERNEL_TMA_UMMA || (kernel == FST_KERNEL_AUTO && fst::prefix_umma_pays(Z, H, H_kv, n_q, prefix, block_m, sm_count(device)))) {
        const fst::PrefixPlan plan = fst::prefix_plan(Z, H, H_kv, n_q, prefix, sm_count(device), true, asked ? clamp(*asked) : 0);
        return {plan.runs, plan.spread, true};
    }
    int runs;
    if (asked) {
        runs = clamp(*asked);
    } else {
        const int64_t ctas = Z * H * ((n_q + block_m - 1) / block_m);
        runs = clamp(std::min(4 * sm_count(device) / std::max<int64_t>(ctas, 1), prefix / 512));
    }
    return {runs, runs > 1};
}
std::optional<long long> optional_int(PyObject *o) {
    if (o == Py_None) return std::nullopt;
    return integer(o);
}

// ---- attention ----------------------------------------------------------------------------------
int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kHalf: return FST_F16;
        case at::kBFloat16: return FST_BF16;
        case at::kFloat: return FST_F32;
        default: return -1;
    }
}
// A kernel takes plain addresses: one of another device, or of the host, would be a fault there.
void on_device(const at::Tensor &t, const at::Device &dev) {
    if (t.device() != dev) raise(PyExc_RuntimeError, "all tensors of a call must be on one device");
}
void head_contiguous(const at::Tensor &t) {
    if (t.stride(3) != 1) raise(PyExc_ValueError, "the head dimension must be contiguous");
}

struct Call {
    at::Tensor q, k, v, o, lse;
    int64_t Z, H, H_kv, n_q, n_kv, D;
    float scale;
    int dtype;
};

// The checks every attention call makes, in the order callers rely on (the reference asserts the
// head dimensions, fstattention.py:155-157), and the output tensors.
Call open_call(PyObject *q, PyObject *k, PyObject *v, PyObject *out, PyObject *scale, bool want_lse) {
    Call c;
    c.q = tensor(q); c.k = tensor(k); c.v = tensor(v);
    if (c.q.dim() != 4 || c.k.dim() != 4 || c.v.dim() != 4) raise(PyExc_ValueError, "q, k, v must have four dimensions");
    c.D = c.q.size(3);
    if (c.D != c.k.size(3) || c.k.size(3) != c.v.size(3)) raise(PyExc_AssertionError, "q, k, v must have equal head dimensions");
    if (c.D != 16 && c.D != 32 && c.D != 64 && c.D != 128) raise(PyExc_AssertionError, "head dimension must be 16, 32, 64 or 128");
    if (!c.q.is_cuda() || !c.k.is_cuda() || !c.v.is_cuda())
        raise(PyExc_RuntimeError, "fst_attention runs on CUDA tensors only; there is no CPU path");
    on_device(c.k, c.q.device());
    on_device(c.v, c.q.device());
    const at::ScalarType type = c.q.scalar_type();
    c.dtype = dtype_code(type);
    if (c.dtype < 0 || c.k.scalar_type() != type || c.v.scalar_type() != type)
        raise(PyExc_TypeError, "q, k, v must share one dtype out of float16, bfloat16, float32");
    c.Z = c.q.size(0); c.H = c.q.size(1); c.n_q = c.q.size(2);
    c.H_kv = c.k.size(1); c.n_kv = c.k.size(2);
    if (c.k.size(0) != c.Z || c.v.sizes() != c.k.sizes() || c.n_kv < c.n_q || c.H_kv < 1 || c.H % c.H_kv)
        raise(PyExc_ValueError, "k and v must be [Z, H_kv, P + N, D] with P >= 0 and H a multiple of H_kv");
    if (out == Py_None) {
        c.o = c.q.is_contiguous() ? empty(c.q.sizes(), type, c.q.device()) : at::empty_like(c.q);
    } else {
        c.o = tensor(out);
        if (c.o.sizes() != c.q.sizes() || c.o.scalar_type() != type || !c.o.is_cuda()) raise(PyExc_ValueError, "out must match q");
        on_device(c.o, c.q.device());
    }
    const double s = real(scale);
    if (!std::isfinite(s)) raise(PyExc_ValueError, "sm_scale must be finite");
    c.scale = float(s);
    head_contiguous(c.q); head_contiguous(c.k); head_contiguous(c.v); head_contiguous(c.o);
    if (want_lse) c.lse = empty({c.Z * c.H, c.n_q}, at::kFloat, c.q.device());
    return c;
}
PyObject *results(const Call &c) {
    if (!c.lse.defined()) return THPVariable_Wrap(c.o);
    PyObject *o = THPVariable_Wrap(c.o), *l = THPVariable_Wrap(c.lse);
    PyObject *pair = PyTuple_Pack(2, o, l);
    Py_DECREF(o);
    Py_DECREF(l);
    return pair;
}
float *lse_ptr(const Call &c) { return c.lse.defined() ? static_cast<float *>(c.lse.data_ptr()) : nullptr; }

#define FST_STRIDES(t) (t).stride(0), (t).stride(1), (t).stride(2)

PyObject *launch(Call &c, const void *packed, size_t tree_stride, int64_t block_m, int64_t ma, int kernel,
                 const std::optional<long long> &kv_splits, void *status, void *stream) {
    const at::Device dev = c.q.device();
    const Splits sp = pick_splits(kv_splits, c.q.scalar_type(), c.Z, c.H, c.H_kv, c.n_q, c.D, c.n_kv - c.n_q, block_m,
                                  c.scale, kernel & FST_KERNEL_MASK, dev.index());
    at::Tensor ws;
    size_t ws_bytes = 0;
    if (sp.workspace) {
        ws_bytes = fst_attention_split_workspace_bytes(int(c.Z), int(c.H), int(c.n_q), int(c.D), sp.runs);
        ws = empty({int64_t(ws_bytes)}, at::kByte, dev);
    }
    int rc;
    {
        pybind11::gil_scoped_release no_gil;
        rc = fst_attention_fwd_gqa(c.q.data_ptr(), c.k.data_ptr(), c.v.data_ptr(), c.o.data_ptr(), lse_ptr(c), packed,
                                   tree_stride, int(c.Z), int(c.H), int(c.H_kv), int(c.n_q), int(c.n_kv), int(c.D),
                                   FST_STRIDES(c.q), FST_STRIDES(c.k), FST_STRIDES(c.v), FST_STRIDES(c.o), int(block_m),
                                   int(ma), c.scale, c.dtype, kernel, sp.runs, ws.defined() ? ws.data_ptr() : nullptr,
                                   ws_bytes, static_cast<int32_t *>(status), stream);
    }
    check_status(rc, "fst_attention_fwd");
    return results(c);
}

template <PyObject *(*F)(PyObject *const *, Py_ssize_t)>
PyObject *guarded(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    try {
        return F(args, n);
    } catch (const PyError &) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}
void want_args(Py_ssize_t n, Py_ssize_t want) {
    if (n != want) raise(PyExc_TypeError, "wrong number of arguments");
}

// attention(q, k, v, out, packed, tree_stride, n_trees, n_blocks, block_m, max_ancestors, sm_scale,
//           kernel, kv_splits, return_lse)
PyObject *attention(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 14);
    Call c = open_call(a[0], a[1], a[2], a[3], a[10], a[13] == Py_True);
    const int64_t n_trees = integer(a[6]), n_blocks = integer(a[7]), bm = integer(a[8]), ma = integer(a[9]);
    if (n_trees != 1 && n_trees != c.Z) raise(PyExc_ValueError, "metadata must describe one tree or one tree per batch element");
    if (n_blocks != (c.n_q + bm - 1) / bm) raise(PyExc_ValueError, "metadata block count does not match q");
    const at::Device dev = c.q.device();
    const c10::cuda::CUDAGuard guard(dev);
    on_device(tensor(a[4]), dev);
    void *status = status_of(dev, true)->data_ptr();
    void *stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    return launch(c, tensor(a[4]).data_ptr(), n_trees > 1 ? size_t(integer(a[5])) : 0, bm, ma, int(integer(a[11])),
                  optional_int(a[12]), status, stream);
}

// The reference's three tensors (fstattention.py:153) in packed form, one launch; index_base (the prefix
// length) is what the caller has added to the indices, as the reference's test does, sentinels included.
struct Packed {
    at::Tensor blob;
    size_t stride;
    int64_t n_trees;
};
Packed pack_reference(PyObject *idx, PyObject *mask, PyObject *leaf, int64_t Z, int64_t n_q, int64_t index_base, int64_t bm,
                      int64_t ma, const at::Device &dev, int32_t *status, void *stream) {
    if (mask == Py_None || leaf == Py_None) raise(PyExc_TypeError, "ancestor_mask and leaf_idx are required with plain tensors");
    at::Tensor ai = tensor(idx), am = tensor(mask), li = tensor(leaf);
    if (!ai.is_cuda() || !am.is_cuda() || !li.is_cuda())
        raise(PyExc_RuntimeError, "metadata tensors must be on the GPU (call .to('cuda') as the reference does)");
    for (const at::Tensor *t : {&ai, &am, &li}) on_device(*t, dev);
    if (bm <= 0 || ma <= 0) raise(PyExc_ValueError, "metadata shapes do not match BLOCK_M / MAX_ANCESTORS / q");
    const int64_t nb = (n_q + bm - 1) / bm, n_meta = ai.dim() == 3 ? ai.size(0) : 1;
    const auto shaped = [](const at::Tensor &t, at::IntArrayRef want) {
        return t.dim() >= int64_t(want.size()) && t.sizes().slice(t.dim() - want.size()) == want;
    };
    if (!shaped(ai, {nb, ma}) || !shaped(am, {nb, bm, ma}) || !shaped(li, {nb, bm}))
        raise(PyExc_ValueError, "metadata shapes do not match BLOCK_M / MAX_ANCESTORS / q");
    if (ai.scalar_type() != at::kLong || li.scalar_type() != at::kLong ||
        (am.scalar_type() != at::kBool && am.scalar_type() != at::kByte))
        raise(PyExc_TypeError, "metadata dtypes must be int64 / bool / int64");
    if (n_meta != 1 && n_meta != Z) raise(PyExc_ValueError, "metadata must describe one tree or one tree per batch element");
    if (am.numel() < n_meta * nb * bm * ma || li.numel() < n_meta * nb * bm)
        raise(PyExc_ValueError, "ancestor_mask and leaf_idx must describe as many trees as ancestor_idx");
    ai = ai.contiguous(); am = am.contiguous(); li = li.contiguous();
    Packed p;
    p.n_trees = n_meta;
    p.stride = fst_packed_meta_bytes(int(nb), int(bm), int(ma));
    p.blob = empty({n_meta, int64_t(p.stride)}, at::kByte, dev);
    check_status(fst_pack_metadata(static_cast<const int64_t *>(ai.data_ptr()), static_cast<const uint8_t *>(am.data_ptr()),
                                   static_cast<const int64_t *>(li.data_ptr()), int(n_meta), int(nb), int(bm), int(ma),
                                   index_base, p.blob.data_ptr(), p.stride, status, stream),
                 "fst_pack_metadata");
    return p;
}

// attention_ref(q, k, v, out, ancestor_idx, ancestor_mask, leaf_idx, block_m, max_ancestors, sm_scale,
//               kernel, kv_splits, return_lse)
PyObject *attention_ref(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 13);
    Call c = open_call(a[0], a[1], a[2], a[3], a[9], a[12] == Py_True);
    const at::Device dev = c.q.device();
    const c10::cuda::CUDAGuard guard(dev);
    int32_t *status = static_cast<int32_t *>(status_of(dev, true)->data_ptr());
    void *stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const int64_t bm = integer(a[7]), ma = integer(a[8]);
    const Packed p = pack_reference(a[4], a[5], a[6], c.Z, c.n_q, c.n_kv - c.n_q, bm, ma, dev, status, stream);
    return launch(c, p.blob.data_ptr(), p.n_trees > 1 ? p.stride : 0, bm, ma, int(integer(a[10])), optional_int(a[11]),
                  status, stream);
}

// pack(ancestor_idx, ancestor_mask, leaf_idx, Z, n_q, index_base, block_m, max_ancestors) -> (packed, tree_stride, n_trees)
PyObject *pack(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 8);
    const at::Device dev = tensor(a[0]).device();
    const c10::cuda::CUDAGuard guard(dev);
    const Packed p = pack_reference(a[0], a[1], a[2], integer(a[3]), integer(a[4]), integer(a[5]), integer(a[6]), integer(a[7]),
                                    dev, static_cast<int32_t *>(status_of(dev, true)->data_ptr()),
                                    c10::cuda::getCurrentCUDAStream(dev.index()).stream());
    return Py_BuildValue("(NnL)", THPVariable_Wrap(p.blob), Py_ssize_t(p.stride), (long long)p.n_trees);
}

// attention_paged(q, k_tree, v_tree, out, packed, tree_stride, n_trees, n_blocks, block_m, max_ancestors,
//                 k_pool, v_pool, nhd, block_table, prefix_lens, max_prefix, sm_scale, kv_splits, return_lse)
PyObject *attention_paged(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 19);
    const at::Tensor &q = tensor(a[0]), &kt = tensor(a[1]), &vt = tensor(a[2]), &kp = tensor(a[10]), &vp = tensor(a[11]),
                     &table = tensor(a[13]), &given_lens = tensor(a[14]);
    for (const at::Tensor *t : {&q, &kt, &vt, &kp, &vp, &table, &given_lens})
        if (!t->is_cuda()) raise(PyExc_RuntimeError, "fst_attention_paged runs on CUDA tensors only; there is no CPU path");
    const at::ScalarType type = q.scalar_type();
    bool same = type == at::kHalf || type == at::kBFloat16;
    for (const at::Tensor *t : {&kt, &vt, &kp, &vp}) same = same && t->scalar_type() == type;
    if (!same) raise(PyExc_TypeError, "q, k_tree, v_tree and the pools must share one dtype out of float16, bfloat16");
    if (q.dim() != 4 || kt.dim() != 4 || vt.dim() != 4) raise(PyExc_ValueError, "q, k_tree, v_tree must have four dimensions");
    const int64_t Z = q.size(0), H = q.size(1), n_q = q.size(2), D = q.size(3), H_kv = kt.size(1);
    if (kt.size(0) != Z || kt.size(2) != n_q || kt.size(3) != D || vt.sizes() != kt.sizes() || H_kv < 1 || H % H_kv)
        raise(PyExc_ValueError, "k_tree and v_tree must be [Z, H_kv, N, D] with H a multiple of H_kv");
    const bool nhd = a[12] == Py_True;
    const int row_dim = nhd ? 1 : 2, head_dim = nhd ? 2 : 1;
    if (kp.dim() != 4 || vp.sizes() != kp.sizes() || kp.size(head_dim) != H_kv || kp.size(3) != D ||
        kp.strides() != vp.strides() || kp.stride(3) != 1)
        raise(PyExc_ValueError, "pools must be two equally laid out [n_pages, page_size, H_kv, D] (or HND) tensors");
    if (table.scalar_type() != at::kInt || given_lens.scalar_type() != at::kInt || table.dim() != 2 || table.size(0) != Z ||
        given_lens.dim() != 1 || given_lens.size(0) != Z || !table.is_contiguous())
        raise(PyExc_ValueError, "block_table must be contiguous int32 [Z, pages], prefix_lens int32 [Z]");
    const int64_t n_trees = integer(a[6]), n_blocks = integer(a[7]), bm = integer(a[8]), ma = integer(a[9]);
    if ((n_trees != 1 && n_trees != Z) || n_blocks != (n_q + bm - 1) / bm) raise(PyExc_ValueError, "metadata does not match q");
    Call c = open_call(a[0], a[1], a[2], a[3], a[16], a[18] == Py_True);
    const int64_t max_prefix = integer(a[15]);
    const at::Device dev = q.device();
    for (const at::Tensor *t : {&kp, &vp, &table, &given_lens, &tensor(a[4])}) on_device(*t, dev);
    std::optional<long long> asked = optional_int(a[17]);
    Splits sp{asked ? int(*asked) : 1, false};
    if (max_prefix > 0 && (!asked || *asked > 0)) {
        const int64_t cap = 65535 / std::max<int64_t>(Z, 1);
        if (!asked || *asked <= cap) {                    // (more than the grid holds is the library's error to give)
            const fst::PrefixPlan plan =
                fst::prefix_plan(Z, H, H_kv, n_q, max_prefix, sm_count(dev.index()), true, asked.value_or(0), kp.size(row_dim));
            sp = {plan.runs, plan.spread};
        }
    }
    const c10::cuda::CUDAGuard guard(dev);
    if (max_prefix <= 0)                                  // no prefix anywhere: plain tree attention
        return launch(c, tensor(a[4]).data_ptr(), n_trees > 1 ? size_t(integer(a[5])) : 0, bm, ma, FST_KERNEL_AUTO, std::nullopt,
                      status_of(dev, true)->data_ptr(), c10::cuda::getCurrentCUDAStream(dev.index()).stream());
    const at::Tensor lens = given_lens.contiguous();      // the kernel reads length z at word z
    at::Tensor ws;
    size_t ws_bytes = 0;
    if (sp.workspace) {
        ws_bytes = fst_attention_split_workspace_bytes(int(Z), int(H), int(n_q), int(D), sp.runs);
        ws = empty({int64_t(ws_bytes)}, at::kByte, dev);
    }
    int32_t *status = static_cast<int32_t *>(status_of(dev, true)->data_ptr());
    void *stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const size_t tree_stride = n_trees > 1 ? size_t(integer(a[5])) : 0;
    const void *packed = tensor(a[4]).data_ptr();
    int rc;
    {
        pybind11::gil_scoped_release no_gil;
        rc = fst_attention_fwd_paged(q.data_ptr(), kt.data_ptr(), vt.data_ptr(), c.o.data_ptr(), lse_ptr(c), packed,
                                     tree_stride, kp.data_ptr(), vp.data_ptr(), static_cast<const int32_t *>(table.data_ptr()),
                                     int(table.size(1)), static_cast<const int32_t *>(lens.data_ptr()), int(max_prefix),
                                     int(kp.size(row_dim)), int(kp.size(0)), kp.stride(0), kp.stride(row_dim),
                                     kp.stride(head_dim), int(Z), int(H), int(H_kv), int(n_q), int(D), FST_STRIDES(q),
                                     FST_STRIDES(kt), FST_STRIDES(vt), FST_STRIDES(c.o), int(bm), int(ma), c.scale, c.dtype,
                                     sp.runs, ws.defined() ? ws.data_ptr() : nullptr, ws_bytes, status, stream);
    }
    check_status(rc, "fst_attention_fwd_paged");
    return results(c);
}

// ---- trees ---------------------------------------------------------------------------------------
// A cleared status record.  Clearing one per call is a launch (about a microsecond in front of a five
// microsecond kernel), so a thread takes them from a block that it cleared in one go on the same stream;
// a new block is made for another stream or device and when one is used up (256 records, 4 KB,
// returned to the allocator with the last record).  A call that is being captured into a graph
// clears its record in the graph, for every replay: `old` if it is given.  That is a fill kernel: kernels
// follow one another faster than a kernel follows a memset node (a 256-node build, 64 of them in a graph:
// 8.2 us with the memset, 5.2 with the fill).
// record_of: record i of a block, a tensor over the block's storage made without the dispatcher (narrow takes a microsecond).
at::Tensor record_of(const at::Tensor &words, int64_t i) {
    auto impl = c10::make_intrusive<c10::TensorImpl>(c10::Storage(words.storage()), c10::DispatchKeySet(c10::DispatchKey::CUDA), words.dtype());
    impl->set_sizes_contiguous({4});
    impl->set_storage_offset(4 * i);
    return at::Tensor(std::move(impl));
}
at::Tensor clear_record(const at::Device &dev, cudaStream_t stream, const at::Tensor &old, const char *what,
                        bool *captured = nullptr) {
    const OrdinaryTensors guard;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess) check_status(FST_ERR_CUDA, what);
    if (captured != nullptr) *captured = capturing != cudaStreamCaptureStatusNone;
    if (capturing != cudaStreamCaptureStatusNone) {
        at::Tensor t = old.defined() ? old : empty({4}, at::kInt, dev);
        t.zero_();
        return t;
    }
    constexpr int64_t kRecords = 256;
    struct Block {
        at::Tensor words;
        cudaStream_t stream = nullptr;
        int64_t next = kRecords;
    };
    static thread_local Block *block = new Block();       // (never destroyed: torch may be gone by then)
    if (block->next == kRecords || block->stream != stream || block->words.device() != dev) {
        block->words = empty({kRecords * 4}, at::kInt, dev);
        block->stream = stream;
        block->next = 0;
        if (cudaMemsetAsync(block->words.data_ptr(), 0, kRecords * 16, stream) != cudaSuccess) {
            block->next = kRecords;
            check_status(FST_ERR_CUDA, what);
        }
    }
    return record_of(block->words, block->next++);
}

void run_precompute(const at::Tensor &par, int64_t n_trees, int64_t n_nodes, int64_t bm, int64_t ma, const at::Tensor &packed,
                    size_t stride, const at::Tensor &status, const at::Tensor &ai, const at::Tensor &am,
                    const at::Tensor &li) {
    const at::Device dev = par.device();
    for (const at::Tensor *t : {&packed, &status, &ai, &am, &li})
        if (t->defined()) on_device(*t, dev);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    check_status(fst_precompute(static_cast<const int32_t *>(par.data_ptr()), int(n_trees), int(n_nodes), int(bm), int(ma),
                                ai.defined() ? static_cast<int64_t *>(ai.data_ptr()) : nullptr,
                                am.defined() ? static_cast<uint8_t *>(am.data_ptr()) : nullptr,
                                li.defined() ? static_cast<int64_t *>(li.data_ptr()) : nullptr, packed.data_ptr(), stride,
                                static_cast<int32_t *>(status.data_ptr()), stream),
                 "fst_precompute");
}
const at::Tensor &parent_arg(PyObject *o) {
    const at::Tensor &par = tensor(o);
    if ((par.dim() != 1 && par.dim() != 2) || par.numel() == 0)
        raise(PyExc_ValueError, "parent must be a non-empty [N] or [T, N] array");
    if (!par.is_cuda() || par.scalar_type() != at::kInt || !par.is_contiguous())
        raise(PyExc_ValueError, "parent must be a contiguous int32 CUDA tensor");
    return par;
}
at::Tensor optional_tensor(PyObject *o) { return o == Py_None ? at::Tensor() : tensor(o); }

// precompute(parent, block_m, max_ancestors, packed, tree_stride, status, ancestor_idx, ancestor_mask, leaf_idx)
//   -> the status record of this build; parent is a contiguous int32 CUDA tensor [N] or [T, N], the buffers belong to the caller and
//   the last three may be None.
PyObject *precompute(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 9);
    const at::Tensor &par = parent_arg(a[0]);
    const at::Device dev = par.device();
    const c10::cuda::CUDAGuard guard(dev);
    const at::Tensor status = clear_record(dev, c10::cuda::getCurrentCUDAStream(dev.index()).stream(), tensor(a[5]), "fst_precompute");
    run_precompute(par, par.dim() == 2 ? par.size(0) : 1, par.size(-1), integer(a[1]), integer(a[2]), tensor(a[3]),
                   size_t(integer(a[4])), status, optional_tensor(a[6]), optional_tensor(a[7]), optional_tensor(a[8]));
    return THPVariable_Wrap(status);
}

PyObject *wrap_or_none(const at::Tensor &t) {
    if (t.defined()) return THPVariable_Wrap(t);
    Py_RETURN_NONE;
}

// buffers for the metadata of n_trees trees of n_nodes nodes, and the build launched into them
struct Built {
    at::Tensor packed, status, ai, am, li;
    size_t stride;
    bool captured = false;
};
Built build_metadata(const at::Tensor &par, bool batched, int64_t n_trees, int64_t n_nodes, int64_t bm, int64_t ma, bool reference_format) {
    if (bm <= 0 || ma <= 0) raise(PyExc_ValueError, "block_m and max_ancestors must be positive");
    const int64_t nb = (n_nodes + bm - 1) / bm;
    const at::Device dev = par.device();
    const OrdinaryTensors guard;
    Built m;
    m.stride = fst_packed_meta_bytes(int(nb), int(bm), int(ma));
    m.packed = empty({n_trees, int64_t(m.stride)}, at::kByte, dev);
    m.status = clear_record(dev, c10::cuda::getCurrentCUDAStream(dev.index()).stream(), at::Tensor(), "fst_precompute", &m.captured);
    if (reference_format) {
        if (batched) {
            m.ai = empty({n_trees, nb, ma}, at::kLong, dev);
            m.am = empty({n_trees, nb, bm, ma}, at::kBool, dev);
            m.li = empty({n_trees, nb, bm}, at::kLong, dev);
        } else {
            m.ai = empty({nb, ma}, at::kLong, dev);
            m.am = empty({nb, bm, ma}, at::kBool, dev);
            m.li = empty({nb, bm}, at::kLong, dev);
        }
    }
    run_precompute(par, n_trees, n_nodes, bm, ma, m.packed, m.stride, m.status, m.ai, m.am, m.li);
    return m;
}

// new_metadata(parent, block_m, max_ancestors, reference_format)
//   -> (n_trees, n_nodes, packed, tree_stride, status, ancestor_idx, ancestor_mask, leaf_idx, whether the call was
//   captured into a graph), buffers made here.
PyObject *new_metadata(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 4);
    const at::Tensor &par = parent_arg(a[0]);
    const int64_t n_trees = par.dim() == 2 ? par.size(0) : 1, n_nodes = par.size(-1);
    const c10::cuda::CUDAGuard guard(par.device());
    const Built m = build_metadata(par, par.dim() == 2, n_trees, n_nodes, integer(a[1]), integer(a[2]), a[3] == Py_True);
    return Py_BuildValue("(LLNnNNNNO)", (long long)n_trees, (long long)n_nodes, THPVariable_Wrap(m.packed), Py_ssize_t(m.stride),
                         THPVariable_Wrap(m.status), wrap_or_none(m.ai), wrap_or_none(m.am), wrap_or_none(m.li),
                         m.captured ? Py_True : Py_False);
}

// dfs_order(parent) -> (order, new_parent, status)
PyObject *dfs_order(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 1);
    const at::Tensor &par = parent_arg(a[0]);
    const at::Device dev = par.device();
    const c10::cuda::CUDAGuard guard(dev);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const at::Tensor order = empty(par.sizes(), at::kInt, dev), npar = empty(par.sizes(), at::kInt, dev),
                     status = clear_record(dev, stream, at::Tensor(), "fst_dfs_order");
    check_status(fst_dfs_order(static_cast<const int32_t *>(par.data_ptr()), int(par.dim() == 2 ? par.size(0) : 1),
                               int(par.size(-1)), static_cast<int32_t *>(order.data_ptr()),
                               static_cast<int32_t *>(npar.data_ptr()), static_cast<int32_t *>(status.data_ptr()), stream),
                 "fst_dfs_order");
    return Py_BuildValue("(NNN)", THPVariable_Wrap(order), THPVariable_Wrap(npar), THPVariable_Wrap(status));
}

// build_tree_topk(scores, depth, topk, left_weight_factor, n or None for as many as the forest has, return_choice, return_scores)
//   -> (parent, choice or None, node scores or None)
PyObject *build_tree_topk(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 7);
    const long long total = fst_tree_topk_nodes(int(integer(a[1])), int(integer(a[2])), real(a[3]));
    if (total < 0)
        raise(PyExc_ValueError, "forest shape beyond the kernel's limits (a level above 4096 nodes, or more than 32 levels)");
    const int64_t nodes = a[4] == Py_None ? total : integer(a[4]);
    if (nodes <= 0) raise(PyExc_ValueError, "max_nodes must be positive");
    const at::Tensor sc = tensor(a[0]).contiguous();
    const bool batched = sc.dim() == 3;
    const int64_t n_trees = batched ? sc.size(0) : 1;
    const at::Device dev = sc.device();
    const c10::cuda::CUDAGuard guard(dev);
    const auto made = [&](at::ScalarType t) { return batched ? empty({n_trees, nodes}, t, dev) : empty({nodes}, t, dev); };
    const at::Tensor parent = made(at::kInt);
    const at::Tensor choice = a[5] == Py_True ? made(at::kInt) : at::Tensor(), score = a[6] == Py_True ? made(at::kFloat) : at::Tensor();
    check_status(fst_build_tree_topk(static_cast<const float *>(sc.data_ptr()), int(n_trees), int(integer(a[1])),
                                     int(integer(a[2])), real(a[3]), int(nodes), static_cast<int32_t *>(parent.data_ptr()),
                                     choice.defined() ? static_cast<int32_t *>(choice.data_ptr()) : nullptr,
                                     score.defined() ? static_cast<float *>(score.data_ptr()) : nullptr,
                                     c10::cuda::getCurrentCUDAStream(dev.index()).stream()),
                 "fst_build_tree_topk");
    return Py_BuildValue("(NNN)", THPVariable_Wrap(parent), wrap_or_none(choice), wrap_or_none(score));
}

// parent[k] = lineage[k, level[k] - 1], -1 on level 0 (utils.py:42-44 of the reference), for int64 CPU tensors; an entry
// is looked at before it is narrowed to 32 bits.
void parents_from(const at::Tensor &lin, const at::Tensor &lvl, int32_t *P) {
    const int64_t N = lin.size(0), W = lin.size(1), s0 = lin.stride(0), s1 = lin.stride(1), t0 = lvl.stride(0);
    const int64_t *L = static_cast<const int64_t *>(lin.data_ptr()), *V = static_cast<const int64_t *>(lvl.data_ptr());
    for (int64_t k = 0; k < N; ++k) {
        const int64_t lv = V[k * t0];
        if (lv > W) raise(PyExc_IndexError, "level_lookup points past the lineage columns");
        const int64_t p = lv > 0 ? L[k * s0 + (lv - 1) * s1] : -1;
        if (p >= k || p < -1) {
            PyErr_Format(PyExc_ValueError, "malformed tree: parent[%lld]=%lld must be -1 or an earlier node", (long long)k, (long long)p);
            throw PyError{};
        }
        P[k] = int32_t(p);
    }
}
// parents_of_lineage(lineage, level_lookup) -> int32 parent array on the host (pinned).  The reference's side effect
// (utils.py:124-125) - every node written into its own lineage row - is a second call.
PyObject *parents_of_lineage(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 2);
    const at::Tensor &lin = tensor(a[0]);
    const at::Tensor parent = at::empty({lin.size(0)}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));   // torch's pinned pool
    parents_from(lin, tensor(a[1]), static_cast<int32_t *>(parent.data_ptr()));
    return THPVariable_Wrap(parent);
}

// What the device status record of a metadata build would say of the ancestor bound, from parents_from's array on the host, so
// that the caller need not wait for the device to learn it.  Every node is marked once per block: the marks of a block are its ancestors.
void check_bound(const int32_t *P, int64_t N, int64_t bm, int64_t ma) {
    std::vector<int32_t> seen(N, -1);                     // last block that met the node
    for (int64_t b = 0; b * bm < N; ++b) {
        int64_t count = 0;
        for (int64_t k = b * bm; k < std::min(N, (b + 1) * bm); ++k)
            for (int32_t x = P[k]; x >= 0 && seen[x] != int32_t(b); x = P[x], ++count) seen[x] = int32_t(b);
        if (count > ma) {
            PyErr_Format(PyExc_RuntimeError, "block %lld of tree 0 has %lld unique ancestors, more than max_ancestors=%lld",
                         (long long)b, (long long)count, (long long)ma);
            throw PyError{};
        }
    }
}
// check_tree(parent, block_m, max_ancestors), parent what parents_of_lineage has returned
PyObject *check_tree(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 3);
    const at::Tensor &par = tensor(a[0]);
    check_bound(static_cast<const int32_t *>(par.data_ptr()), par.size(0), integer(a[1]), integer(a[2]));
    Py_RETURN_NONE;
}

// metadata_of_lineage(lineage, level_lookup, block_m, max_ancestors) -> (packed, tree_stride, ancestor_idx, ancestor_mask, leaf_idx), checked, for
// int64 CPU tensors; None where the call is for the general path: more parents than the driver takes from pageable
// memory at once (it would wait for the stream), or a stream that is being captured (a replay would read
// memory that is gone).  The driver has copied the parents when cudaMemcpyAsync returns, so neither a pinned buffer nor an event of
// torch's pool is needed: 16 us from the parents on the host to the launch, 8 without them.
PyObject *metadata_of_lineage(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 4);
    constexpr int64_t kInline = 8192;                     // parents: 32 KB, the driver stages up to 64
    const at::Tensor &lin = tensor(a[0]), &lvl = tensor(a[1]);
    const int64_t N = lin.size(0), bm = integer(a[2]), ma = integer(a[3]);
    if (N == 0 || N > kInline) Py_RETURN_NONE;
    std::vector<int32_t> P(N);
    parents_from(lin, lvl, P.data());
    const at::Tensor par = empty({N}, at::kInt, at::Device(at::kCUDA, c10::cuda::current_device()));
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(par.device().index()).stream();
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess) check_status(FST_ERR_CUDA, "fst_precompute");
    if (capturing != cudaStreamCaptureStatusNone) Py_RETURN_NONE;
    if (cudaMemcpyAsync(par.data_ptr(), P.data(), size_t(N) * 4, cudaMemcpyHostToDevice, stream) != cudaSuccess)
        check_status(FST_ERR_CUDA, "fst_precompute");
    const Built m = build_metadata(par, false, 1, N, bm, ma, true);
    check_bound(P.data(), N, bm, ma);
    return Py_BuildValue("(NnNNN)", THPVariable_Wrap(m.packed), Py_ssize_t(m.stride), THPVariable_Wrap(m.ai), THPVariable_Wrap(m.am),
                         THPVariable_Wrap(m.li));
}

// write_self(lineage, level_lookup): lineage[k, level[k]] = k (utils.py:124-125), int64 CPU tensors
PyObject *write_self(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 2);
    const at::Tensor &lin = tensor(a[0]), &lvl = tensor(a[1]);
    const int64_t N = lin.size(0), W = lin.size(1), s0 = lin.stride(0), s1 = lin.stride(1), t0 = lvl.stride(0);
    int64_t *L = static_cast<int64_t *>(lin.data_ptr());
    const int64_t *V = static_cast<const int64_t *>(lvl.data_ptr());
    for (int64_t k = 0; k < N; ++k) {
        const int64_t lv = V[k * t0];
        if (lv < 0 || lv >= W) raise(PyExc_IndexError, "level_lookup points past the lineage columns");
        L[k * s0 + lv * s1] = k;
    }
    lin.unsafeGetTensorImpl()->bump_version();
    Py_RETURN_NONE;
}

// read_status(record) -> its four words, once everything ahead on the current stream has run
PyObject *read_status(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 1);
    const at::Tensor &t = tensor(a[0]);
    const at::Device dev = t.device();
    const c10::cuda::CUDAGuard guard(dev);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    int32_t w[4] = {};
    cudaError_t e;
    {
        pybind11::gil_scoped_release no_gil;
        e = cudaMemcpyAsync(w, t.data_ptr(), sizeof(w), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    }
    if (e != cudaSuccess) {
        PyErr_Format(PyExc_RuntimeError, "reading a status record: %s", cudaGetErrorString(e));
        throw PyError{};
    }
    return Py_BuildValue("(iiii)", w[0], w[1], w[2], w[3]);
}

// status_record(device_index) -> the attention status record of that device, or None before its first launch
PyObject *status_record(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 1);
    const at::Tensor *t = status_of(at::Device(at::kCUDA, at::DeviceIndex(integer(a[0]))), false);
    if (t == nullptr) Py_RETURN_NONE;
    return THPVariable_Wrap(*t);
}
// attention_status(device_index) -> the same, made on first use
PyObject *attention_status(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 1);
    return THPVariable_Wrap(*status_of(at::Device(at::kCUDA, at::DeviceIndex(integer(a[0]))), true));
}

// splits(q, prefix, block_m, kernel, kv_splits, sm_scale, kv_heads) -> (runs, whether a workspace is needed, whether the tcgen05
//   prefix kernel takes the call)
PyObject *splits(PyObject *const *a, Py_ssize_t n) {
    want_args(n, 7);
    const at::Tensor &q = tensor(a[0]);
    const int64_t H = q.size(1), H_kv = integer(a[6]);
    if (H_kv < 1 || H % H_kv) raise(PyExc_ValueError, "the heads of q must be a multiple of kv_heads");
    const Splits s = pick_splits(optional_int(a[4]), q.scalar_type(), q.size(0), H, H_kv, q.size(2), q.size(3), integer(a[1]),
                                 integer(a[2]), real(a[5]), int(integer(a[3])), q.device().index());
    return Py_BuildValue("(iOO)", s.runs, s.workspace ? Py_True : Py_False, s.umma ? Py_True : Py_False);
}

#define FST_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(&guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FST_METHOD(attention),      FST_METHOD(attention_ref), FST_METHOD(attention_paged), FST_METHOD(pack),
    FST_METHOD(precompute),     FST_METHOD(new_metadata),  FST_METHOD(dfs_order),
    FST_METHOD(build_tree_topk), FST_METHOD(parents_of_lineage), FST_METHOD(write_self), FST_METHOD(check_tree), FST_METHOD(metadata_of_lineage), FST_METHOD(read_status), FST_METHOD(status_record), FST_METHOD(attention_status),
    FST_METHOD(splits),         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fst_host", "tensor-level calls into libfstattn_b200.so", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__fst_host() { return PyModule_Create(&module); }
