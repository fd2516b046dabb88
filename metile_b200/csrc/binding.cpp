// Native call path of the torch operators in metile_b200/backends: checks the tensors, allocates the
// result and calls the C ABI (include/metile_b200.h) without going through the interpreter.
//
// Why.  A decode-sized kernel takes 4 to 20 us on the GPU; the same call written in Python (argument
// checks, torch.empty, ctypes marshalling of a dozen pointers) took 12 to 25 us of host time, so a stream
// of such calls was bound by the interpreter (one-row projection 1536 -> 8960: 16.3 us per call for a
// 6.2 us kernel).  Here it is 3 to 5 us, most of it the launch itself.
//
// Contract with the Python callers: a function returns the result tensor(s); or None when anything about
// the arguments is not the plain case (another type, dtype, device, layout or shape) -- the caller then
// runs its Python form, which copies what must be copied and raises the operator's own exceptions; or the
// library's negative status code as an int.  Nothing is queued unless a tensor is returned or the code
// says so.  A C++ exception -- a tensor without strides or storage, no memory for the result -- becomes the
// Python exception torch raises for it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/core/GradMode.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/metile_b200.h"

namespace {

using at::Tensor;

// A plain tensor (not a subclass, which may intercept operations) or null.
inline const Tensor* plain(PyObject* object) {
    return THPVariable_CheckExact(object) ? &THPVariable_Unpack(object) : nullptr;
}

inline bool bf16_on(const Tensor& t, c10::Device device) {
    return t.scalar_type() == at::kBFloat16 && t.device() == device && t.is_contiguous();
}

inline void* address(const Tensor& t) { return t.data_ptr(); }

// The device the call runs on made current (the usual case: it already is), and its current stream.
class Launch {
public:
    explicit Launch(c10::Device device) {
        if (c10::cuda::current_device() != device.index()) guard_.set_device(device);
        stream_ = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    }
    void* stream() const { return stream_; }

private:
    c10::cuda::OptionalCUDAGuard guard_;
    cudaStream_t stream_;
};

// Other Python threads may run while this lives.  An exception that leaves its block -- a tensor under vmap has no
// address -- meets the interpreter with its lock held again.
class Unlocked {
public:
    Unlocked() : thread_(PyEval_SaveThread()) {}
    ~Unlocked() { PyEval_RestoreThread(thread_); }
    Unlocked(const Unlocked&) = delete;
    Unlocked& operator=(const Unlocked&) = delete;

private:
    PyThreadState* thread_;
};

inline Tensor new_bf16(at::IntArrayRef sizes, c10::Device device) {
    return at::detail::empty_cuda(sizes, at::kBFloat16, device, std::nullopt);
}

// Scratch of one call: the caching allocator hands it to later work of the same stream, and keeps it for the graph when
// the call is captured.
inline c10::DataPtr call_scratch(size_t bytes) { return c10::cuda::CUDACachingAllocator::get()->allocate(bytes); }

inline Tensor new_like(const Tensor& t) { return new_bf16(t.sizes(), t.device()); }

inline PyObject* code_or(int code, Tensor&& result) {
    if (code != 0) return PyLong_FromLong(code);
    return THPVariable_Wrap(std::move(result));
}

// Activations of an INT4 projection: contiguous bf16 [..., K] on a CUDA device.
inline bool activations_ok(const Tensor* x) {
    return x && x->is_cuda() && x->dim() >= 1 && x->numel() > 0 && x->scalar_type() == at::kBFloat16 && x->is_contiguous();
}

// One affine triple against activations of width `k`; -1 when it is not the plain case, else N.
inline int64_t triple_rows(const Tensor* w, const Tensor* s, const Tensor* b, int64_t k, c10::Device device) {
    if (!w || !s || !b || w->dim() != 2 || s->dim() != 2 || b->dim() != 2) return -1;
    const auto type = w->scalar_type();
    if ((type != at::kUInt32 && type != at::kInt) || w->device() != device || !w->is_contiguous()) return -1;
    const int64_t n = w->size(0);
    if (k % 64 || w->size(1) * 8 != k || s->size(0) != n || s->size(1) * 64 != k || b->size(0) != n || b->size(1) * 64 != k)
        return -1;
    return bf16_on(*s, device) && bf16_on(*b, device) ? n : -1;
}

inline bool fits_int(int64_t v) { return v <= 0x7FFFFFFF; }

// project(values, weight, scales, biases, residual | None, group_size, bits, flags)
PyObject* project(PyObject* const* args) {
    const Tensor* x = plain(args[0]);
    const Tensor* residual = args[4] == Py_None ? nullptr : plain(args[4]);
    const long group = PyLong_AsLong(args[5]), bits = PyLong_AsLong(args[6]), flags = PyLong_AsLong(args[7]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if (!activations_ok(x) || group != 64 || bits != 4 || (args[4] != Py_None && !residual)) Py_RETURN_NONE;
    const auto device = x->device();
    const int64_t k = x->size(-1), rows = x->numel() / k;
    const Tensor *w = plain(args[1]), *s = plain(args[2]), *b = plain(args[3]);
    const int64_t n = triple_rows(w, s, b, k, device);
    if (n < 1 || !fits_int(rows) || !fits_int(n) || !fits_int(k)) Py_RETURN_NONE;
    c10::SmallVector<int64_t, 6> sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = n;
    if (residual && (residual->sizes() != at::IntArrayRef(sizes) || !bf16_on(*residual, device))) Py_RETURN_NONE;
    const Launch launch(device);
    Tensor out = new_bf16(sizes, device);
    int code;
    {
        const Unlocked unlocked;
        code = mt_affine_qmv(address(*x), static_cast<const uint32_t*>(address(*w)), address(*s), address(*b),
                             residual ? address(*residual) : nullptr, address(out), (int)rows, (int)k, (int)n, (int)group,
                             (int)bits, (unsigned int)flags, launch.stream());
    }
    return code_or(code, std::move(out));
}

// swiglu(values, gate_weight, gate_scales, gate_biases, up_weight, up_scales, up_biases, flags)
PyObject* swiglu(PyObject* const* args) {
    const Tensor* x = plain(args[0]);
    const long flags = PyLong_AsLong(args[7]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if (!activations_ok(x)) Py_RETURN_NONE;
    const auto device = x->device();
    const int64_t k = x->size(-1), rows = x->numel() / k;
    const Tensor* t[6];
    for (int i = 0; i < 6; ++i) t[i] = plain(args[1 + i]);
    const int64_t n = triple_rows(t[0], t[1], t[2], k, device);
    if (n < 1 || triple_rows(t[3], t[4], t[5], k, device) != n || !fits_int(rows) || !fits_int(n) || !fits_int(k))
        Py_RETURN_NONE;
    c10::SmallVector<int64_t, 6> sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = n;
    const Launch launch(device);
    Tensor out = new_bf16(sizes, device);
    int code;
    {
        const Unlocked unlocked;
        code = mt_affine_swiglu(address(*x), static_cast<const uint32_t*>(address(*t[0])), address(*t[1]), address(*t[2]),
                                static_cast<const uint32_t*>(address(*t[3])), address(*t[4]), address(*t[5]), address(out),
                                (int)rows, (int)k, (int)n, 64, 4, (unsigned int)flags, launch.stream());
    }
    return code_or(code, std::move(out));
}

// The nine weight addresses of a bound MLP and its shape; the Python executor owns the tensors.
struct MlpPlan {
    void* weights[9];
    int64_t hidden, inter;
    c10::Device device{c10::kCUDA, 0};
};
constexpr const char* kMlpPlanName = "metile_b200.mlp_plan";

void free_mlp_plan(PyObject* capsule) { delete static_cast<MlpPlan*>(PyCapsule_GetPointer(capsule, kMlpPlanName)); }

// mlp_plan(nine weight tensors as for mlx_affine_mlp_executor, already checked) -> capsule, or None
PyObject* mlp_plan(PyObject* const* args) {
    MlpPlan plan;
    for (int i = 0; i < 9; ++i) {
        const Tensor* t = plain(args[i]);
        if (!t || !t->is_cuda()) Py_RETURN_NONE;
        plan.weights[i] = address(*t);
        if (i == 0) {
            plan.device = t->device();
            plan.hidden = t->size(1) * 8;
            plan.inter = t->size(0);
        }
    }
    if (!fits_int(plan.hidden) || !fits_int(plan.inter)) Py_RETURN_NONE;
    return PyCapsule_New(new MlpPlan(plan), kMlpPlanName, free_mlp_plan);
}

// mlp(plan, values, residual | None, flags)
PyObject* mlp(PyObject* const* args) {
    if (!PyCapsule_IsValid(args[0], kMlpPlanName)) Py_RETURN_NONE;
    const MlpPlan& plan = *static_cast<const MlpPlan*>(PyCapsule_GetPointer(args[0], kMlpPlanName));
    const Tensor* x = plain(args[1]);
    const Tensor* residual = args[2] == Py_None ? nullptr : plain(args[2]);
    const long flags = PyLong_AsLong(args[3]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if (!activations_ok(x) || x->device() != plan.device || x->size(-1) != plan.hidden) Py_RETURN_NONE;
    if (args[2] != Py_None && (!residual || residual->sizes() != x->sizes() || !bf16_on(*residual, plan.device))) Py_RETURN_NONE;
    const int64_t rows = x->numel() / plan.hidden;
    if (!fits_int(rows)) Py_RETURN_NONE;
    const Launch launch(plan.device);
    Tensor out = new_like(*x);
    const size_t needed = mt_affine_mlp_workspace_bytes((int)rows, (int)plan.hidden, (int)plan.inter);
    const c10::DataPtr scratch = call_scratch(needed);
    void* const* w = plan.weights;
    int code;
    {
        const Unlocked unlocked;
        code = mt_affine_mlp(address(*x), static_cast<const uint32_t*>(w[0]), w[1], w[2], static_cast<const uint32_t*>(w[3]),
                             w[4], w[5], static_cast<const uint32_t*>(w[6]), w[7], w[8],
                             residual ? address(*residual) : nullptr, scratch.get(), needed,
                             address(out), (int)rows, (int)plan.hidden, (int)plan.inter, 64, 4, (unsigned int)flags,
                             launch.stream());
    }
    return code_or(code, std::move(out));
}

// norm(values, residual | None, weight, eps): the normalised rows, or (summed, normalised) with a residual.
PyObject* norm(PyObject* const* args) {
    const Tensor *x = plain(args[0]), *weight = plain(args[2]);
    const Tensor* residual = args[1] == Py_None ? nullptr : plain(args[1]);
    const double eps = PyFloat_AsDouble(args[3]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if (!activations_ok(x) || !weight || weight->dim() != 1 || weight->size(0) != x->size(-1) || !bf16_on(*weight, x->device()))
        Py_RETURN_NONE;
    if (args[1] != Py_None && (!residual || residual->sizes() != x->sizes() || !bf16_on(*residual, x->device()))) Py_RETURN_NONE;
    const int64_t width = x->size(-1), rows = x->numel() / width;
    if (!fits_int(rows) || !fits_int(width)) Py_RETURN_NONE;
    const Launch launch(x->device());
    Tensor normalized = new_like(*x), summed;
    int code;
    if (residual) summed = new_like(*x);
    {
        const Unlocked unlocked;
        code = residual ? mt_add_rmsnorm(address(*x), address(*residual), address(*weight), address(summed), address(normalized),
                                         (int)rows, (int)width, (float)eps, launch.stream())
                        : mt_rmsnorm(address(*x), address(*weight), address(normalized), (int)rows, (int)width, (float)eps,
                                     launch.stream());
    }
    if (!residual || code != 0) return code_or(code, std::move(normalized));
    PyObject* pair = PyTuple_New(2);
    if (!pair) return nullptr;
    PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(summed)));
    PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(std::move(normalized)));
    return pair;
}

// dense(values, weight, up_weight | None, residual | None): with an up weight the SwiGLU of both.
PyObject* dense(PyObject* const* args) {
    const Tensor *x = plain(args[0]), *w = plain(args[1]);
    const Tensor* up = args[2] == Py_None ? nullptr : plain(args[2]);
    const Tensor* residual = args[3] == Py_None ? nullptr : plain(args[3]);
    if (!activations_ok(x) || !w || w->dim() != 2 || w->size(1) != x->size(-1) || !bf16_on(*w, x->device())) Py_RETURN_NONE;
    const auto device = x->device();
    const int64_t k = x->size(-1), rows = x->numel() / k, n = w->size(0);
    if (args[2] != Py_None && (!up || up->sizes() != w->sizes() || !bf16_on(*up, device))) Py_RETURN_NONE;
    if (k % 128 || n < 1 || !fits_int(rows) || !fits_int(n) || !fits_int(k)) Py_RETURN_NONE;
    c10::SmallVector<int64_t, 6> sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = n;
    if (args[3] != Py_None && (!residual || residual->sizes() != at::IntArrayRef(sizes) || !bf16_on(*residual, device)))
        Py_RETURN_NONE;
    const Launch launch(device);
    Tensor out = new_bf16(sizes, device);
    int code;
    {
        const Unlocked unlocked;
        code = up ? mt_dense_swiglu(address(*x), address(*w), address(*up), address(out), (int)rows, (int)k, (int)n, launch.stream())
                  : mt_dense_rows(address(*x), address(*w), residual ? address(*residual) : nullptr, address(out), (int)rows, (int)k,
                                  (int)n, launch.stream());
    }
    return code_or(code, std::move(out));
}

// Tokens per head a [B, H, N, D] cache (or a view of its first N tokens) has room for; -1: another layout.
inline int64_t cache_capacity(const Tensor& t) {
    const int64_t dim = t.size(3);
    if (t.stride(3) != 1 || t.stride(2) != dim || t.stride(1) % dim || t.stride(0) != t.size(1) * t.stride(1)) return -1;
    const int64_t capacity = t.stride(1) / dim;
    return capacity >= t.size(2) ? capacity : -1;
}

// attention(query, key, value, scale, lengths | None)
PyObject* attention(PyObject* const* args) {
    const Tensor *q = plain(args[0]), *k = plain(args[1]), *v = plain(args[2]);
    const Tensor* lengths = args[4] == Py_None ? nullptr : plain(args[4]);
    const double scale = PyFloat_AsDouble(args[3]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if (!q || !k || !v || (args[4] != Py_None && !lengths)) Py_RETURN_NONE;
    if (q->dim() != 4 || k->dim() != 4 || v->dim() != 4 || !q->is_cuda() || !q->is_contiguous()) Py_RETURN_NONE;
    const auto device = q->device();
    const int64_t batch = q->size(0), heads = q->size(1), dim = q->size(3), kv_heads = k->size(1), tokens = k->size(2);
    if (q->size(2) != 1 || k->sizes() != v->sizes() || k->size(0) != batch || k->size(3) != dim || (dim != 64 && dim != 128) ||
        batch < 1 || kv_heads < 1 || heads % kv_heads || heads / kv_heads > 8 || heads < 1 || tokens < 1)
        Py_RETURN_NONE;
    if (q->scalar_type() != at::kBFloat16 || k->scalar_type() != at::kBFloat16 || v->scalar_type() != at::kBFloat16 ||
        k->device() != device || v->device() != device)
        Py_RETURN_NONE;
    const int64_t capacity = cache_capacity(*k);
    if (capacity < 0 || cache_capacity(*v) != capacity || !fits_int(capacity) || !fits_int(batch * heads)) Py_RETURN_NONE;
    if (lengths && (lengths->device() != device || lengths->scalar_type() != at::kInt || !lengths->is_contiguous() ||
                    lengths->numel() < batch))
        Py_RETURN_NONE;
    const Launch launch(device);
    Tensor out = new_like(*q);
    const size_t needed = mt_attention_decode_workspace_bytes((int)batch, (int)heads, (int)tokens, (int)dim);
    c10::DataPtr scratch;
    if (needed) scratch = call_scratch(needed);
    int code;
    {
        const Unlocked unlocked;
        code = mt_attention_decode(address(*q), address(*k), address(*v), lengths ? static_cast<const int*>(address(*lengths)) : nullptr,
                                   address(out), scratch.get(), needed, (int)batch, (int)heads, (int)kv_heads, (int)tokens,
                                   (int)capacity, (int)dim, (float)scale, launch.stream());
    }
    return code_or(code, std::move(out));
}

int append(const void* q, const void* k, const void* v, long long row_stride, int* positions, void* q_out, void* k_cache,
           void* v_cache, int batch, int q_heads, int kv_heads, int capacity, int head_dim, float theta, void* stream) {
    return mt_rope_kv_append(q, k, v, row_stride, positions, q_out, k_cache, v_cache, batch, q_heads, kv_heads, capacity,
                             head_dim, theta, stream);
}

inline bool head_major(const Tensor& t, int64_t dim) { return t.stride(2) == 1 && t.stride(1) == dim; }

// rope_kv_append(query, key, value, positions, key_cache, value_cache, theta, advance)
PyObject* rope_kv_append(PyObject* const* args) {
    const Tensor* t[6];
    for (int i = 0; i < 6; ++i)
        if (!(t[i] = plain(args[i]))) Py_RETURN_NONE;
    const bool advance = args[7] == Py_True;
    const double theta = PyFloat_AsDouble(args[6]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    const Tensor &q = *t[0], &k = *t[1], &v = *t[2], &positions = *t[3], &keys = *t[4], &values = *t[5];
    if (!q.is_cuda() || q.dim() != 3 || k.dim() != 3 || v.dim() != 3 || keys.dim() != 4) Py_RETURN_NONE;
    const auto device = q.device();
    const int64_t batch = q.size(0), heads = q.size(1), dim = q.size(2), kv_heads = keys.size(1), capacity = keys.size(2);
    if (batch < 1 || heads < 1 || k.size(0) != batch || k.size(1) != kv_heads || k.size(2) != dim || v.sizes() != k.sizes() ||
        keys.size(0) != batch || keys.size(3) != dim || values.sizes() != keys.sizes())
        Py_RETURN_NONE;
    if (!bf16_on(keys, device) || !bf16_on(values, device) || q.scalar_type() != at::kBFloat16 || k.scalar_type() != at::kBFloat16 ||
        v.scalar_type() != at::kBFloat16 || k.device() != device || v.device() != device)
        Py_RETURN_NONE;
    if (positions.device() != device || positions.scalar_type() != at::kInt || !positions.is_contiguous() || positions.numel() < batch)
        Py_RETURN_NONE;
    if (!head_major(q, dim) || !head_major(k, dim) || !head_major(v, dim) ||
        (batch > 1 && (q.stride(0) != k.stride(0) || q.stride(0) != v.stride(0))))
        Py_RETURN_NONE;
    if (!fits_int(batch * (heads + 2 * kv_heads)) || !fits_int(capacity)) Py_RETURN_NONE;
    const int64_t row_stride = batch > 1 ? q.stride(0) : (heads + 2 * kv_heads) * dim;
    const Launch launch(device);
    Tensor out = new_bf16({batch, heads, dim}, device);
    int code;
    {
        const Unlocked unlocked;
        code = (advance ? mt_rope_kv_append_advance : append)(
            address(q), address(k), address(v), row_stride, static_cast<int*>(address(positions)), address(out), address(keys),
            address(values), (int)batch, (int)heads, (int)kv_heads, (int)capacity, (int)dim, (float)theta, launch.stream());
    }
    return code_or(code, std::move(out));
}

// rope_kv_prefill(query, key, value, inverse, positions, first, key_cache, value_cache)
PyObject* rope_kv_prefill(PyObject* const* args) {
    const Tensor* t[8] = {};
    for (int i : {0, 1, 2, 3, 4, 6, 7})
        if (!(t[i] = plain(args[i]))) Py_RETURN_NONE;
    const long first = PyLong_AsLong(args[5]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    const Tensor &q = *t[0], &k = *t[1], &v = *t[2], &inverse = *t[3], &positions = *t[4], &keys = *t[6], &values = *t[7];
    if (!q.is_cuda() || q.dim() != 4 || k.dim() != 4 || keys.dim() != 4 || q.numel() == 0) Py_RETURN_NONE;
    const auto device = q.device();
    const int64_t batch = q.size(0), steps = q.size(1), heads = q.size(2), dim = q.size(3);
    const int64_t kv_heads = keys.size(1), capacity = keys.size(2);
    if (k.size(0) != batch || k.size(1) != steps || k.size(2) != kv_heads || k.size(3) != dim || v.sizes() != k.sizes() ||
        keys.size(0) != batch || keys.size(3) != dim || values.sizes() != keys.sizes() || kv_heads < 1 || dim % 2 || dim > 4096)
        Py_RETURN_NONE;
    for (const Tensor* tensor : {&q, &k, &v, &keys, &values})
        if (!bf16_on(*tensor, device)) Py_RETURN_NONE;
    if (inverse.device() != device || inverse.scalar_type() != at::kFloat || !inverse.is_contiguous() || inverse.numel() != dim / 2)
        Py_RETURN_NONE;
    if (positions.device() != device || positions.scalar_type() != at::kInt || !positions.is_contiguous() || positions.numel() < batch)
        Py_RETURN_NONE;
    if (!fits_int(batch * steps) || !fits_int(capacity) || first < 0 || first + steps > capacity) Py_RETURN_NONE;
    const Launch launch(device);
    Tensor out = new_like(q);
    int code;
    {
        const Unlocked unlocked;
        code = mt_rope_kv_prefill(address(q), address(k), address(v), static_cast<const float*>(address(inverse)), address(out),
                                  address(keys), address(values), static_cast<int*>(address(positions)), (int)batch, (int)steps,
                                  (int)first, (int)heads, (int)kv_heads, (int)capacity, (int)dim, launch.stream());
    }
    return code_or(code, std::move(out));
}

// greedy_token(logits [rows, vocabulary] bf16, tokens [rows] or [rows, 1] int64) -> logits as float32
PyObject* greedy_token(PyObject* const* args) {
    const Tensor *logits = plain(args[0]), *tokens = plain(args[1]);
    if (!logits || !tokens || !logits->is_cuda() || logits->dim() != 2 || logits->numel() == 0) Py_RETURN_NONE;
    const auto device = logits->device();
    const int64_t rows = logits->size(0), vocabulary = logits->size(1);
    if (!bf16_on(*logits, device) || tokens->device() != device || tokens->scalar_type() != at::kLong || !tokens->is_contiguous() ||
        tokens->numel() != rows || rows > MT_GREEDY_MAX_ROWS || vocabulary > MT_GREEDY_MAX_VOCABULARY)
        Py_RETURN_NONE;
    const Launch launch(device);
    Tensor out = at::detail::empty_cuda({rows, vocabulary}, at::kFloat, device, std::nullopt);
    int code;
    {
        const Unlocked unlocked;
        code = mt_greedy_token(address(*logits), static_cast<float*>(address(out)), static_cast<long long*>(address(*tokens)), (int)rows,
                               (int)vocabulary, launch.stream());
    }
    return code_or(code, std::move(out));
}

// embedding(tokens int64 [...], table [V, H] bf16) -> [..., H]
PyObject* embedding(PyObject* const* args) {
    const Tensor *tokens = plain(args[0]), *table = plain(args[1]);
    if (!tokens || !table || !table->is_cuda() || table->dim() != 2 || (table->requires_grad() && c10::GradMode::is_enabled())) Py_RETURN_NONE;
    const auto device = table->device();
    const int64_t rows = tokens->numel(), width = table->size(1);
    if (!bf16_on(*table, device) || tokens->device() != device || tokens->scalar_type() != at::kLong || !tokens->is_contiguous() ||
        rows < 1 || !fits_int(rows) || width < 8 || width % 8 || !fits_int(width) || reinterpret_cast<uintptr_t>(address(*table)) % 16)
        Py_RETURN_NONE;
    const Launch launch(device);
    c10::SmallVector<int64_t, 6> sizes(tokens->sizes().begin(), tokens->sizes().end());
    sizes.push_back(width);
    Tensor out = new_bf16(sizes, device);
    int code;
    {
        const Unlocked unlocked;
        code = mt_gather_rows(address(*table), static_cast<const long long*>(address(*tokens)), address(out), (int)rows, table->size(0), (int)width,
                              launch.stream());
    }
    return code_or(code, std::move(out));
}

template <PyObject* (*kBody)(PyObject* const*), Py_ssize_t kCount>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t count) {
    try {
        if (count != kCount) Py_RETURN_NONE;
        return kBody(args);
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

#define MT_METHOD(name, count) \
    {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(entry<name, count>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {MT_METHOD(project, 8), MT_METHOD(swiglu, 8), MT_METHOD(mlp_plan, 9), MT_METHOD(mlp, 4), MT_METHOD(norm, 4),
                         MT_METHOD(dense, 4), MT_METHOD(attention, 5), MT_METHOD(rope_kv_append, 8), MT_METHOD(rope_kv_prefill, 8),
                         MT_METHOD(greedy_token, 2), MT_METHOD(embedding, 2), {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
