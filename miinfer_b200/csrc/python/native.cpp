// CPython module under the Python mirror's per-token launchers: takes the tensors themselves, reads pointers, dtypes and
// the current stream through torch's C++ interface, and calls the C ABI through addresses handed over by _lib.py (so
// that the one loaded libb200kv.so serves both).  It holds no state of a call and does no arithmetic.
//
// Why it exists: through ctypes a launcher spent 10-14 us of Python time per call (argument conversion, three attribute
// calls per tensor, a Stream object per call), more than the kernels of a short-context step take; here it is about 1 us.
// The interpreter lock is released around every library call, as ctypes does: a launch can block when the stream's
// queue is full.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstring>
#include <vector>

#include "b200kv.h"

namespace {

struct Api {
    decltype(&b200kv_append) append;
    decltype(&b200kv_q_split_norm_rope) q_split_norm_rope;
    decltype(&b200kv_decode_attn) decode_attn;
    decltype(&b200kv_decode_step) decode_step;
    decltype(&b200kv_decode_attn_batched) decode_attn_batched;
    decltype(&b200kv_prefill_attn_prepared) prefill_attn_prepared;
    decltype(&b200kv_pool_capture) pool_capture;
    decltype(&b200kv_pool_restore) pool_restore;
} g_api;
PyObject* g_view_type;   // the ctypes structure of a cache view

// One call's arguments, read left to right; the first failure sticks and leaves a Python exception set.
class Args {
public:
    Args(PyObject* const* args, Py_ssize_t n, Py_ssize_t want) : args_(args) {
        if (n != want) {
            PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
            ok_ = false;
        }
    }
    ~Args() {
        for (int i = 0; i < held_; ++i) PyBuffer_Release(&buffers_[i]);
    }
    bool ok() const { return ok_; }

    void* tensor(int64_t* numel = nullptr, int* dtype = nullptr) {   // None = null pointer
        if (!ok_) return nullptr;
        PyObject* o = args_[i_++];
        if (numel) *numel = 0;
        if (o == Py_None) {
            if (dtype) fail(PyExc_ValueError, "a tensor is required");
            return nullptr;
        }
        if (!THPVariable_Check(o)) return fail(PyExc_TypeError, "a torch tensor is required");
        const at::Tensor& t = THPVariable_Unpack(o);
        if (!t.is_cuda() || !t.is_contiguous()) return fail(PyExc_ValueError, "expected a contiguous CUDA tensor");
        if (numel) *numel = t.numel();
        if (dtype) {
            const auto type = t.scalar_type();
            if (type == at::kHalf) *dtype = B200KV_F16;
            else if (type == at::kFloat) *dtype = B200KV_F32;
            else return fail(PyExc_ValueError, (std::string("unsupported dtype ") + c10::toString(type) + ": fp16 or fp32 expected").c_str());
        }
        return t.data_ptr();
    }
    template <typename T> T* tensor_as(int64_t* numel = nullptr, int* dtype = nullptr) { return static_cast<T*>(tensor(numel, dtype)); }

    uint32_t u32() {   // as a C unsigned conversion: higher bits are dropped
        if (!ok_) return 0;
        PyObject* o = args_[i_++];
        if (PyLong_Check(o)) return checked(static_cast<uint32_t>(PyLong_AsUnsignedLongMask(o)));
        PyObject* v = PyNumber_Index(o);
        if (v == nullptr) { ok_ = false; return 0; }
        const uint32_t r = static_cast<uint32_t>(PyLong_AsUnsignedLongMask(v));
        Py_DECREF(v);
        return checked(r);
    }
    float f32() {
        if (!ok_) return 0.0f;
        const double v = PyFloat_AsDouble(args_[i_++]);
        if (v == -1.0 && PyErr_Occurred()) ok_ = false;
        return static_cast<float>(v);
    }
    int rope() {   // an enum member, or anything else that int() takes
        if (!ok_) return 0;
        PyObject* v = PyNumber_Long(args_[i_++]);
        if (v == nullptr) { ok_ = false; return 0; }
        const uint32_t r = checked(static_cast<uint32_t>(PyLong_AsUnsignedLongMask(v)));
        Py_DECREF(v);
        return static_cast<int>(r);
    }
    // A cache view (the ctypes structure and nothing else): its memory, through the buffer protocol.
    const b200kv_view* view() {
        if (!ok_) return nullptr;
        const int is_view = PyObject_IsInstance(args_[i_], g_view_type);
        if (is_view <= 0) {
            if (is_view == 0) PyErr_Format(PyExc_TypeError, "expected a cache view, got %s", Py_TYPE(args_[i_])->tp_name);
            ok_ = false;
            return nullptr;
        }
        return views(1, false);
    }
    // An array of them (the caller has built it), or None.
    const b200kv_view* views(uint32_t count, bool optional) {
        if (!ok_) return nullptr;
        PyObject* o = args_[i_++];
        if (optional && o == Py_None) return nullptr;
        if (PyObject_GetBuffer(o, &buffers_[held_], PyBUF_SIMPLE) != 0) { ok_ = false; return nullptr; }
        const Py_buffer& b = buffers_[held_++];
        if (static_cast<size_t>(b.len) < sizeof(b200kv_view) * static_cast<size_t>(count)) {
            fail(PyExc_ValueError, "not a cache view");
            return nullptr;
        }
        return static_cast<const b200kv_view*>(b.buf);
    }
    void* stream() {   // None = torch's current stream
        if (!ok_) return nullptr;
        PyObject* o = args_[i_++];
        if (o == Py_None) return c10::cuda::getCurrentCUDAStream().stream();
        PyObject* h = PyObject_GetAttrString(o, "cuda_stream");
        if (h == nullptr) { ok_ = false; return nullptr; }
        void* s = PyLong_AsVoidPtr(h);
        Py_DECREF(h);
        if (s == nullptr && PyErr_Occurred()) ok_ = false;
        return s;
    }
    void* handle() {   // an address as an int, None = null
        if (!ok_) return nullptr;
        PyObject* o = args_[i_++];
        if (o == Py_None) return nullptr;
        void* p = PyLong_AsVoidPtr(o);
        if (p == nullptr && PyErr_Occurred()) ok_ = false;
        return p;
    }
    PyObject* object() { return ok_ ? args_[i_++] : nullptr; }
    void* fail(PyObject* type, const char* text) {
        if (ok_) PyErr_SetString(type, text);
        ok_ = false;
        return nullptr;
    }

private:
    uint32_t checked(uint32_t v) {
        if (v == 0xffffffffu && PyErr_Occurred()) ok_ = false;
        return v;
    }
    PyObject* const* args_;
    Py_ssize_t i_ = 0;
    bool ok_ = true;
    int held_ = 0;
    Py_buffer buffers_[2];
};

template <typename F>
PyObject* call(Args& a, F&& f) {
    if (!a.ok()) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f();
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

PyObject* py_append(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Args a(args, n, 12);
    int kd = 0, vd = 0;
    const b200kv_view* view = a.view();
    const void* key = a.tensor(nullptr, &kd);
    const void* value = a.tensor(nullptr, &vd);
    if (a.ok() && kd != vd) a.fail(PyExc_ValueError, "key and value must share a dtype");
    const float* w = a.tensor_as<const float>();
    const int rope = a.rope();
    const float theta = a.f32(), eps = a.f32();
    const uint32_t count = a.u32(), base = a.u32();
    const auto* ps = a.tensor_as<const b200kv_prefill_state>();
    const auto* ds = a.tensor_as<const b200kv_decode_state>();
    void* s = a.stream();
    return call(a, [&] { return g_api.append(view, key, value, kd, w, rope, theta, eps, count, base, ps, ds, s); });
}

PyObject* py_q_split_norm_rope(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Args a(args, n, 14);
    int id = 0, od = 0;
    const void* qfull = a.tensor(nullptr, &id);
    const float* w = a.tensor_as<const float>();
    void* query = a.tensor(nullptr, &od);
    float* gate = a.tensor_as<float>();
    const uint32_t count = a.u32(), base = a.u32(), heads = a.u32(), dim = a.u32();
    const int rope = a.rope();
    const float theta = a.f32(), eps = a.f32();
    const auto* ps = a.tensor_as<const b200kv_prefill_state>();
    const auto* ds = a.tensor_as<const b200kv_decode_state>();
    void* s = a.stream();
    return call(a, [&] { return g_api.q_split_norm_rope(qfull, id, w, query, od, gate, count, base, heads, dim, rope, theta, eps, ps, ds, s); });
}

PyObject* py_decode_attn(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Args a(args, n, 13);
    int qd = 0;
    int64_t ws_bytes = 0;
    const b200kv_view* view = a.view();
    const void* q = a.tensor(nullptr, &qd);
    const float* gate = a.tensor_as<const float>();
    float* out = a.tensor_as<float>();
    float* gated = a.tensor_as<float>();
    auto* q8 = a.tensor_as<b200kv_q8_1_block>();
    const uint32_t heads = a.u32();
    const float scale = a.f32();
    const uint32_t length = a.u32();
    const auto* ds = a.tensor_as<const b200kv_decode_state>();
    void* ws = a.tensor(&ws_bytes);
    const uint32_t splits = a.u32();
    void* s = a.stream();
    return call(a, [&] {
        return g_api.decode_attn(view, q, qd, gate, out, gated, q8, heads, scale, length, ds, ws, static_cast<size_t>(ws_bytes), splits, s);
    });
}

PyObject* py_decode_step(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Args a(args, n, 19);
    int kd = 0, vd = 0, qd = 0;
    int64_t ws_bytes = 0;
    const b200kv_view* view = a.view();
    const void* key = a.tensor(nullptr, &kd);
    const void* value = a.tensor(nullptr, &vd);
    if (a.ok() && kd != vd) a.fail(PyExc_ValueError, "key and value must share a dtype");
    const float* w = a.tensor_as<const float>();
    const int rope = a.rope();
    const float theta = a.f32(), eps = a.f32();
    const void* q = a.tensor(nullptr, &qd);
    const float* gate = a.tensor_as<const float>();
    float* out = a.tensor_as<float>();
    float* gated = a.tensor_as<float>();
    auto* q8 = a.tensor_as<b200kv_q8_1_block>();
    const uint32_t heads = a.u32();
    const float scale = a.f32();
    const uint32_t position = a.u32();
    const auto* ds = a.tensor_as<const b200kv_decode_state>();
    void* ws = a.tensor(&ws_bytes);
    const uint32_t splits = a.u32();
    void* s = a.stream();
    return call(a, [&] {
        return g_api.decode_step(view, key, value, kd, w, rope, theta, eps, q, qd, gate, out, gated, q8, heads, scale, position, ds, ws,
                                 static_cast<size_t>(ws_bytes), splits, s);
    });
}

PyObject* py_decode_attn_batched(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Args a(args, n, 13);
    int qd = 0;
    int64_t ws_bytes = 0, sessions = 0;
    PyObject* views_arg = a.object();
    void* table = a.tensor();
    const uint32_t* lengths = a.tensor_as<const uint32_t>(&sessions);
    const uint32_t max_length = a.u32();
    const void* q = a.tensor(nullptr, &qd);
    const float* gate = a.tensor_as<const float>();
    float* out = a.tensor_as<float>();
    float* gated = a.tensor_as<float>();
    const uint32_t heads = a.u32();
    const float scale = a.f32();
    void* ws = a.tensor(&ws_bytes);
    const uint32_t splits = a.u32();
    void* s = a.stream();
    Args v(&views_arg, 1, 1);
    const b200kv_view* views = a.ok() ? v.views(static_cast<uint32_t>(sessions), true) : nullptr;
    if (a.ok() && !v.ok()) return nullptr;
    return call(a, [&] {
        return g_api.decode_attn_batched(views, table, lengths, static_cast<uint32_t>(sessions), max_length, q, qd, gate, out, gated, heads, scale,
                                         ws, static_cast<size_t>(ws_bytes), splits, s);
    });
}

PyObject* py_suffix_attn(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Args a(args, n, 12);
    int qd = 0;
    int64_t ws_bytes = 0;
    const b200kv_view* view = a.view();
    const void* q = a.tensor(nullptr, &qd);
    const float* gate = a.tensor_as<const float>();
    float* gated = a.tensor_as<float>();
    const uint32_t count = a.u32(), base = a.u32(), heads = a.u32();
    const float scale = a.f32();
    const auto* ps = a.tensor_as<const b200kv_prefill_state>();
    void* ws = a.tensor(&ws_bytes);
    const uint32_t prepared = a.u32();
    void* s = a.stream();
    return call(a, [&] {
        return g_api.prefill_attn_prepared(view, q, qd, gate, gated, count, base, heads, scale, ps, ws, static_cast<size_t>(ws_bytes), prepared, s);
    });
}

// ---- the snapshot pool: token ids and storage objects in, one library call ------------------------------------

// Anything with a length that can be iterated over, as a list or tuple.
PyObject* items_of(PyObject* o, const char* text) { return PyObject_Size(o) < 0 ? nullptr : PySequence_Fast(o, text); }

bool read_tokens(PyObject* seq, std::vector<uint32_t>& out) {
    PyObject* fast = items_of(seq, "a sequence of token ids is required");
    if (fast == nullptr) return false;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
    PyObject** items = PySequence_Fast_ITEMS(fast);
    out.resize(static_cast<size_t>(n));
    for (Py_ssize_t i = 0; i < n; ++i) {
        if (PyLong_Check(items[i])) {
            out[i] = static_cast<uint32_t>(PyLong_AsUnsignedLongMask(items[i]));
            continue;
        }
        PyObject* v = PyNumber_Index(items[i]);
        if (v == nullptr) { Py_DECREF(fast); return false; }
        out[i] = static_cast<uint32_t>(PyLong_AsUnsignedLongMask(v));
        Py_DECREF(v);
    }
    Py_DECREF(fast);
    return true;
}

enum Name { KEY, VALUE, KEY_Q8, KEY_SCALES, VALUE_Q8, VALUE_SCALES, CAPACITY, KV_HEADS, HEAD_DIM, QBLOCK, QUANT_MODE, VIEW, NAMES };
PyObject* g_names[NAMES];

bool plane(PyObject* o, Name name, void** out) {
    PyObject* t = PyObject_GetAttr(o, g_names[name]);
    if (t == nullptr) return false;
    *out = nullptr;
    if (t != Py_None) {
        if (!THPVariable_Check(t) || !THPVariable_Unpack(t).is_cuda() || !THPVariable_Unpack(t).is_contiguous()) {
            Py_DECREF(t);
            PyErr_SetString(PyExc_ValueError, "expected a contiguous CUDA tensor");
            return false;
        }
        *out = THPVariable_Unpack(t).data_ptr();
    }
    Py_DECREF(t);
    return true;
}
bool number(PyObject* o, Name name, uint64_t* out) {
    PyObject* v = PyObject_GetAttr(o, g_names[name]);
    if (v == nullptr) return false;
    *out = PyLong_AsUnsignedLongLongMask(v);
    Py_DECREF(v);
    return !(*out == ~0ull && PyErr_Occurred());
}

PyObject* g_storage_view;   // AttentionLayerKvCacheStorage.view

// The views of a sequence of cache storages: what their view() returns.  Where that is AttentionLayerKvCacheStorage's own, its
// result is read from the attributes it would take it from (a view() in Python costs 3 us a layer).
bool read_view(PyObject* o, b200kv_view& v) {
    PyObject* method = PyObject_GetAttr(o, g_names[VIEW]);
    if (method == nullptr) return false;
    const bool own = PyMethod_Check(method) && PyMethod_GET_FUNCTION(method) == g_storage_view && PyMethod_GET_SELF(method) == o;
    PyObject* result = own ? nullptr : PyObject_CallNoArgs(method);
    Py_DECREF(method);
    if (!own) {
        if (result == nullptr) return false;
        Args a(&result, 1, 1);
        const b200kv_view* view = a.view();
        if (view != nullptr) v = *view;
        Py_DECREF(result);
        return a.ok();
    }
    void *kq, *vq;
    uint64_t cap, heads, dim, qb, mode;
    if (!(plane(o, KEY, &v.key_f16) && plane(o, VALUE, &v.value_f16) && plane(o, KEY_Q8, &kq) && plane(o, KEY_SCALES, &v.key_scales) &&
          plane(o, VALUE_Q8, &vq) && plane(o, VALUE_SCALES, &v.value_scales) && number(o, CAPACITY, &cap) && number(o, KV_HEADS, &heads) &&
          number(o, HEAD_DIM, &dim) && number(o, QBLOCK, &qb) && number(o, QUANT_MODE, &mode)))
        return false;
    v.key_q8 = static_cast<int8_t*>(kq);
    v.value_q8 = static_cast<int8_t*>(vq);
    v.capacity = cap;
    v.kv_heads = static_cast<uint32_t>(heads);
    v.head_dim = static_cast<uint32_t>(dim);
    v.qblock = static_cast<uint32_t>(qb);
    v.quant_mode = static_cast<uint32_t>(mode);
    return true;
}
bool read_views(PyObject* storages, std::vector<b200kv_view>& out) {
    PyObject* fast = items_of(storages, "a sequence of cache storages is required");
    if (fast == nullptr) return false;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
    out.resize(static_cast<size_t>(n));
    bool ok = true;
    for (Py_ssize_t i = 0; i < n && ok; ++i) ok = read_view(PySequence_Fast_GET_ITEM(fast, i), out[i]);
    Py_DECREF(fast);
    return ok;
}

// (pool, tokens, storages, stream) -> (status, captured or matched length)
template <bool CAPTURE>
PyObject* py_pool(PyObject*, PyObject* const* args, Py_ssize_t n) {
    Args a(args, n, 4);
    auto* pool = static_cast<b200kv_pool*>(a.handle());
    PyObject* tokens_arg = a.object();
    PyObject* storages = a.object();
    void* s = a.stream();
    if (!a.ok()) return nullptr;
    std::vector<uint32_t> tokens;
    std::vector<b200kv_view> views;
    if (!read_tokens(tokens_arg, tokens) || !read_views(storages, views)) return nullptr;
    const uint32_t count = static_cast<uint32_t>(tokens.size()), layers = static_cast<uint32_t>(views.size());
    static const uint32_t no_token = 0;   // an empty sequence still passes an address
    const uint32_t* ids = count ? tokens.data() : &no_token;
    const b200kv_view empty{};
    const b200kv_view* layer_views = layers ? views.data() : &empty;
    int rc, captured = 0;
    uint32_t matched = 0;
    Py_BEGIN_ALLOW_THREADS
    if (CAPTURE) rc = g_api.pool_capture(pool, ids, count, layer_views, layers, s, &captured);
    else rc = g_api.pool_restore(pool, ids, count, layer_views, layers, s, &matched);
    Py_END_ALLOW_THREADS
    return Py_BuildValue("iI", rc, CAPTURE ? static_cast<unsigned>(captured) : matched);
}

PyObject* py_bind(PyObject*, PyObject* arg) {   // {name: address}, and "View": the structure
    PyObject* view = PyDict_GetItemString(arg, "View");
    if (view == nullptr || !PyType_Check(view)) return PyErr_Format(PyExc_KeyError, "View");
    Py_INCREF(view);
    Py_XSETREF(g_view_type, view);
    struct { const char* name; void** slot; } table[] = {
        {"b200kv_append", reinterpret_cast<void**>(&g_api.append)},
        {"b200kv_q_split_norm_rope", reinterpret_cast<void**>(&g_api.q_split_norm_rope)},
        {"b200kv_decode_attn", reinterpret_cast<void**>(&g_api.decode_attn)},
        {"b200kv_decode_step", reinterpret_cast<void**>(&g_api.decode_step)},
        {"b200kv_decode_attn_batched", reinterpret_cast<void**>(&g_api.decode_attn_batched)},
        {"b200kv_prefill_attn_prepared", reinterpret_cast<void**>(&g_api.prefill_attn_prepared)},
        {"b200kv_pool_capture", reinterpret_cast<void**>(&g_api.pool_capture)},
        {"b200kv_pool_restore", reinterpret_cast<void**>(&g_api.pool_restore)},
    };
    for (auto& e : table) {
        PyObject* v = PyDict_GetItemString(arg, e.name);
        if (v == nullptr) return PyErr_Format(PyExc_KeyError, "%s", e.name);
        *e.slot = PyLong_AsVoidPtr(v);
        if (*e.slot == nullptr) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "%s has no address", e.name);
    }
    Py_RETURN_NONE;
}

PyObject* py_bind_storage(PyObject*, PyObject* view) {   // AttentionLayerKvCacheStorage.view
    Py_INCREF(view);
    Py_XSETREF(g_storage_view, view);
    Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n) {   // no C++ exception reaches the interpreter
    try {
        return F(self, args, n);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}
#define ENTRY(name, f) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<f>)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {{"bind", py_bind, METH_O, nullptr},
                           {"bind_storage", py_bind_storage, METH_O, nullptr},
                           ENTRY("append", py_append),
                           ENTRY("q_split_norm_rope", py_q_split_norm_rope),
                           ENTRY("decode_attn", py_decode_attn),
                           ENTRY("decode_step", py_decode_step),
                           ENTRY("decode_attn_batched", py_decode_attn_batched),
                           ENTRY("suffix_attn", py_suffix_attn),
                           ENTRY("pool_capture", py_pool<true>),
                           ENTRY("pool_restore", py_pool<false>),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    const char* names[NAMES] = {"key_cache", "value_cache", "key_cache_q8", "key_scales", "value_cache_q8", "value_scales",
                                "capacity", "kv_heads", "head_dim", "qblock", "quant_mode", "view"};
    for (int i = 0; i < NAMES; ++i) {
        g_names[i] = PyUnicode_InternFromString(names[i]);
        if (g_names[i] == nullptr) return nullptr;
    }
    return PyModule_Create(&g_module);
}
