// The host side of the per-layer launches, natively: what kernel.ChainBatch and core.decode_batch do between the caller
// and the C ABI -- unwrap the views, check every extent against the geometry, pick the stream, launch.
//
// A decode step makes one such call per layer.  In Python the checks and the foreign call of 33 arguments take about
// 20 us (chain) and 15 us (core) a layer, several times what the kernel of a small batch runs for (4 us at one slot):
// the GPU waits for the host.  Here a call is 2 to 4 us, most of it the launch itself.
//
// Every function answers -1 when the call is not the plain accepted one: a check fails, an argument is of a type it
// does not know, a subclass, a tensor on the CPU.  Nothing has been enqueued then and the caller runs the Python code,
// which holds the same checks and raises the errors.  Any other answer is the launcher's status.

#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "glm53f_kda.h"

namespace {

constexpr int64_t kD = 128, kWindow = 3;

// Interned attribute names.
struct Names {
    PyObject *t, *buf, *offset, *stride, *weights, *heads, *conv_w, *a_log, *dt_bias, *norm_w, *eps, *lower, *p, *b_off, *a, *g, *conv, *state, *state_out,
        *out, *saves, *kind, *rows, *k, *v, *b, *fast, *cu_rows, *conv_off, *state_off, *stream, *cuda_stream;
} N;

// The exact Python types the fast path knows (set once by bind()).
PyObject *T_buffer = nullptr, *T_view = nullptr, *T_weights = nullptr, *T_saves = nullptr, *T_chain = nullptr, *T_meta = nullptr, *T_stream = nullptr;

struct Miss {};  // thrown to leave for the Python path

struct Ref {  // an owned reference
    PyObject* o;
    explicit Ref(PyObject* x) : o(x) {
        if (o == nullptr) throw Miss{};
    }
    Ref(const Ref&) = delete;
    Ref& operator=(const Ref&) = delete;
    ~Ref() { Py_DECREF(o); }
};
inline PyObject* get(PyObject* o, PyObject* name) { return PyObject_GetAttr(o, name); }
inline int64_t to_i64(PyObject* o) {
    if (!PyLong_CheckExact(o)) throw Miss{};
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw Miss{};
    return v;
}
inline int64_t get_i64(PyObject* o, PyObject* name) {
    Ref r(get(o, name));
    return to_i64(r.o);
}
inline double get_f64(PyObject* o, PyObject* name) {
    Ref r(get(o, name));
    if (!PyFloat_CheckExact(r.o)) throw Miss{};
    return PyFloat_AS_DOUBLE(r.o);
}
inline void is_exactly(PyObject* o, PyObject* type) {
    if (reinterpret_cast<PyObject*>(Py_TYPE(o)) != type) throw Miss{};
}
// A launch without the interpreter's lock, as a foreign call makes it: a full launch queue blocks the caller, and what it waits for
// may be a host function that needs the lock.  Everything Python has been read by then.
template <typename F>
int unlocked(F&& launch) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = launch();
    Py_END_ALLOW_THREADS
    return rc;
}

inline const at::Tensor& tensor(PyObject* o) {
    if (!THPVariable_Check(o)) throw Miss{};
    return THPVariable_Unpack(o);
}

// The tensors whose addresses a launch takes, held until it is out: another thread may let go of them meanwhile.
struct Held {
    PyObject* o[24];
    int n = 0;
    PyObject* add(PyObject* x) {
        if (n == 24) throw Miss{};
        Py_INCREF(x);
        return o[n++] = x;
    }
    ~Held() {
        while (n > 0) Py_DECREF(o[--n]);
    }
};

struct Buffer {  // a DeviceBuffer: address and bytes
    unsigned char* ptr;
    int64_t bytes;
};
inline Buffer buffer(PyObject* o, Held& held) {
    is_exactly(o, T_buffer);
    Ref t(get(o, N.t));
    const at::Tensor& x = tensor(held.add(t.o));
    if (!x.is_cuda()) throw Miss{};
    const int64_t n = x.numel();
    return {n != 0 ? static_cast<unsigned char*>(x.data_ptr()) : nullptr, n};
}
inline Buffer get_buffer(PyObject* o, PyObject* name, Held& held) {
    Ref r(get(o, name));
    return buffer(r.o, held);
}
// a * b + c, exactly.
inline int64_t mul_add(int64_t a, int64_t b, int64_t c) {
    int64_t r;
    if (__builtin_mul_overflow(a, b, &r) || __builtin_add_overflow(r, c, &r)) throw Miss{};
    return r;
}
// Elements [offset, offset + n) of `size` bytes lie inside the buffer.
inline void region(const Buffer& b, int64_t size, int64_t offset, int64_t n) {
    if (offset < 0 || mul_add(offset, 1, n) > b.bytes / size) throw Miss{};
}

struct Rows {
    glm53f_bf16* ptr;
    int64_t stride;
};
// A RowView of bf16 rows whose columns [lo, hi) lie inside its buffer for `rows` rows.
inline Rows rows_of(PyObject* owner, PyObject* name, int64_t rows, int64_t lo, int64_t hi, Held& held) {
    Ref v(get(owner, name));
    is_exactly(v.o, T_view);
    const Buffer b = get_buffer(v.o, N.buf, held);
    const int64_t offset = get_i64(v.o, N.offset), stride = get_i64(v.o, N.stride);
    if (rows > 0 && (mul_add(offset, 1, lo) < 0 || mul_add(rows - 1, stride, mul_add(offset, 1, hi)) > b.bytes / 2)) throw Miss{};
    return {reinterpret_cast<glm53f_bf16*>(b.ptr) + offset, stride};
}

inline glm53f_stream_t stream_of(PyObject* s) {
    is_exactly(s, T_stream);
    Ref given(get(s, N.stream));
    if (given.o == Py_None) return reinterpret_cast<glm53f_stream_t>(c10::cuda::getCurrentCUDAStream().stream());
    Ref raw(get(given.o, N.cuda_stream));
    return reinterpret_cast<glm53f_stream_t>(static_cast<uintptr_t>(to_i64(raw.o)));
}

// chain_batch(ChainBatch, BatchMeta, Stream, bf16_state) -> status, or -1.  kernel.ChainBatch._launch_as holds the checks
// in the order they raise.
int chain_batch(PyObject* cb, PyObject* meta, PyObject* stream, bool bf16) {
    is_exactly(cb, T_chain);
    is_exactly(meta, T_meta);
    // (requests, rows, then per kind of offset: least, greatest, least distance between two), kept by BatchMeta.set
    Ref fast(get(meta, N.fast));
    if (!PyTuple_CheckExact(fast.o) || PyTuple_GET_SIZE(fast.o) != 8) throw Miss{};
    int64_t m[8];
    for (int i = 0; i < 8; ++i) m[i] = to_i64(PyTuple_GET_ITEM(fast.o, i));
    const int64_t batch = m[0], total = m[1];
    Held held;
    Ref w(get(cb, N.weights));
    is_exactly(w.o, T_weights);
    const int64_t heads = get_i64(w.o, N.heads), es = bf16 ? 2 : 4;
    if (heads < 1 || heads > 65535 || batch < 1) throw Miss{};
    const int64_t channels = 3 * heads * kD, width = heads * kD, state_len = heads * kD * kD;
    const int64_t b_off = get_i64(cb, N.b_off);
    const int64_t b_end = mul_add(b_off, 1, heads);
    const Rows p = rows_of(cb, N.p, total, b_off < 0 ? b_off : 0, b_end > channels ? b_end : channels, held);
    const Rows a = rows_of(cb, N.a, total, 0, width, held), g = rows_of(cb, N.g, total, 0, width, held), out = rows_of(cb, N.out, total, 0, width, held);
    if (total > 1 && out.stride < width) throw Miss{};
    const Buffer conv = get_buffer(cb, N.conv, held), state = get_buffer(cb, N.state, held);
    region(conv, 2, m[2], kWindow * channels);
    region(conv, 2, m[3], kWindow * channels);
    region(state, es, m[5], state_len);
    region(state, es, m[6], state_len);
    if (m[7] < state_len) throw Miss{};
    void* state_out = nullptr;
    {
        Ref so(get(cb, N.state_out));
        Ref kind(get(so.o, N.kind));
        if (!PyUnicode_CheckExact(kind.o)) throw Miss{};
        if (PyUnicode_CompareWithASCIIString(kind.o, "in_place") == 0) state_out = state.ptr;
        else if (PyUnicode_CompareWithASCIIString(kind.o, "skip") != 0) throw Miss{};
    }
    void *ks = nullptr, *vs = nullptr, *gs = nullptr, *bs = nullptr;
    {
        Ref s(get(cb, N.saves));
        if (s.o != Py_None) {
            is_exactly(s.o, T_saves);
            if (get_i64(s.o, N.heads) != heads || get_i64(s.o, N.rows) < total) throw Miss{};
            ks = get_buffer(s.o, N.k, held).ptr;
            vs = get_buffer(s.o, N.v, held).ptr;
            gs = get_buffer(s.o, N.g, held).ptr;
            bs = get_buffer(s.o, N.b, held).ptr;
        }
    }
    const auto* cu = reinterpret_cast<const int32_t*>(get_buffer(meta, N.cu_rows, held).ptr);
    const auto* conv_off = reinterpret_cast<const int64_t*>(get_buffer(meta, N.conv_off, held).ptr);
    const auto* state_off = reinterpret_cast<const int64_t*>(get_buffer(meta, N.state_off, held).ptr);
    const auto* conv_w = reinterpret_cast<const glm53f_bf16*>(get_buffer(w.o, N.conv_w, held).ptr);
    const auto* a_log = reinterpret_cast<const float*>(get_buffer(w.o, N.a_log, held).ptr);
    const auto* dt_bias = reinterpret_cast<const float*>(get_buffer(w.o, N.dt_bias, held).ptr);
    const auto* norm_w = reinterpret_cast<const glm53f_bf16*>(get_buffer(w.o, N.norm_w, held).ptr);
    const float eps = (float)get_f64(w.o, N.eps), lower = (float)get_f64(w.o, N.lower);
    const glm53f_stream_t st = stream_of(stream);
    auto launch = [&](auto fn, auto* s_in, auto* s_out) {
        return unlocked([&] {
            return fn((int32_t)heads, (int32_t)batch, cu, p.ptr, p.stride, b_off, a.ptr, a.stride, g.ptr, g.stride, reinterpret_cast<const glm53f_bf16*>(conv.ptr),
                      conv_off, conv_w, s_in, s_out, state_off, a_log, dt_bias, norm_w, eps, lower, out.ptr, out.stride, static_cast<float*>(ks),
                      static_cast<glm53f_bf16*>(vs), static_cast<float*>(gs), static_cast<float*>(bs), st);
        });
    };
    if (bf16) return launch(glm53f_kda_chain_batch_bf16state, reinterpret_cast<const glm53f_bf16*>(state.ptr), static_cast<glm53f_bf16*>(state_out));
    return launch(glm53f_kda_chain_batch, reinterpret_cast<const float*>(state.ptr), static_cast<float*>(state_out));
}

// A contiguous CUDA tensor of the kind's element type with at least n elements.
enum Kind { kBf16, kF32, kI32, kI64 };
template <typename T>
T* need(PyObject* o, Kind kind, int64_t n) {
    const at::Tensor& t = tensor(o);
    const auto d = t.scalar_type();
    const bool ok = kind == kBf16  ? d == at::kBFloat16 || d == at::kShort || d == at::kUInt16
                    : kind == kF32 ? d == at::kFloat
                    : kind == kI32 ? d == at::kInt
                                   : d == at::kLong;
    if (!ok || !t.is_cuda() || !t.is_contiguous() || t.numel() < n) throw Miss{};
    return static_cast<T*>(t.data_ptr());
}

// core_decode(heads, rows, cu_rows, q, k, v, g, beta, state, state_off, state_out, flags, gate, norm_w, eps, out, saves,
// max_state_off) -> status, or -1.  core.decode_batch holds the checks in the order they raise.
int core_decode(PyObject* const* a) {
    const int64_t heads = to_i64(a[0]), rows = to_i64(a[1]), flags = to_i64(a[11]);
    if (heads < 1 || heads > 65535 || rows < 0 || rows > 0x7fffffff || flags < 0 || flags > 0x7fffffff) throw Miss{};
    const int64_t n = rows * heads * kD;
    const auto* cu = need<const int32_t>(a[2], kI32, 2);
    const int64_t batch = tensor(a[2]).numel() - 1;
    if (batch > 65535) throw Miss{};
    const auto *q = need<const glm53f_bf16>(a[3], kBf16, n), *k = need<const glm53f_bf16>(a[4], kBf16, n), *v = need<const glm53f_bf16>(a[5], kBf16, n);
    const auto* g = need<const float>(a[6], kF32, n);
    const auto* beta = need<const float>(a[7], kF32, rows * heads);
    const auto* off = need<const int64_t>(a[9], kI64, batch);
    const at::Tensor& state = tensor(a[8]);
    const auto sd = state.scalar_type();
    if (!state.is_cuda()) throw Miss{};
    const int32_t kind = sd == at::kFloat ? 0 : sd == at::kBFloat16 || sd == at::kShort || sd == at::kUInt16 ? 1 : -1;
    if (kind < 0) throw Miss{};
    if (a[17] != Py_None && state.numel() < mul_add(to_i64(a[17]), 1, heads * kD * kD)) throw Miss{};
    void* so = nullptr;
    if (PyUnicode_Check(a[10])) so = state.data_ptr();
    else if (a[10] != Py_None) {
        const at::Tensor& t = tensor(a[10]);
        if (!t.is_cuda() || t.scalar_type() != sd || t.numel() < state.numel()) throw Miss{};
        so = t.data_ptr();
    }
    const glm53f_bf16 *gate = nullptr, *norm_w = nullptr;
    if (a[12] != Py_None) {
        gate = need<const glm53f_bf16>(a[12], kBf16, n);
        norm_w = need<const glm53f_bf16>(a[13], kBf16, kD);
    } else if (a[13] != Py_None) {
        norm_w = static_cast<const glm53f_bf16*>(tensor(a[13]).data_ptr());
    }
    if (!PyFloat_CheckExact(a[14])) throw Miss{};
    const float eps = (float)PyFloat_AS_DOUBLE(a[14]);
    auto* out = need<glm53f_bf16>(a[15], kBf16, n);
    const auto st = reinterpret_cast<glm53f_stream_t>(c10::cuda::getCurrentCUDAStream().stream());
    const void* si = state.data_ptr();
    // (the caller's frame holds the tensors)
    if (a[16] == Py_None)
        return unlocked([&] {
            return glm53f_kda_core_decode_batch((int32_t)heads, (int32_t)batch, cu, q, k, v, g, beta, si, so, off, kind, (int32_t)flags, gate, norm_w, eps, out, st);
        });
    if (!PyTuple_CheckExact(a[16]) || PyTuple_GET_SIZE(a[16]) != 4) throw Miss{};
    auto* ks = need<float>(PyTuple_GET_ITEM(a[16], 0), kF32, n);
    auto* vs = need<glm53f_bf16>(PyTuple_GET_ITEM(a[16], 1), kBf16, n);
    auto* gs = need<float>(PyTuple_GET_ITEM(a[16], 2), kF32, n);
    auto* bs = need<float>(PyTuple_GET_ITEM(a[16], 3), kF32, rows * heads);
    return unlocked([&] {
        return glm53f_kda_core_verify_batch((int32_t)heads, (int32_t)batch, cu, q, k, v, g, beta, si, so, off, kind, (int32_t)flags, gate, norm_w, eps, out, ks, vs,
                                            gs, bs, st);
    });
}

template <typename F>
PyObject* answer(F&& f) {
    long code = -1;
    try {
        code = f();
    } catch (const Miss&) {
        PyErr_Clear();
        code = -1;
    } catch (const std::exception&) {
        PyErr_Clear();
        code = -1;
    }
    return PyLong_FromLong(code);
}

PyObject* py_chain_batch(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return answer([&] { return n == 4 && T_chain != nullptr ? chain_batch(args[0], args[1], args[2], args[3] == Py_True) : -1; });
}
PyObject* py_core_decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return answer([&] { return n == 18 ? core_decode(args) : -1; });
}
// raw_stream(Stream) -> the CUDA stream's address, or None for a stream it does not know.
PyObject* py_raw_stream(PyObject*, PyObject* s) {
    try {
        return PyLong_FromVoidPtr(stream_of(s));
    } catch (const std::exception&) {
    } catch (const Miss&) {
    }
    PyErr_Clear();
    Py_RETURN_NONE;
}
// bind(DeviceBuffer, RowView, Weights, Saves, ChainBatch, BatchMeta, Stream): the types the fast path accepts, exactly.
PyObject* py_bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 7) {
        PyErr_SetString(PyExc_TypeError, "bind takes seven types");
        return nullptr;
    }
    PyObject** slots[7] = {&T_buffer, &T_view, &T_weights, &T_saves, &T_chain, &T_meta, &T_stream};
    for (int i = 0; i < 7; ++i) {
        Py_INCREF(args[i]);
        Py_XDECREF(*slots[i]);
        *slots[i] = args[i];
    }
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_bind)), METH_FASTCALL, nullptr},
    {"chain_batch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_chain_batch)), METH_FASTCALL, nullptr},
    {"raw_stream", py_raw_stream, METH_O, nullptr},
    {"core_decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_core_decode)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host path of the per-layer launches.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
#define NAME(field, text) N.field = PyUnicode_InternFromString(text)
    NAME(t, "t"); NAME(buf, "buf"); NAME(offset, "offset"); NAME(stride, "stride"); NAME(weights, "weights"); NAME(heads, "heads"); NAME(conv_w, "conv_w");
    NAME(a_log, "a_log"); NAME(dt_bias, "dt_bias"); NAME(norm_w, "norm_w"); NAME(eps, "eps"); NAME(lower, "lower"); NAME(p, "p"); NAME(b_off, "b_off");
    NAME(a, "a"); NAME(g, "g"); NAME(conv, "conv"); NAME(state, "state"); NAME(state_out, "state_out"); NAME(out, "out"); NAME(saves, "saves");
    NAME(kind, "kind"); NAME(rows, "rows"); NAME(k, "k"); NAME(v, "v"); NAME(b, "b"); NAME(fast, "_extent"); NAME(cu_rows, "cu_rows");
    NAME(conv_off, "conv_off"); NAME(state_off, "state_off"); NAME(stream, "stream"); NAME(cuda_stream, "cuda_stream");
#undef NAME
    PyObject* m = PyModule_Create(&module);
    if (m != nullptr && PyModule_AddStringConstant(m, "built_for", HOST_BUILT_FOR) != 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
