// Python module over the C ABI (include/b200attn.h): argument checks, the current stream, the scratch buffers and the
// call itself in one native function per operator.
//
// What bounds it: nothing but the launches should.  Through ctypes an operator cost 15-25 us of host time on B200's
// host (per tensor five attribute and method calls, a device context manager, a stream object, fifteen argument
// conversions), more than the kernels of a small problem take on the GPU.  Here the same checks read the tensors' C++
// fields: an operator costs 0.6 to 1.2 us beside the C ABI call under it, which is 2.5 us for the append or the decode and
// 3.3 us for the forward, nearly all of it the driver's launch.
//
// The Python functions keep names, defaults and documentation (flash_attn.py, rope_norm.py, kv_cache.py); the checks,
// their order and their messages are here: every dtype first, then every device, like the reference
// (llm/src/model/flash_attn.cu:386-407,433-455).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstring>
#include <list>
#include <memory>
#include <mutex>
#include <vector>

#include "../../include/b200attn.h"

namespace {

using at::ScalarType;

// ---- errors: the Python error is set, nullptr / false says so
PyObject* value_error(const char* fmt, ...) {
    char buf[256];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    PyErr_SetString(PyExc_ValueError, buf);
    return nullptr;
}

// status -> the reference's exception types (std::invalid_argument, std::runtime_error)
PyObject* finish(int status, const char* where) {
    if (status == B200ATTN_OK) Py_RETURN_NONE;
    const bool arg = status == B200ATTN_ERR_INVALID_ARG || status == B200ATTN_ERR_UNSUPPORTED ||
                     status == B200ATTN_ERR_ALIGNMENT || status == B200ATTN_ERR_WORKSPACE || status == B200ATTN_ERR_TOO_LARGE;
    PyErr_Format(arg ? PyExc_ValueError : PyExc_RuntimeError, "%s: %s (status %d)", where, b200attn_strerror(status), status);
    return nullptr;
}

// ---- arguments
struct Item {  // one tensor argument
    PyObject* obj;
    const char* name;  // in messages
    ScalarType type;
};

const at::Tensor& unpack(PyObject* o) { return THPVariable_Unpack(o); }
void* ptr(PyObject* o) { return unpack(o).data_ptr(); }
int64_t numel(PyObject* o) { return unpack(o).numel(); }

const char* type_name(ScalarType t) { return t == ScalarType::BFloat16 ? "BF16" : "FP32"; }

// every dtype first, then every device, then contiguity
bool check_tensors(const char* fn, const Item* items, int n) {
    for (int i = 0; i < n; ++i) {
        if (!THPVariable_Check(items[i].obj)) {
            value_error("%s: %s must be a tensor", fn, items[i].name);
            return false;
        }
        if (unpack(items[i].obj).scalar_type() != items[i].type) {
            value_error("%s: %s must be %s", fn, items[i].name, type_name(items[i].type));
            return false;
        }
    }
    for (int i = 0; i < n; ++i)
        if (!unpack(items[i].obj).is_cuda()) {
            value_error("%s: %s must be CUDA", fn, items[i].name);
            return false;
        }
    for (int i = 0; i < n; ++i)
        if (!unpack(items[i].obj).is_contiguous()) {
            value_error("%s: %s must be contiguous", fn, items[i].name);
            return false;
        }
    return true;
}

// the element type of a projection: BF16 or FP32
bool x_dtype(const char* fn, PyObject* x, ScalarType* type, int* code) {
    if (!THPVariable_Check(x)) {
        value_error("%s: x must be a tensor", fn);
        return false;
    }
    *type = unpack(x).scalar_type();
    if (*type != ScalarType::BFloat16 && *type != ScalarType::Float) {
        value_error("%s: x must be BF16 or FP32", fn);
        return false;
    }
    *code = *type == ScalarType::BFloat16 ? B200ATTN_DTYPE_BF16 : B200ATTN_DTYPE_F32;
    return true;
}

// n consecutive int arguments
bool ints(PyObject* const* args, int n, int* out) {
    for (int i = 0; i < n; ++i) {
        const long v = PyLong_AsLong(args[i]);
        if (v == -1 && PyErr_Occurred()) return false;
        if (v != static_cast<int>(v)) {
            PyErr_SetString(PyExc_OverflowError, "size does not fit 32 bits");
            return false;
        }
        out[i] = static_cast<int>(v);
    }
    return true;
}

// a layout name; -1 and no Python error when it is not one
int layout_of(PyObject* o) {
    if (!PyUnicode_Check(o)) return -1;
    if (PyUnicode_CompareWithASCIIString(o, "BHTD") == 0) return B200ATTN_LAYOUT_BHTD;
    if (PyUnicode_CompareWithASCIIString(o, "BTHD") == 0) return B200ATTN_LAYOUT_BTHD;
    return -1;
}

// a softmax scale or None (0: the default scale)
bool scale_of(PyObject* o, float* out) {
    *out = 0.f;
    if (o == Py_None) return true;
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) return false;
    *out = static_cast<float>(v);
    return true;
}

// ---- device, stream and scratch of a call
struct Call {
    c10::cuda::CUDAGuard guard;
    c10::cuda::CUDAStream stream;
    explicit Call(c10::Device d) : guard(d), stream(c10::cuda::getCurrentCUDAStream(d.index())) {}
    explicit Call(PyObject* t) : Call(unpack(t).device()) {}
    void* st() const { return stream.stream(); }
};

// The GIL is released for a scope (a full launch queue blocks in the driver) and taken again also when an exception leaves it.
struct NoGil {
    PyThreadState* state;
    NoGil() : state(PyEval_SaveThread()) {}
    NoGil(const NoGil&) = delete;
    ~NoGil() { PyEval_RestoreThread(state); }
};

// Private temporaries of the operators (the reference allocates its D vector per call, llm/src/model/flash_attn.cu:463):
// one buffer per (device, stream), so that calls issued on different streams never share scratch memory.  Calls on one
// stream follow each other on the GPU and may, provided that a call's launches follow each other without another call's in
// between (a backward is two launches with the row vectors alive between them): a call holds the buffer's lock from sizing
// it to its last launch, without the GIL.  A buffer grows when a call needs more and goes back to torch's
// allocator when it is replaced, when it is the least recently used of more than kMaxScratch (torch itself has 32
// streams per device and priority) and when the interpreter ends.  A captured launch keeps the address, so a buffer that one
// has used is not given back before the end; it then grows at least by doubling, so what is kept that way is less than the
// buffer itself.  The list is accessed under the GIL; a call keeps its entry alive.
struct Scratch {
    int device;
    cudaStream_t stream;
    std::mutex lock;  // of buf, and over the launches of the call that uses it
    at::Tensor buf;
    std::vector<at::Tensor> kept;        // outgrown buffers that captured launches may still use
    std::atomic<bool> captured{false};  // a capture has used buf: the entry stays
    Scratch(int d, cudaStream_t s) : device(d), stream(s) {}
};
constexpr size_t kMaxScratch = 128;
std::list<std::shared_ptr<Scratch>>& scratch_list() {
    static auto* l = new std::list<std::shared_ptr<Scratch>>;  // emptied by release_scratch at exit, never destroyed
    return *l;
}

std::shared_ptr<Scratch> scratch_entry(const Call& c) {
    std::list<std::shared_ptr<Scratch>>& l = scratch_list();
    const int dev = c.stream.device_index();
    auto it = l.begin();
    while (it != l.end() && !((*it)->device == dev && (*it)->stream == c.stream.stream())) ++it;
    if (it == l.end()) {
        l.push_front(std::make_shared<Scratch>(dev, c.stream.stream()));
        if (l.size() > kMaxScratch) {
            auto last = std::find_if(l.rbegin(), l.rend(), [](const auto& s) { return !s->captured; });
            if (last != l.rend()) l.erase(std::next(last).base());
        }
    } else if (it != l.begin()) {
        l.splice(l.begin(), l, it);
    }
    return l.front();
}

// Runs `launch(workspace, its bytes)` with the stream's scratch buffer, at least `bytes` of it.
template <typename Launch>
int with_scratch(const Call& c, size_t bytes, Launch launch) {
    const std::shared_ptr<Scratch> s = scratch_entry(c);
    const NoGil no_gil;
    const std::lock_guard<std::mutex> hold(s->lock);
    if (!s->buf.defined() || static_cast<size_t>(s->buf.numel()) < bytes) {
        if (s->captured && s->buf.defined()) {
            bytes = std::max(bytes, 2 * static_cast<size_t>(s->buf.numel()));
            s->kept.push_back(std::move(s->buf));
        }
        s->buf = at::Tensor();  // the smaller buffer first goes back to the allocator
        s->buf = at::empty({static_cast<int64_t>(std::max<size_t>(bytes, 4096))},
                           at::TensorOptions().dtype(at::kByte).device(at::kCUDA, static_cast<c10::DeviceIndex>(s->device)));
    }
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) s->captured = true;
    return launch(s->buf.data_ptr(), static_cast<size_t>(s->buf.numel()));
}

PyObject* release_scratch(PyObject*, PyObject*) {
    scratch_list().clear();
    Py_RETURN_NONE;
}

bool arg_count(Py_ssize_t got, Py_ssize_t want) {
    if (got == want) return true;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
    return false;
}

// C++ exceptions (torch's) become RuntimeError.
#define B200ATTN_TRY try {
#define B200ATTN_CATCH                                  \
    }                                                   \
    catch (const std::exception& e) {                   \
        PyErr_SetString(PyExc_RuntimeError, e.what());  \
        return nullptr;                                 \
    }

// ---- operators.  Arguments arrive positionally from the Python wrappers.

// q, k, v, ctx, L, B, T, Hq, Hkv, D, layout, softmax_scale
PyObject* fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const char* fn = "flash_attn_forward";
    B200ATTN_TRY
    if (!arg_count(n, 12)) return nullptr;
    const ScalarType bf = ScalarType::BFloat16;
    const Item items[] = {{a[0], "q", bf}, {a[1], "k", bf}, {a[2], "v", bf}, {a[3], "ctx", bf}, {a[4], "L", ScalarType::Float}};
    if (!check_tensors(fn, items, 5)) return nullptr;
    int d[5];
    if (!ints(a + 5, 5, d)) return nullptr;
    const int64_t B = d[0], T = d[1], Hq = d[2], Hkv = d[3], D = d[4];
    const int layout = layout_of(a[10]);
    if (layout < 0) return value_error("%s: layout must be BHTD or BTHD", fn);
    const int64_t nq = B * Hq * T * D, nkv = B * Hkv * T * D;
    if (numel(a[0]) != nq || numel(a[3]) != nq || numel(a[1]) != nkv || numel(a[2]) != nkv)
        return value_error("%s: shape mismatch (qkv/ctx)", fn);
    if (numel(a[4]) != B * Hq * T) return value_error("%s: L must be [B, T]", fn);
    float scale;
    if (!scale_of(a[11], &scale)) return nullptr;
    const Call c(a[0]);
    void *q = ptr(a[0]), *k = ptr(a[1]), *v = ptr(a[2]), *o = ptr(a[3]), *lse = ptr(a[4]), *st = c.st();
    int rc;
    {
        const NoGil no_gil;
        rc = b200attn_fwd(q, k, v, o, static_cast<float*>(lse), d[0], d[1], d[2], d[3], d[4], layout, scale, st);
    }
    return finish(rc, fn);
    B200ATTN_CATCH
}

// q, k, v, ctx, L, d_ctx, d_q, d_k, d_v, B, T, Hq, Hkv, D, layout, softmax_scale, mode
PyObject* bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const char* fn = "flash_attn_backward";
    B200ATTN_TRY
    if (!arg_count(n, 17)) return nullptr;
    const ScalarType bf = ScalarType::BFloat16;
    const Item items[] = {{a[0], "q", bf}, {a[1], "k", bf}, {a[2], "v", bf}, {a[3], "ctx", bf}, {a[4], "L", ScalarType::Float},
                                   {a[5], "d_ctx", bf}, {a[6], "d_q", bf}, {a[7], "d_k", bf}, {a[8], "d_v", bf}};
    if (!check_tensors(fn, items, 9)) return nullptr;
    int d[5];
    if (!ints(a + 9, 5, d)) return nullptr;
    const int64_t B = d[0], T = d[1], Hq = d[2], Hkv = d[3], D = d[4];
    const int layout = layout_of(a[14]);
    if (layout < 0) return value_error("%s: layout must be BHTD or BTHD", fn);
    const int64_t nq = B * Hq * T * D, nkv = B * Hkv * T * D;
    if (numel(a[0]) != nq || numel(a[3]) != nq || numel(a[5]) != nq || numel(a[6]) != nq || numel(a[1]) != nkv ||
        numel(a[2]) != nkv || numel(a[7]) != nkv || numel(a[8]) != nkv)
        return value_error("%s: shape mismatch", fn);
    if (numel(a[4]) != B * Hq * T) return value_error("%s: L must be [B, T]", fn);
    int mode = -1;
    if (PyUnicode_Check(a[16])) {
        if (PyUnicode_CompareWithASCIIString(a[16], "auto") == 0) mode = B200ATTN_BWD_AUTO;
        else if (PyUnicode_CompareWithASCIIString(a[16], "two_pass") == 0) mode = B200ATTN_BWD_TWO_PASS;
        else if (PyUnicode_CompareWithASCIIString(a[16], "one_pass") == 0) mode = B200ATTN_BWD_ONE_PASS;
    }
    if (mode < 0) return value_error("%s: mode must be auto, two_pass or one_pass", fn);
    float scale;
    if (!scale_of(a[15], &scale)) return nullptr;
    const Call c(a[0]);
    void *q = ptr(a[0]), *k = ptr(a[1]), *v = ptr(a[2]), *o = ptr(a[3]), *lse = ptr(a[4]), *dout = ptr(a[5]), *dq = ptr(a[6]),
         *dk = ptr(a[7]), *dv = ptr(a[8]), *st = c.st();
    const int rc = with_scratch(c, b200attn_bwd_workspace_bytes_mode(d[0], d[1], d[2], d[3], d[4], mode), [&](void* wp, size_t wn) {
        return b200attn_bwd_mode(q, k, v, o, static_cast<float*>(lse), dout, dq, dk, dv, d[0], d[1], d[2], d[3], d[4], layout, scale,
                                 mode, wp, wn, st);
    });
    return finish(rc, fn);
    B200ATTN_CATCH
}

// q, kcache, vcache, o, lse or None, B, L, Hq, Hkv, D, softmax_scale, n_splits
PyObject* decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const char* fn = "flash_attn_decode";
    B200ATTN_TRY
    if (!arg_count(n, 12)) return nullptr;
    const ScalarType bf = ScalarType::BFloat16;
    const bool with_lse = a[4] != Py_None;
    const Item items[] = {{a[0], "q", bf}, {a[1], "kcache", bf}, {a[2], "vcache", bf}, {a[3], "o", bf}, {a[4], "lse", ScalarType::Float}};
    if (!check_tensors(fn, items, with_lse ? 5 : 4)) return nullptr;
    int d[5], splits;
    if (!ints(a + 5, 5, d) || !ints(a + 11, 1, &splits)) return nullptr;
    const int64_t B = d[0], L = d[1], Hq = d[2], Hkv = d[3], D = d[4];
    if (with_lse && numel(a[4]) != B * Hq) return value_error("%s: lse must be [B, Hq]", fn);
    if (numel(a[0]) != B * Hq * D || numel(a[3]) != B * Hq * D) return value_error("%s: shape mismatch (q/o)", fn);
    if (numel(a[1]) != B * Hkv * L * D || numel(a[2]) != B * Hkv * L * D) return value_error("%s: shape mismatch (cache)", fn);
    float scale;
    if (!scale_of(a[10], &scale)) return nullptr;
    const Call c(a[0]);
    void *q = ptr(a[0]), *k = ptr(a[1]), *v = ptr(a[2]), *o = ptr(a[3]), *lse = with_lse ? ptr(a[4]) : nullptr, *st = c.st();
    const int rc = with_scratch(c, b200attn_decode_workspace_bytes(d[0], d[1], d[2], d[3], d[4], splits), [&](void* wp, size_t wn) {
        return b200attn_decode(q, k, v, o, static_cast<float*>(lse), d[0], d[1], d[2], d[3], d[4], scale, splits, wp, wn, st);
    });
    return finish(rc, fn);
    B200ATTN_CATCH
}

// ---- KVCache (kv_cache.py): the object itself is the first argument; its sizes are read in front of the checks, its
// buffers behind them
struct Ref {  // an owned reference
    PyObject* o;
    explicit Ref(PyObject* p) : o(p) {}
    Ref(const Ref&) = delete;
    ~Ref() { Py_XDECREF(o); }
};
PyObject* intern(const char* name) { return PyUnicode_InternFromString(name); }

struct CacheSizes {
    int B, Hq, Hkv, D, L_cap, n_layers, length;
};
bool cache_sizes(PyObject* self, CacheSizes* c) {
    static PyObject* const names[7] = {intern("B"), intern("Hq"), intern("Hkv"), intern("D"), intern("L_cap"), intern("n_layers"), intern("length")};
    int* const out[7] = {&c->B, &c->Hq, &c->Hkv, &c->D, &c->L_cap, &c->n_layers, &c->length};
    for (int i = 0; i < 7; ++i) {
        const Ref r(PyObject_GetAttr(self, names[i]));
        if (!r.o || !ints(&r.o, 1, out[i])) return false;
    }
    return true;
}
bool layer_ok(const char* fn, const CacheSizes& c, int layer) {
    if (layer >= 0 && layer < c.n_layers) return true;
    value_error("%s: layer %d out of range", fn, layer);
    return false;
}
// a tensor attribute of the cache; the attribute keeps it alive while the call is being issued
bool cache_tensor(PyObject* self, PyObject* name, at::Tensor* t) {
    const Ref r(PyObject_GetAttr(self, name));
    if (!r.o) return false;
    if (!THPVariable_Check(r.o)) {
        PyErr_Format(PyExc_ValueError, "KVCache: %U must be a tensor", name);
        return false;
    }
    *t = unpack(r.o);
    return true;
}
struct CacheLayer {
    at::Tensor kt, vt;
    char *k, *v;
};
bool cache_layer(PyObject* self, const CacheSizes& c, int layer, CacheLayer* l) {
    static PyObject* const names[2] = {intern("k"), intern("v")};
    if (!cache_tensor(self, names[0], &l->kt) || !cache_tensor(self, names[1], &l->vt)) return false;
    const size_t off = size_t(layer) * c.B * c.Hkv * c.L_cap * c.D * 2;
    l->k = static_cast<char*>(l->kt.data_ptr()) + off;
    l->v = static_cast<char*>(l->vt.data_ptr()) + off;
    return true;
}

// cache, layer, xq, xk, xv, gamma_q, gamma_k, q_out
PyObject* kv_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const char* fn = "KVCache.append";
    static PyObject* const n_lengths = intern("lengths"), * const n_cos = intern("cos"), * const n_sin = intern("sin"), * const n_eps = intern("eps");
    B200ATTN_TRY
    if (!arg_count(n, 8)) return nullptr;
    PyObject *self = a[0], *xq = a[2], *xk = a[3], *xv = a[4], *gq = a[5], *gk = a[6], *q_out = a[7];
    int layer, xd;
    CacheSizes c;
    if (!cache_sizes(self, &c) || !ints(a + 1, 1, &layer) || !layer_ok(fn, c, layer)) return nullptr;
    ScalarType xt;
    if (!x_dtype(fn, xq, &xt, &xd)) return nullptr;
    const Item items[] = {{xq, "xq", xt}, {xk, "xk", xt}, {xv, "xv", xt}, {q_out, "q_out", ScalarType::BFloat16},
                          {gq, "gamma_q", ScalarType::Float}, {gk, "gamma_k", ScalarType::Float}};
    if (!check_tensors(fn, items, 6)) return nullptr;
    const at::Tensor& tq = unpack(xq);
    if (tq.dim() != 4 || tq.size(0) != c.B || tq.size(2) != c.Hq || tq.size(3) != c.D)
        return value_error("%s: xq must be [B, n_new, Hq, D]", fn);
    const int64_t n_new = tq.size(1);
    if (n_new <= 0) return value_error("%s: no tokens", fn);
    for (PyObject* x : {xk, xv}) {
        const at::Tensor& t = unpack(x);
        if (t.dim() != 4 || t.size(0) != c.B || t.size(1) != n_new || t.size(2) != c.Hkv || t.size(3) != c.D)
            return value_error("%s: xk and xv must be [B, n_new, Hkv, D]", fn);
    }
    if (numel(q_out) != tq.numel()) return value_error("%s: q_out numel mismatch", fn);
    if (numel(gq) != c.D || numel(gk) != c.D) return value_error("%s: gamma_q and gamma_k must have d_h elements", fn);
    if (c.length + n_new > c.L_cap)
        return value_error("%s: %d + %d tokens exceed the capacity %d", fn, c.length, int(n_new), c.L_cap);
    const Ref lengths(PyObject_GetAttr(self, n_lengths)), eps_o(PyObject_GetAttr(self, n_eps));
    if (!lengths.o || !eps_o.o) return nullptr;
    const bool ragged = lengths.o != Py_None;
    if (ragged && n_new != 1) return value_error("%s: one token per sequence once the lengths differ", fn);
    const double eps = PyFloat_AsDouble(eps_o.o);
    if (eps == -1.0 && PyErr_Occurred()) return nullptr;
    CacheLayer l;
    at::Tensor cos_t, sin_t, pos_t;
    if (!cache_layer(self, c, layer, &l) || !cache_tensor(self, n_cos, &cos_t) || !cache_tensor(self, n_sin, &sin_t) ||
        (ragged && !cache_tensor(self, n_lengths, &pos_t)))
        return nullptr;
    const Call call(l.kt.device());
    const float *gqp = static_cast<float*>(ptr(gq)), *gkp = static_cast<float*>(ptr(gk)),
                *cp = static_cast<float*>(cos_t.data_ptr()), *sp = static_cast<float*>(sin_t.data_ptr());
    const int* pos = ragged ? static_cast<int*>(pos_t.data_ptr()) : nullptr;
    void *pq = ptr(xq), *pk = ptr(xk), *pv = ptr(xv), *po = ptr(q_out), *st = call.st();
    int rc;
    {
        const NoGil no_gil;
        rc = ragged ? b200attn_kv_append_at(pq, pk, pv, xd, po, l.k, l.v, gqp, gkp, cp, sp, pos, c.B, 1, c.L_cap, c.Hq, c.Hkv, c.D,
                                            static_cast<float>(eps), st)
                    : b200attn_kv_append(pq, pk, pv, xd, po, l.k, l.v, gqp, gkp, cp, sp, c.B, int(n_new), c.length, c.L_cap, c.Hq,
                                         c.Hkv, c.D, static_cast<float>(eps), st);
    }
    return finish(rc, fn);
    B200ATTN_CATCH
}

// cache, layer, q, ctx, lse or None, n_new, softmax_scale
PyObject* kv_attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const char* fn = "KVCache.attend";
    static PyObject* const n_lens_next = intern("_lens_next");
    B200ATTN_TRY
    if (!arg_count(n, 7)) return nullptr;
    PyObject *self = a[0], *q = a[2], *ctx = a[3], *lse = a[4];
    int layer, n_new;
    CacheSizes c;
    if (!cache_sizes(self, &c) || !ints(a + 1, 1, &layer) || !ints(a + 5, 1, &n_new) || !layer_ok(fn, c, layer)) return nullptr;
    const bool with_lse = lse != Py_None;
    const ScalarType bf = ScalarType::BFloat16;
    const Item items[] = {{q, "q", bf}, {ctx, "ctx", bf}, {lse, "lse", ScalarType::Float}};
    if (!check_tensors(fn, items, with_lse ? 3 : 2)) return nullptr;
    if (n_new <= 0 || int64_t(c.length) + n_new > c.L_cap) return value_error("%s: n_new out of range", fn);
    const int64_t rows = int64_t(c.B) * c.Hq * n_new;
    if (numel(q) != rows * c.D || numel(ctx) != rows * c.D) return value_error("%s: q and ctx must be [B, Hq, n_new, D]", fn);
    if (with_lse && numel(lse) != rows) return value_error("%s: lse must be [B, Hq, n_new]", fn);
    const Ref lens_o(PyObject_GetAttr(self, n_lens_next));
    if (!lens_o.o) return nullptr;
    const bool ragged = lens_o.o != Py_None;
    if (n_new > 1 && ragged) return value_error("%s: several tokens at once only while the sequences advance in lock step", fn);
    if (n_new > 1 && !with_lse) return value_error("%s: lse is required for n_new > 1", fn);
    float scale;
    if (!scale_of(a[6], &scale)) return nullptr;
    CacheLayer l;
    at::Tensor lens_t;
    if (!cache_layer(self, c, layer, &l) || (ragged && !cache_tensor(self, n_lens_next, &lens_t))) return nullptr;
    const Call call(l.kt.device());
    void *pq = ptr(q), *po = ptr(ctx), *st = call.st();
    float* pl = with_lse ? static_cast<float*>(ptr(lse)) : nullptr;
    const int* lens = ragged ? static_cast<int*>(lens_t.data_ptr()) : nullptr;
    int rc;
    if (n_new == 1) {
        rc = with_scratch(call, b200attn_decode_workspace_bytes(c.B, c.length + 1, c.Hq, c.Hkv, c.D, 0), [&](void* wp, size_t wn) {
            return b200attn_decode_ragged(pq, l.k, l.v, po, pl, lens, c.B, c.length + 1, c.L_cap, c.Hq, c.Hkv, c.D, scale, 0, wp, wn, st);
        });
    } else {
        const NoGil no_gil;
        rc = b200attn_fwd_kvcache_at(pq, l.k, l.v, po, pl, c.B, n_new, c.length, c.L_cap, c.Hq, c.Hkv, c.D, B200ATTN_LAYOUT_BHTD, scale, st);
    }
    return finish(rc, fn);
    B200ATTN_CATCH
}

// What q and k share in the RoPE + QK-Norm calls: tables [>= T, D / 2], layouts, sizes
struct NormArgs {
    float *cos_t, *sin_t;
    int x_layout, y_layout, B, T, D;
};
bool norm_args(const char* fn, PyObject* x_layout, PyObject* y_layout, int B, int T, int D, NormArgs* p) {
    p->x_layout = layout_of(x_layout);
    p->y_layout = layout_of(y_layout);
    if (p->x_layout < 0 || p->y_layout < 0) {
        value_error("%s: %s must be BHTD or BTHD", fn, p->x_layout < 0 ? "x_layout" : "y_layout");
        return false;
    }
    if (D % 2 != 0) {
        value_error("%s: d_h must be even", fn);
        return false;
    }
    p->B = B, p->T = T, p->D = D;
    return true;
}
bool norm_tables(const char* fn, PyObject* cos_t, PyObject* sin_t, NormArgs* p) {
    const at::Tensor &c = unpack(cos_t), &s = unpack(sin_t);
    const int64_t need = int64_t(p->T) * (p->D / 2);
    if (c.numel() < need || s.numel() < need || c.dim() == 0 || c.size(-1) != p->D / 2) {
        value_error("%s: cos/sin tables must be [>= T, d_h / 2]", fn);
        return false;
    }
    p->cos_t = static_cast<float*>(c.data_ptr());
    p->sin_t = static_cast<float*>(s.data_ptr());
    return true;
}

// x, cos, sin, gamma, eps, y, rstd, B, T, H, D, x_layout, y_layout
PyObject* rope_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const char* fn = "rope_qknorm_forward";
    B200ATTN_TRY
    if (!arg_count(n, 13)) return nullptr;
    ScalarType xt;
    int xd, d[4];
    if (!x_dtype(fn, a[0], &xt, &xd)) return nullptr;
    const ScalarType f = ScalarType::Float;
    const Item items[] = {{a[0], "x", xt}, {a[5], "y", ScalarType::BFloat16}, {a[1], "cos", f}, {a[2], "sin", f}, {a[3], "gamma", f}, {a[6], "rstd", f}};
    if (!check_tensors(fn, items, 6) || !ints(a + 7, 4, d)) return nullptr;
    const int64_t rows = int64_t(d[0]) * d[1] * d[2];
    NormArgs p;
    if (!norm_args(fn, a[11], a[12], d[0], d[1], d[3], &p)) return nullptr;
    if (numel(a[0]) != rows * p.D) return value_error("%s: x numel mismatch", fn);
    if (!norm_tables(fn, a[1], a[2], &p)) return nullptr;
    if (numel(a[3]) != p.D) return value_error("%s: gamma must have d_h elements", fn);
    if (numel(a[6]) != rows) return value_error("%s: rstd must have B * H * T elements", fn);
    if (numel(a[5]) != rows * p.D) return value_error("%s: y numel mismatch", fn);
    const double eps = PyFloat_AsDouble(a[4]);
    if (eps == -1.0 && PyErr_Occurred()) return nullptr;
    const Call c(a[0]);
    void *x = ptr(a[0]), *y = ptr(a[5]), *st = c.st();
    float *gamma = static_cast<float*>(ptr(a[3])), *rstd = static_cast<float*>(ptr(a[6]));
    int rc;
    {
        const NoGil no_gil;
        rc = b200attn_rope_norm_fwd(x, xd, p.x_layout, y, p.y_layout, rstd, gamma, p.cos_t, p.sin_t, d[0], d[1], d[2], d[3],
                                    static_cast<float>(eps), st);
    }
    return finish(rc, fn);
    B200ATTN_CATCH
}

// d_y, x, cos, sin, gamma, rstd, d_x, d_gamma, B, T, H, D, x_layout, y_layout
PyObject* rope_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const char* fn = "rope_qknorm_backward";
    B200ATTN_TRY
    if (!arg_count(n, 14)) return nullptr;
    ScalarType xt;
    int xd, d[4];
    if (!x_dtype(fn, a[1], &xt, &xd)) return nullptr;
    const ScalarType f = ScalarType::Float;
    const Item items[] = {{a[0], "d_y", ScalarType::BFloat16}, {a[1], "x", xt}, {a[6], "d_x", xt}, {a[7], "d_gamma", f},
                                   {a[2], "cos", f}, {a[3], "sin", f}, {a[4], "gamma", f}, {a[5], "rstd", f}};
    if (!check_tensors(fn, items, 8) || !ints(a + 8, 4, d)) return nullptr;
    const int64_t rows = int64_t(d[0]) * d[1] * d[2];
    NormArgs p;
    if (!norm_args(fn, a[12], a[13], d[0], d[1], d[3], &p)) return nullptr;
    if (numel(a[1]) != rows * p.D) return value_error("%s: x numel mismatch", fn);
    if (!norm_tables(fn, a[2], a[3], &p)) return nullptr;
    if (numel(a[4]) != p.D) return value_error("%s: gamma must have d_h elements", fn);
    if (numel(a[5]) != rows) return value_error("%s: rstd must have B * H * T elements", fn);
    if (numel(a[0]) != rows * p.D || numel(a[6]) != rows * p.D || numel(a[7]) != p.D)
        return value_error("%s: shape mismatch (d_y/d_x/d_gamma)", fn);
    const Call c(a[1]);
    void *dy = ptr(a[0]), *x = ptr(a[1]), *dx = ptr(a[6]), *st = c.st();
    float *gamma = static_cast<float*>(ptr(a[4])), *rstd = static_cast<float*>(ptr(a[5])), *dg = static_cast<float*>(ptr(a[7]));
    const int rc = with_scratch(c, b200attn_rope_norm_bwd_workspace_bytes(p.D), [&](void* wp, size_t wn) {
        return b200attn_rope_norm_bwd(dy, p.y_layout, x, xd, p.x_layout, rstd, gamma, p.cos_t, p.sin_t, dx, dg, d[0], d[1], d[2], d[3], wp,
                                      wn, st);
    });
    return finish(rc, fn);
    B200ATTN_CATCH
}

// xq, xk, cos, sin, gamma_q, gamma_k, eps, yq, yk, rstd_q, rstd_k, B, T, Hq, Hkv, D, x_layout, y_layout
PyObject* rope_fwd_qk(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const char* fn = "rope_qknorm_forward";
    B200ATTN_TRY
    if (!arg_count(n, 18)) return nullptr;
    ScalarType xt;
    int xd, d[5];
    if (!x_dtype(fn, a[0], &xt, &xd)) return nullptr;
    if (!THPVariable_Check(a[1]) || unpack(a[1]).scalar_type() != xt) return value_error("%s: xq and xk must have the same dtype", fn);
    const ScalarType f = ScalarType::Float, bf = ScalarType::BFloat16;
    const Item items[] = {{a[0], "xq", xt}, {a[1], "xk", xt}, {a[7], "yq", bf}, {a[8], "yk", bf}, {a[5], "gamma_k", f},
                                   {a[10], "rstd_k", f}, {a[2], "cos", f}, {a[3], "sin", f}, {a[4], "gamma", f}, {a[9], "rstd", f}};
    if (!check_tensors(fn, items, 10) || !ints(a + 11, 5, d)) return nullptr;
    const int64_t rq = int64_t(d[0]) * d[1] * d[2], rk = int64_t(d[0]) * d[1] * d[3];
    NormArgs p;
    if (!norm_args(fn, a[16], a[17], d[0], d[1], d[4], &p)) return nullptr;
    if (numel(a[0]) != rq * p.D) return value_error("%s: x numel mismatch", fn);
    if (!norm_tables(fn, a[2], a[3], &p)) return nullptr;
    if (numel(a[4]) != p.D) return value_error("%s: gamma must have d_h elements", fn);
    if (numel(a[9]) != rq) return value_error("%s: rstd must have B * H * T elements", fn);
    if (numel(a[1]) != rk * p.D || numel(a[7]) != rq * p.D || numel(a[8]) != rk * p.D)
        return value_error("%s: shape mismatch (xk/yq/yk)", fn);
    if (numel(a[5]) != p.D || numel(a[10]) != rk) return value_error("%s: shape mismatch (gamma_k/rstd_k)", fn);
    const double eps = PyFloat_AsDouble(a[6]);
    if (eps == -1.0 && PyErr_Occurred()) return nullptr;
    const Call c(a[0]);
    void *xq = ptr(a[0]), *xk = ptr(a[1]), *yq = ptr(a[7]), *yk = ptr(a[8]), *st = c.st();
    float *gq = static_cast<float*>(ptr(a[4])), *gk = static_cast<float*>(ptr(a[5])), *sq = static_cast<float*>(ptr(a[9])),
          *sk = static_cast<float*>(ptr(a[10]));
    int rc;
    {
        const NoGil no_gil;
        rc = b200attn_rope_norm_fwd_qk(xq, xk, xd, p.x_layout, yq, yk, p.y_layout, sq, sk, gq, gk, p.cos_t, p.sin_t, d[0], d[1], d[2],
                                       d[3], d[4], static_cast<float>(eps), st);
    }
    return finish(rc, fn);
    B200ATTN_CATCH
}

// d_yq, d_yk, xq, xk, cos, sin, gamma_q, gamma_k, rstd_q, rstd_k, d_xq, d_xk, d_gamma_q, d_gamma_k, B, T, Hq, Hkv, D, x_layout, y_layout
PyObject* rope_bwd_qk(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const char* fn = "rope_qknorm_backward";
    B200ATTN_TRY
    if (!arg_count(n, 21)) return nullptr;
    ScalarType xt;
    int xd, d[5];
    if (!x_dtype(fn, a[2], &xt, &xd)) return nullptr;
    if (!THPVariable_Check(a[3]) || unpack(a[3]).scalar_type() != xt) return value_error("%s: xq and xk must have the same dtype", fn);
    const ScalarType f = ScalarType::Float, bf = ScalarType::BFloat16;
    const Item items[] = {{a[0], "d_yq", bf}, {a[1], "d_yk", bf}, {a[2], "xq", xt}, {a[3], "xk", xt}, {a[10], "d_xq", xt},
                                   {a[11], "d_xk", xt}, {a[12], "d_gamma_q", f}, {a[13], "d_gamma_k", f}, {a[7], "gamma_k", f},
                                   {a[9], "rstd_k", f}, {a[4], "cos", f}, {a[5], "sin", f}, {a[6], "gamma", f}, {a[8], "rstd", f}};
    if (!check_tensors(fn, items, 14) || !ints(a + 14, 5, d)) return nullptr;
    const int64_t rq = int64_t(d[0]) * d[1] * d[2], rk = int64_t(d[0]) * d[1] * d[3];
    NormArgs p;
    if (!norm_args(fn, a[19], a[20], d[0], d[1], d[4], &p)) return nullptr;
    if (numel(a[2]) != rq * p.D) return value_error("%s: x numel mismatch", fn);
    if (!norm_tables(fn, a[4], a[5], &p)) return nullptr;
    if (numel(a[6]) != p.D) return value_error("%s: gamma must have d_h elements", fn);
    if (numel(a[8]) != rq) return value_error("%s: rstd must have B * H * T elements", fn);
    if (numel(a[3]) != rk * p.D || numel(a[0]) != rq * p.D || numel(a[1]) != rk * p.D || numel(a[10]) != rq * p.D ||
        numel(a[11]) != rk * p.D)
        return value_error("%s: shape mismatch (xk/d_y/d_x)", fn);
    if (numel(a[7]) != p.D || numel(a[9]) != rk || numel(a[12]) != p.D || numel(a[13]) != p.D)
        return value_error("%s: shape mismatch (gamma_k/rstd_k/d_gamma)", fn);
    const Call c(a[2]);
    void *dyq = ptr(a[0]), *dyk = ptr(a[1]), *xq = ptr(a[2]), *xk = ptr(a[3]), *dxq = ptr(a[10]), *dxk = ptr(a[11]), *st = c.st();
    float *gq = static_cast<float*>(ptr(a[6])), *gk = static_cast<float*>(ptr(a[7])), *sq = static_cast<float*>(ptr(a[8])),
          *sk = static_cast<float*>(ptr(a[9])), *dgq = static_cast<float*>(ptr(a[12])), *dgk = static_cast<float*>(ptr(a[13]));
    const int rc = with_scratch(c, b200attn_rope_norm_bwd_workspace_bytes(p.D), [&](void* wp, size_t wn) {
        return b200attn_rope_norm_bwd_qk(dyq, dyk, p.y_layout, xq, xk, xd, p.x_layout, sq, sk, gq, gk, p.cos_t, p.sin_t, dxq, dxk, dgq,
                                         dgk, d[0], d[1], d[2], d[3], d[4], wp, wn, st);
    });
    return finish(rc, fn);
    B200ATTN_CATCH
}

#define B200ATTN_FAST(name) \
    { #name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr }
PyMethodDef methods[] = {
    B200ATTN_FAST(fwd),      B200ATTN_FAST(bwd),      B200ATTN_FAST(decode),      B200ATTN_FAST(kv_append),
    B200ATTN_FAST(kv_attend), B200ATTN_FAST(rope_fwd), B200ATTN_FAST(rope_bwd),    B200ATTN_FAST(rope_fwd_qk),
    B200ATTN_FAST(rope_bwd_qk), {"release_scratch", release_scratch, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
