// Python's way to the op launches: the checks and the marshalling of `inferi_b200/ops.py`, for the calls that pass them.
//
// A launch through ctypes is 4 us of host time, twice what the launch itself takes, and most small ops run for 3 us: a host
// that composes a model from them was bound by its own thread (two layers of the 1B architecture, 31 launches: 142 us where the GPU needs 87).
// Every function here returns the library's status, or -1 where it has not launched anything because an argument is not what the fast
// way takes (no plain tensor, another type, wrong lengths, a closed handle): the caller then goes through the checked Python path, which
// raises the error or does the call.
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/inferi_b200.h"

namespace {

struct Entry {
    decltype(&ib_gemv_quant) gemv;
    decltype(&ib_gemm_quant) gemm;
    decltype(&ib_rms_norm) rms_norm;
    decltype(&ib_rope) rope;
    decltype(&ib_silu_mul) silu;
    decltype(&ib_add_assign) add;
    decltype(&ib_attention) attention;
    decltype(&ib_argmax) argmax;
    decltype(&ib_sample) sample;
} lib;
constexpr Py_ssize_t ENTRIES = sizeof(Entry) / sizeof(void *);

constexpr long NOT_TAKEN = -1;

// A plain tensor on a GPU in one piece (subclasses have a say in what their attributes are: the Python path asks them)
const at::Tensor *dense(PyObject *o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    return t.is_cuda() && t.is_contiguous() ? &t : nullptr;
}
const at::Tensor *dense_f32(PyObject *o) {
    const at::Tensor *t = dense(o);
    return t && t->scalar_type() == at::kFloat ? t : nullptr;
}
float *at_f32(const at::Tensor *t) { return static_cast<float *>(t->data_ptr()); }
template <class T>
T *handle(PyObject *o) { return static_cast<T *>(PyLong_AsVoidPtr(o)); }
float f32(PyObject *o) {   // a Python number (others, numpy's among them, are not what ctypes takes for a float)
    if (PyFloat_Check(o) || PyLong_Check(o)) return static_cast<float>(PyFloat_AsDouble(o));
    PyErr_SetString(PyExc_TypeError, "not a number");
    return 0.f;
}
uint32_t u32(PyObject *o) {
    const unsigned long v = PyLong_AsUnsignedLong(o);
    if (v > 0xFFFFFFFFul && !PyErr_Occurred()) PyErr_SetString(PyExc_OverflowError, "not 32 bits");
    return static_cast<uint32_t>(v);
}

// The call on the current device's current stream, without the interpreter's lock (a launch waits where the stream's queue is full)
template <class F>
long on_stream(F &&f) {
    void *s = c10::cuda::getCurrentCUDAStream().stream();
    long rc;
    Py_BEGIN_ALLOW_THREADS rc = f(s);
    Py_END_ALLOW_THREADS return rc;
}

// What an argument of another kind raises on the way is the Python path's to say
template <long (*F)(PyObject *const *), Py_ssize_t N>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    long rc = NOT_TAKEN;
    if (n == N) {
        try {
            rc = F(args);
        } catch (...) {
            rc = NOT_TAKEN;
        }
        if (PyErr_Occurred()) PyErr_Clear();
    }
    return PyLong_FromLong(rc);
}

long gemv(PyObject *const *a) {   // ctx, out, m, rows, cols, v
    ib_ctx *ctx = handle<ib_ctx>(a[0]);
    const ib_qtensor *m = handle<ib_qtensor>(a[2]);
    const at::Tensor *out = dense_f32(a[1]), *v = dense_f32(a[5]);
    if (!ctx || !m || !out || !v || out->numel() != PyLong_AsLongLong(a[3]) || v->numel() != PyLong_AsLongLong(a[4])) return NOT_TAKEN;
    float *po = at_f32(out), *pv = at_f32(v);
    return on_stream([&](void *s) { return lib.gemv(ctx, s, po, m, pv); });
}

long gemm(PyObject *const *a) {   // ctx, out, m, rows, cols, x
    ib_ctx *ctx = handle<ib_ctx>(a[0]);
    const ib_qtensor *m = handle<ib_qtensor>(a[2]);
    const at::Tensor *out = dense_f32(a[1]), *x = dense_f32(a[5]);
    if (!ctx || !m || !out || !x || x->dim() != 2 || out->dim() != 2) return NOT_TAKEN;
    const int64_t n = x->size(0);
    if (n > 0xFFFFFFFFll || out->size(0) != n || out->size(1) != PyLong_AsLongLong(a[3]) || x->size(1) != PyLong_AsLongLong(a[4])) return NOT_TAKEN;
    float *po = at_f32(out), *px = at_f32(x);
    return on_stream([&](void *s) { return lib.gemm(ctx, s, po, m, px, static_cast<uint32_t>(n)); });
}

long rms_norm(PyObject *const *a) {   // ctx, result, value, weight, eps
    ib_ctx *ctx = handle<ib_ctx>(a[0]);
    const at::Tensor *r = dense_f32(a[1]), *v = dense_f32(a[2]), *w = dense_f32(a[3]);
    const float eps = f32(a[4]);
    if (!ctx || !r || !v || !w || r->numel() != v->numel() || w->numel() != v->numel() || v->numel() > 0xFFFFFFFFll || PyErr_Occurred()) return NOT_TAKEN;
    float *pr = at_f32(r), *pv = at_f32(v), *pw = at_f32(w);
    const uint32_t n = static_cast<uint32_t>(v->numel());
    return on_stream([&](void *s) { return lib.rms_norm(ctx, s, pr, pv, pw, n, eps); });
}

long rope(PyObject *const *a) {   // ctx, variant, q, k, kv_dim, head_size, pos, base_freq
    ib_ctx *ctx = handle<ib_ctx>(a[0]);
    const at::Tensor *q = dense_f32(a[2]), *k = dense_f32(a[3]);
    if (!ctx || !q || !k) return NOT_TAKEN;
    const long variant = PyLong_AsLong(a[1]);
    const uint32_t kv_dim = u32(a[4]), head_size = u32(a[5]), pos = u32(a[6]);
    const float base = f32(a[7]);
    if (variant < 0 || variant > 0x7FFFFFFF || k->numel() < kv_dim || q->numel() > 0xFFFFFFFFll || PyErr_Occurred()) return NOT_TAKEN;
    float *pq = at_f32(q), *pk = at_f32(k);
    const uint32_t q_len = static_cast<uint32_t>(q->numel());
    return on_stream([&](void *s) { return lib.rope(ctx, s, static_cast<int32_t>(variant), pq, q_len, pk, kv_dim, head_size, pos, base); });
}

template <decltype(lib.silu) Entry::*F>
long pairwise(PyObject *const *a) {   // ctx, in/out, in
    ib_ctx *ctx = handle<ib_ctx>(a[0]);
    const at::Tensor *x = dense_f32(a[1]), *y = dense_f32(a[2]);
    if (!ctx || !x || !y || x->numel() != y->numel() || x->numel() > 0xFFFFFFFFll) return NOT_TAKEN;
    float *px = at_f32(x), *py = at_f32(y);
    const uint32_t n = static_cast<uint32_t>(x->numel());
    return on_stream([&](void *s) { return (lib.*F)(ctx, s, px, py, n); });
}

long attention(PyObject *const *a) {   // ctx, params, q, key cache, value cache, out
    ib_ctx *ctx = handle<ib_ctx>(a[0]);
    const at::Tensor *q = dense_f32(a[2]), *k = dense(a[3]), *v = dense(a[4]), *out = dense_f32(a[5]);
    if (!ctx || !q || !k || !v || !out || k->scalar_type() != v->scalar_type()) return NOT_TAKEN;
    const bool f16 = k->scalar_type() == at::kHalf;
    if (!f16 && k->scalar_type() != at::kFloat) return NOT_TAKEN;
    Py_buffer view;
    if (PyObject_GetBuffer(a[1], &view, PyBUF_SIMPLE)) return NOT_TAKEN;
    ib_attn_params p;
    const bool whole = view.len == static_cast<Py_ssize_t>(sizeof p);
    if (whole) memcpy(&p, view.buf, sizeof p);
    PyBuffer_Release(&view);
    if (!whole) return NOT_TAKEN;
    const int64_t need = static_cast<int64_t>(static_cast<uint64_t>(p.seq_len) * p.kv_dim), n = static_cast<int64_t>(static_cast<uint64_t>(p.n_heads) * p.head_size);
    if (need < 0 || k->numel() < need || v->numel() < need || n < 0 || q->numel() != n || out->numel() != n) return NOT_TAKEN;
    float *pq = at_f32(q), *po = at_f32(out);
    void *pk = k->data_ptr(), *pv = v->data_ptr();
    return on_stream([&](void *s) { return lib.attention(ctx, s, &p, pq, pk, pv, f16 ? IB_KV_F16 : IB_KV_F32, po); });
}

long argmax(PyObject *const *a) {   // ctx, logits, out
    ib_ctx *ctx = handle<ib_ctx>(a[0]);
    const at::Tensor *x = dense_f32(a[1]);
    if (!ctx || !x || x->numel() > 0xFFFFFFFFll || !THPVariable_CheckExact(a[2])) return NOT_TAKEN;
    const at::Tensor &out = THPVariable_Unpack(a[2]);
    if (!out.is_cuda() || out.element_size() != 4) return NOT_TAKEN;
    float *px = at_f32(x);
    uint32_t *po = static_cast<uint32_t *>(out.data_ptr());
    const uint32_t n = static_cast<uint32_t>(x->numel());
    return on_stream([&](void *s) { return lib.argmax(ctx, s, px, n, po); });
}

long sample(PyObject *const *a) {   // ctx, logits, vocabulary, temperature, topp, coin, out
    ib_ctx *ctx = handle<ib_ctx>(a[0]);
    const at::Tensor *x = dense_f32(a[1]);
    if (!ctx || !x || !THPVariable_CheckExact(a[6])) return NOT_TAKEN;
    const uint32_t n = u32(a[2]);
    const float temperature = f32(a[3]), topp = f32(a[4]), coin = f32(a[5]);
    const at::Tensor &out = THPVariable_Unpack(a[6]);
    if (x->numel() != n || !out.is_cuda() || PyErr_Occurred()) return NOT_TAKEN;
    float *px = at_f32(x);
    uint32_t *po = static_cast<uint32_t *>(out.data_ptr());
    return on_stream([&](void *s) { return lib.sample(ctx, s, px, n, temperature, topp, coin, po); });
}

// The library's entry points, in the order of `Entry`, from whoever loaded it
PyObject *bind(PyObject *, PyObject *const *args, Py_ssize_t n) {
    if (n != ENTRIES) {
        PyErr_SetString(PyExc_TypeError, "bind: one address per entry point");
        return nullptr;
    }
    void *to[ENTRIES];
    for (Py_ssize_t i = 0; i < n; i++) {
        to[i] = PyLong_AsVoidPtr(args[i]);
        if (PyErr_Occurred()) return nullptr;
    }
    memcpy(&lib, to, sizeof lib);
    Py_RETURN_NONE;
}

template <long (*F)(PyObject *const *), Py_ssize_t N>
PyMethodDef method(const char *name) {
    return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<F, N>)), METH_FASTCALL, nullptr};
}
PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&bind)), METH_FASTCALL, nullptr},
    method<gemv, 6>("gemv"),
    method<gemm, 6>("gemm"),
    method<rms_norm, 5>("rms_norm"),
    method<rope, 8>("rope"),
    method<pairwise<&Entry::silu>, 3>("silu"),
    method<pairwise<&Entry::add>, 3>("add"),
    method<attention, 6>("attention"),
    method<argmax, 3>("argmax"),
    method<sample, 7>("sample"),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// `stamp`: the torch that this was compiled against.  Tensors are read through its headers' inline code, so it serves no other one.
PyMODINIT_FUNC PyInit__binding() {
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "stamp", IB_BINDING_STAMP)) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
