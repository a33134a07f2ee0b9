// Host side of the ops in native code: argument checks, output allocation and the launch of one op per call from
// Python, as a CPython extension over the C ABI (fastcall, no binding layer).
//
// Every function here is the common case of the function of the same name in native.py and returns None for anything
// else: tensors that are not plain, dense CUDA tensors of the current device, active dispatch modes or transforms,
// shapes, types and alignments it does not know, and everything that is to be refused.  The Python function then does
// the whole of its own work, so what is accepted, what is refused and how is decided in one place.  An error of a
// launch itself is raised from here, by _lib.check.
//
// What it is for: a ctypes call with its argument conversions, torch.empty and the checks in Python cost 4 to 8 us an op,
// more than the kernels of a short call take.

#include <Python.h>

#include <ATen/ops/empty.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include <cmath>

#include "../../include/q8_kernels_b200.h"

namespace {

PyObject* g_check = nullptr;                                   // _lib.check(rc, op): raises Q8KernelError
constexpr int kMaxDevices = 64;
at::Tensor* g_status[kMaxDevices] = {};                        // the devices' status words (set_status_word)

using Dt = at::ScalarType;

int dt_code(Dt t) {
    switch (t) {
        case Dt::Float: return Q8K_DT_F32;
        case Dt::BFloat16: return Q8K_DT_BF16;
        case Dt::Float8_e4m3fn: return Q8K_DT_E4M3;
        case Dt::Char: return Q8K_DT_I8;
        default: return -1;                                    // not on a fast path
    }
}

// The arguments of one call.  `ok` turns false as soon as one of them is not what the fast path takes, their number first of
// all; from then on none is looked at any more.
struct Call {
    PyObject* const* args;
    bool ok;
    c10::DeviceIndex dev = -1;

    Call(PyObject* const* a, Py_ssize_t n, Py_ssize_t want) : args(a), ok(n == want) {
        // a transform, a tracer or a mode that wants to see the ops
        if (c10::impl::TorchDispatchModeTLS::any_modes_set()) ok = false;
        const auto tls = c10::impl::tls_local_dispatch_key_set();
        if (tls.included_.has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchDynamicLayerFrontMode,
                                                       c10::DispatchKey::FuncTorchDynamicLayerBackMode,
                                                       c10::DispatchKey::FuncTorchBatched,
                                                       c10::DispatchKey::FuncTorchVmapMode, c10::DispatchKey::VmapMode,
                                                       c10::DispatchKey::Functionalize, c10::DispatchKey::Tracer,
                                                       c10::DispatchKey::Python, c10::DispatchKey::PreDispatch})))
            ok = false;
    }
    // A plain CUDA tensor of the device that is current; contiguous unless `strided`.
    const at::Tensor* tensor(int i, bool strided = false) { return ok ? tensor_of(args[i], strided) : nullptr; }
    const at::Tensor* tensor_of(PyObject* o, bool strided = false) {
        static const uint64_t plain =
            c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutogradCUDA,
                                 c10::DispatchKey::AutocastCUDA}).raw_repr();
        ok = false;
        if (!THPVariable_Check(o)) return nullptr;
        const at::Tensor& t = THPVariable_Unpack(o);
        if (!t.defined() || !t.is_cuda() || (t.key_set().raw_repr() & ~plain) != 0) return nullptr;
        if (!strided && !t.is_contiguous()) return nullptr;
        const c10::DeviceIndex d = t.device().index();
        if (dev < 0) {
            if (d >= kMaxDevices || d != c10::cuda::current_device()) return nullptr;
            dev = d;
        } else if (d != dev) {
            return nullptr;
        }
        ok = true;
        return &t;
    }
    const at::Tensor* tensor(int i, Dt type, bool strided = false) {
        const at::Tensor* t = tensor(i, strided);
        if (t != nullptr && t->scalar_type() != type) ok = false;
        return t;
    }
    const at::Tensor* optional(int i, Dt type) { return !ok || args[i] == Py_None ? nullptr : tensor(i, type); }
    Dt dtype(int i, Dt none) {
        if (!ok || args[i] == Py_None) return none;
        if (!THPDtype_Check(args[i])) { ok = false; return none; }
        return reinterpret_cast<THPDtype*>(args[i])->scalar_type;
    }
    bool flag(int i) {
        if (!ok) return false;
        if (args[i] == Py_True) return true;
        if (args[i] != Py_False) ok = false;
        return false;
    }
    long integer(int i) {
        if (!ok) return 0;
        if (!PyLong_CheckExact(args[i])) { ok = false; return 0; }
        const long v = PyLong_AsLong(args[i]);
        if (v < 0 || v > 0x7fffffff) { PyErr_Clear(); ok = false; }
        return v;
    }
    float real(int i) {
        if (!ok) return 0.f;
        if (!PyFloat_CheckExact(args[i])) { ok = false; return 0.f; }
        return (float)PyFloat_AS_DOUBLE(args[i]);
    }
    int* status() {
        if (ok && g_status[dev] == nullptr) ok = false;        // the Python path makes it
        return ok ? g_status[dev]->data_ptr<int>() : nullptr;
    }
    void* stream() const { return c10::cuda::getCurrentCUDAStream(dev).stream(); }
    void need(bool cond) { ok = ok && cond; }
    at::Tensor empty(at::IntArrayRef shape, Dt type) const {
        return at::empty(shape, at::TensorOptions().dtype(type).device(c10::Device(c10::kCUDA, dev)));
    }
};

// Allocation and launch without the interpreter lock, as torch and ctypes do them.  (The caller's references keep the
// arguments alive.)
struct WithoutGil {
    PyThreadState* state = PyEval_SaveThread();
    ~WithoutGil() { PyEval_RestoreThread(state); }
};
template <typename F> int launch(F&& f) {
    WithoutGil unlocked;
    return f();
}

// True when the launch was taken; otherwise the Python error is set.
bool launched(int rc, const char* op) {
    if (rc == Q8K_OK) return true;
    PyObject* r = PyObject_CallFunction(g_check, "is", rc, op);
    Py_XDECREF(r);
    if (r != nullptr) PyErr_SetString(PyExc_RuntimeError, "q8_kernels_b200: a launch failed");
    return false;
}

PyObject* wrap(at::Tensor&& t) { return THPVariable_Wrap(std::move(t)); }
PyObject* list2(at::Tensor&& a, at::Tensor&& b) {
    PyObject* l = PyList_New(2);
    if (l == nullptr) return nullptr;
    PyList_SET_ITEM(l, 0, wrap(std::move(a)));
    PyList_SET_ITEM(l, 1, wrap(std::move(b)));
    return l;
}
PyObject* tuple_of(at::Tensor (&t)[3]) {                       // of those that are defined
    PyObject* r = PyTuple_New(t[0].defined() + t[1].defined() + t[2].defined());
    if (r == nullptr) return nullptr;
    Py_ssize_t k = 0;
    for (at::Tensor& x : t)
        if (x.defined()) PyTuple_SET_ITEM(r, k++, wrap(std::move(x)));
    return r;
}

const void* cptr(const at::Tensor* t) { return t == nullptr ? nullptr : t->const_data_ptr(); }
const float* fptr(const at::Tensor* t) { return static_cast<const float*>(cptr(t)); }
bool int_sized(int64_t v) { return v >= 0 && v <= 0x7fffffffLL; }
at::IntArrayRef lead(const at::Tensor& t) { return t.sizes().slice(0, t.dim() - 1); }   // shape without the last dim
bool has_rows(const at::Tensor* t) { return t->dim() >= 1 && t->size(-1) > 0 && int_sized(t->size(-1)); }
bool quant_type(Dt t) { return t == Dt::Char || t == Dt::Float8_e4m3fn; }

#define FAST_BEGIN HANDLE_TH_ERRORS
#define FAST_END END_HANDLE_TH_ERRORS                          // torch's own exceptions, out of memory among them
#define OR_NONE(c) \
    if (!(c).ok) Py_RETURN_NONE

// ---------------------------------------------------------------- rows
// tokenwise_quant(x, out_type)
PyObject* tokenwise_quant(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 2);
    const at::Tensor* x = c.tensor(0);
    const Dt out = c.dtype(1, Dt::Char);
    OR_NONE(c);
    c.need(has_rows(x) && quant_type(out) && dt_code(x->scalar_type()) >= 0);
    OR_NONE(c);
    const int dim = (int)x->size(-1);
    at::Tensor q, s;
    const int rc = launch([&] {
        q = c.empty(x->sizes(), out);
        s = c.empty(lead(*x), Dt::Float);
        return q8k_tokenwise_quant(cptr(x), dt_code(x->scalar_type()), q.data_ptr(), dt_code(out), s.data_ptr<float>(),
                                   x->numel() / dim, dim, dim, c.stream());
    });
    return launched(rc, "tokenwise_quant") ? list2(std::move(q), std::move(s)) : nullptr;
    FAST_END
}

// hadamard_quant(x, scale, out_type)
PyObject* hadamard_quant(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 3);
    const at::Tensor* x = c.tensor(0);
    const float scale = c.real(1);
    const Dt out = c.dtype(2, Dt::Char);
    OR_NONE(c);
    c.need(has_rows(x) && quant_type(out) && dt_code(x->scalar_type()) >= 0);
    OR_NONE(c);
    const int dim = (int)x->size(-1);
    at::Tensor q, s;
    const int rc = launch([&] {
        q = c.empty(x->sizes(), out);
        s = c.empty(lead(*x), Dt::Float);
        return q8k_hadamard_quant(cptr(x), dt_code(x->scalar_type()), q.data_ptr(), dt_code(out), s.data_ptr<float>(),
                                  x->numel() / dim, dim, dim, scale, c.stream());
    });
    return launched(rc, "hadamard_quant") ? list2(std::move(q), std::move(s)) : nullptr;
    FAST_END
}

// fast_hadamard_transform(x, scale, out_type)
PyObject* fast_hadamard_transform(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 3);
    const at::Tensor* x = c.tensor(0);
    const float scale = c.real(1);
    OR_NONE(c);
    const Dt in = x->scalar_type();
    const Dt out = c.dtype(2, in);
    c.need(has_rows(x) && x->size(-1) % 8 == 0 && (in == Dt::BFloat16 || in == Dt::Float8_e4m3fn) && dt_code(out) >= 0);
    OR_NONE(c);
    const int dim = (int)x->size(-1);
    at::Tensor y;
    const int rc = launch([&] {
        y = c.empty(x->sizes(), out);
        return q8k_fast_hadamard_transform(cptr(x), dt_code(in), y.data_ptr(), dt_code(out), x->numel() / dim, dim, dim,
                                           scale, c.stream());
    });
    return launched(rc, "fast_hadamard_transform") ? wrap(std::move(y)) : nullptr;
    FAST_END
}

// norm_modulate_quant(x, mod_scale, mod_shift, out_type)
PyObject* norm_modulate_quant(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 4);
    const at::Tensor* x = c.tensor(0, Dt::BFloat16);
    const at::Tensor* sc = c.tensor(1, Dt::BFloat16);
    const at::Tensor* sh = c.tensor(2, Dt::BFloat16);
    const Dt out = c.dtype(3, Dt::Char);
    OR_NONE(c);
    c.need(x->dim() == 3 && has_rows(x) && quant_type(out));
    OR_NONE(c);
    const int64_t B = x->size(0), S = x->size(1), dim = x->size(2);
    for (const at::Tensor* m : {sc, sh}) c.need(m->dim() == 3 && m->size(0) == B && m->size(1) == 1 && m->size(2) == dim);
    OR_NONE(c);
    at::Tensor q, s;
    const float scale = (float)(1.0 / std::sqrt((double)dim));
    const int rc = launch([&] {
        q = c.empty(x->sizes(), out);
        s = c.empty({B, S}, Dt::Float);
        return q8k_norm_modulate_quant(cptr(x), cptr(sc), cptr(sh), q.data_ptr(), dt_code(out), s.data_ptr<float>(), B * S,
                                       (int)dim, S, scale, c.stream());
    });
    return launched(rc, "norm_modulate_quant") ? list2(std::move(q), std::move(s)) : nullptr;
    FAST_END
}

// transpose_quant(x, row_scales | None)
PyObject* transpose_quant(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 2);
    const at::Tensor* x = c.tensor(0);
    const at::Tensor* rs = c.optional(1, Dt::Float);
    OR_NONE(c);
    c.need(x->dim() == 2 && int_sized(x->size(0)) && int_sized(x->size(1)) && dt_code(x->scalar_type()) >= 0 &&
           (rs == nullptr || rs->numel() == x->size(0)));
    OR_NONE(c);
    const int64_t rows = x->size(0), k = x->size(1);
    at::Tensor q, s;
    const int rc = launch([&] {
        q = c.empty({k, rows}, Dt::Float8_e4m3fn);
        s = c.empty({k}, Dt::Float);
        return q8k_transpose_quant(cptr(x), dt_code(x->scalar_type()), fptr(rs), q.data_ptr(), s.data_ptr<float>(), (int)rows,
                                   (int)k, c.stream());
    });
    return launched(rc, "transpose_quant") ? list2(std::move(q), std::move(s)) : nullptr;
    FAST_END
}

// dequant_hadamard(x, row_scales, scale)
PyObject* dequant_hadamard(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 3);
    const at::Tensor* x = c.tensor(0, Dt::Char);
    const at::Tensor* rs = c.tensor(1, Dt::Float);
    const float scale = c.real(2);
    OR_NONE(c);
    c.need(x->dim() == 2 && int_sized(x->size(1)) && rs->numel() == x->size(0));
    OR_NONE(c);
    at::Tensor y;
    const int rc = launch([&] {
        y = c.empty(x->sizes(), Dt::BFloat16);
        return q8k_dequant_hadamard(cptr(x), fptr(rs), y.data_ptr(), x->size(0), (int)x->size(1), scale, c.stream());
    });
    return launched(rc, "dequant_hadamard") ? wrap(std::move(y)) : nullptr;
    FAST_END
}

// rms_norm(x, weights | None, out_type)
PyObject* rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 3);
    const at::Tensor* x = c.tensor(0);
    const at::Tensor* w = c.optional(1, Dt::Float);
    OR_NONE(c);
    const Dt out = c.dtype(2, x->scalar_type());
    c.need(has_rows(x) && dt_code(x->scalar_type()) >= 0 && dt_code(out) >= 0 && (w == nullptr || w->numel() == x->size(-1)));
    OR_NONE(c);
    const int dim = (int)x->size(-1);
    at::Tensor y, r;
    const int rc = launch([&] {
        y = c.empty(x->sizes(), out);
        r = c.empty(lead(*x), Dt::Float);
        return q8k_rms_norm(cptr(x), dt_code(x->scalar_type()), fptr(w), y.data_ptr(), dt_code(out), r.data_ptr<float>(),
                            x->numel() / dim, dim, c.stream());
    });
    return launched(rc, "rms_norm") ? list2(std::move(y), std::move(r)) : nullptr;
    FAST_END
}

// rms_norm_backward(x_normed, x_norms, grad_out, weights | None, out_type)
PyObject* rms_norm_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 5);
    const at::Tensor* y = c.tensor(0);
    const at::Tensor* r = c.tensor(1, Dt::Float);
    const at::Tensor* g = c.tensor(2);
    const at::Tensor* w = c.optional(3, Dt::Float);
    OR_NONE(c);
    const Dt out = c.dtype(4, y->scalar_type());
    c.need(has_rows(y) && dt_code(y->scalar_type()) >= 0 && dt_code(out) >= 0 && g->scalar_type() == out &&
           g->sizes() == y->sizes() && (w == nullptr || w->numel() == y->size(-1)));
    OR_NONE(c);
    const int dim = (int)y->size(-1);
    const int64_t rows = y->numel() / dim;
    c.need(r->numel() == rows);
    OR_NONE(c);
    at::Tensor gx;
    const int rc = launch([&] {
        gx = c.empty(y->sizes(), out);
        return q8k_rms_norm_backward(cptr(y), dt_code(y->scalar_type()), fptr(r), cptr(g), fptr(w), gx.data_ptr(), dt_code(out),
                                     rows, dim, c.stream());
    });
    return launched(rc, "rms_norm_backward") ? wrap(std::move(gx)) : nullptr;
    FAST_END
}

// rope(x, cos, sin, out_type) and rope_backward(grad, cos, sin, out_type)
using RopeFn = int (*)(const void*, int, const float*, const float*, void*, int, int64_t, int, int64_t, void*);
PyObject* rope_like(RopeFn fn, const char* op, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 4);
    const at::Tensor* x = c.tensor(0);
    const at::Tensor* co = c.tensor(1, Dt::Float);
    const at::Tensor* si = c.tensor(2, Dt::Float);
    OR_NONE(c);
    const Dt out = c.dtype(3, x->scalar_type());
    c.need(has_rows(x) && dt_code(x->scalar_type()) >= 0 && dt_code(out) >= 0 && co->sizes() == si->sizes() && co->dim() >= 1 &&
           co->size(-1) == x->size(-1));
    OR_NONE(c);
    const int dim = (int)x->size(-1);
    const int64_t rows = x->numel() / dim, table = co->numel() / dim;
    c.need(table > 0 && (table == rows || (rows % table == 0 && co->dim() == x->dim() && co->size(0) == 1)));
    OR_NONE(c);
    at::Tensor y;
    const int rc = launch([&] {
        y = c.empty(x->sizes(), out);
        return fn(cptr(x), dt_code(x->scalar_type()), fptr(co), fptr(si), y.data_ptr(), dt_code(out), rows, dim,
                  table == rows ? 0 : table, c.stream());
    });
    return launched(rc, op) ? wrap(std::move(y)) : nullptr;
    FAST_END
}
PyObject* rope(PyObject*, PyObject* const* args, Py_ssize_t n) { return rope_like(q8k_rope, "rope", args, n); }
PyObject* rope_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return rope_like(q8k_rope_backward, "rope_backward", args, n);
}

// ---------------------------------------------------------------- products
// mm(a, b, bias | None, a_scales, b_scales, fuse_gelu, out_type, in_type, op): in_type int8 or e4m3, op the public name
PyObject* mm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 9);
    const Dt in = c.dtype(7, Dt::Undefined);
    const at::Tensor* a = c.tensor(0, in);
    const at::Tensor* b = c.tensor(1, in);
    const at::Tensor* bias = c.optional(2, Dt::Float);
    const at::Tensor* sa = c.tensor(3, Dt::Float);
    const at::Tensor* sb = c.tensor(4, Dt::Float);
    const bool gelu = c.flag(5);
    const Dt out = c.dtype(6, Dt::Float8_e4m3fn);
    c.need(c.ok && PyUnicode_Check(args[8]));
    OR_NONE(c);
    c.need(quant_type(in) && dt_code(out) >= 0 &&
           (a->dim() == 2 || a->dim() == 3) && (b->dim() == 2 || b->dim() == 3));
    OR_NONE(c);
    const int64_t ba = a->dim() == 3 ? a->size(0) : 1, m = a->size(-2), k = a->size(-1);
    const int64_t bb = b->dim() == 3 ? b->size(0) : 1, nn = b->size(-2);
    c.need(b->size(-1) == k && (ba == bb || ba == 1 || bb == 1) && int_sized(ba * m) && int_sized(bb * nn) && int_sized(k) &&
           sa->numel() == ba * m && sb->numel() == bb * nn && (bias == nullptr || bias->numel() == nn));
    int* word = c.status();
    OR_NONE(c);
    at::Tensor y;
    const bool i8 = in == Dt::Char;
    const int rc = launch([&] {
        y = c.empty({ba > bb ? ba : bb, m, nn}, out);
        return (i8 ? q8k_q8_mm : q8k_fp8_mm)(cptr(a), cptr(b), fptr(bias), fptr(sa), fptr(sb), y.data_ptr(), dt_code(out), (int)ba,
                                             (int)bb, (int)m, (int)nn, (int)k, gelu, word, c.stream());
    });
    const char* op = rc == Q8K_OK ? "" : PyUnicode_AsUTF8(args[8]);
    return op != nullptr && launched(rc, op) ? wrap(std::move(y)) : nullptr;
    FAST_END
}

// mm_gate_residual(a, b, bias | None, a_scales, b_scales, gate | None, resid)
PyObject* mm_gate_residual(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 7);
    const at::Tensor* a = c.tensor(0);
    const at::Tensor* b = c.tensor(1);
    const at::Tensor* bias = c.optional(2, Dt::Float);
    const at::Tensor* sa = c.tensor(3, Dt::Float);
    const at::Tensor* sb = c.tensor(4, Dt::Float);
    const at::Tensor* gate = c.optional(5, Dt::BFloat16);
    const at::Tensor* resid = c.tensor(6, Dt::BFloat16);
    OR_NONE(c);
    c.need(quant_type(a->scalar_type()) && b->scalar_type() == a->scalar_type() && (a->dim() == 2 || a->dim() == 3) &&
           b->dim() == 2);
    OR_NONE(c);
    const int64_t ba = a->dim() == 3 ? a->size(0) : 1, m = a->size(-2), k = a->size(-1), nn = b->size(0);
    c.need(b->size(1) == k && int_sized(ba * m) && int_sized(nn) && int_sized(k) && sa->numel() == ba * m && sb->numel() == nn &&
           (bias == nullptr || bias->numel() == nn) && resid->numel() == ba * m * nn &&
           (gate == nullptr || gate->numel() == ba * nn));
    int* word = c.status();
    OR_NONE(c);
    at::Tensor y;
    const int rc = launch([&] {
        y = c.empty({ba, m, nn}, Dt::BFloat16);
        return q8k_mm_gate_residual(a->scalar_type() == Dt::Char, cptr(a), cptr(b), fptr(bias), fptr(sa), fptr(sb), cptr(gate),
                                    cptr(resid), gate == nullptr ? 1 : m, y.data_ptr(), (int)ba, 1, (int)m, (int)nn, (int)k, word,
                                    c.stream());
    });
    return launched(rc, "mm_gate_residual") ? wrap(std::move(y)) : nullptr;
    FAST_END
}

// linear(x, w, w_scales, bias | None, use_hadamard, fuse_gelu, out_type)
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 7);
    const at::Tensor* x = c.tensor(0);
    const at::Tensor* w = c.tensor(1);
    const at::Tensor* ws = c.tensor(2, Dt::Float);
    const at::Tensor* bias = c.optional(3, Dt::Float);
    const bool had = c.flag(4), gelu = c.flag(5);
    const Dt out = c.dtype(6, Dt::Undefined);
    OR_NONE(c);
    c.need((x->dim() == 2 || x->dim() == 3) && w->dim() == 2 && quant_type(w->scalar_type()) && dt_code(x->scalar_type()) >= 0 &&
           dt_code(out) >= 0 && has_rows(x) && w->size(1) == x->size(-1) && int_sized(w->size(0)) && ws->numel() == w->size(0) &&
           (bias == nullptr || bias->numel() == w->size(0)));
    int* word = c.status();
    OR_NONE(c);
    const int64_t k = x->size(-1), m = x->numel() / k, nn = w->size(0);
    c.need(int_sized(m));
    OR_NONE(c);
    // Scratch for the quantised rows, given back to the allocator when the call returns: it is handed out again only to
    // work that is queued behind these kernels on the same stream.
    const size_t need = q8k_linear_workspace_bytes((int)m, (int)k);
    at::Tensor scratch, y;
    const int rc = launch([&] {
        scratch = c.empty({(int64_t)(need > 0 ? need : 1)}, Dt::Byte);
        y = x->dim() == 3 ? c.empty({x->size(0), x->size(1), nn}, out) : c.empty({1, m, nn}, out);
        return q8k_linear(cptr(x), dt_code(x->scalar_type()), cptr(w), dt_code(w->scalar_type()), fptr(ws), fptr(bias),
                          y.data_ptr(), dt_code(out), (int)m, (int)nn, (int)k, had, gelu, scratch.data_ptr(), need, word, c.stream());
    });
    return launched(rc, "linear") ? wrap(std::move(y)) : nullptr;
    FAST_END
}

// ---------------------------------------------------------------- attention
// flash_attention(q, k, v, scale, key_lens | None, out_type, token_major): v as rows [B,H,N,64]
PyObject* flash_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 7);
    const at::Tensor* q = c.tensor(0, Dt::Float8_e4m3fn);
    const at::Tensor* k = c.tensor(1, Dt::Float8_e4m3fn);
    const at::Tensor* v = c.tensor(2, Dt::Float8_e4m3fn);
    const float scale = c.real(3);
    const at::Tensor* lens = c.optional(4, Dt::Int);
    const Dt out = c.dtype(5, Dt::Float8_e4m3fn);
    const bool token_major = c.flag(6);
    OR_NONE(c);
    c.need(q->dim() == 4 && k->dim() == 4 && v->sizes() == k->sizes() && dt_code(out) >= 0);
    OR_NONE(c);
    const int64_t B = q->size(0), H = q->size(1), M = q->size(2), N = k->size(2);
    c.need(q->size(3) == 64 && k->size(3) == 64 && k->size(0) == B && k->size(1) == H && int_sized(B) && int_sized(H) &&
           int_sized(M) && int_sized(N) && (lens == nullptr || (lens->dim() == 1 && lens->size(0) == B)));
    int* word = c.status();
    OR_NONE(c);
    at::Tensor o;
    const int rc = launch([&] {
        o = token_major ? c.empty({B, M, H, 64}, out) : c.empty({B, H, M, 64}, out);
        void* outs[1] = {o.data_ptr()};
        return q8k_flash_attention_v_rows(cptr(q), cptr(k), cptr(v), outs, 1, dt_code(out), (int)B, (int)H, (int)M, (int)N,
                                          H * M * 64, token_major ? 64 : M * 64, token_major ? H * 64 : 64, scale,
                                          static_cast<const int*>(cptr(lens)), word, c.stream());
    });
    if (!launched(rc, "flash_attention")) return nullptr;
    return wrap(token_major ? o.transpose(1, 2) : std::move(o));
    FAST_END
}

// attention_prep_rows(q, k, v, apply_hadamard, scale): [B,H,S,64] views of any batch, head and token strides
PyObject* attention_prep_rows(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 5);
    const at::Tensor* t[3];
    for (int i = 0; i < 3; ++i) t[i] = c.tensor(i, Dt::BFloat16, true);
    const bool had = c.flag(3);
    const float scale = c.real(4);
    OR_NONE(c);
    for (int i = 0; i < 3; ++i)
        c.need(t[i]->dim() == 4 && t[i]->size(3) == 64 && t[i]->stride(3) == 1 && t[i]->stride(0) % 8 == 0 &&
               t[i]->stride(1) % 8 == 0 && t[i]->stride(2) % 8 == 0 && (uintptr_t)cptr(t[i]) % 16 == 0 && int_sized(t[i]->size(2)));
    OR_NONE(c);
    const int64_t B = t[0]->size(0), H = t[0]->size(1);
    c.need(t[1]->size(0) == B && t[1]->size(1) == H && t[2]->sizes() == t[1]->sizes() && int_sized(B) && int_sized(H));
    OR_NONE(c);
    at::Tensor o[3];
    const int rc = launch([&] {
        for (int i = 0; i < 3; ++i) o[i] = c.empty({B, H, t[i]->size(2), 64}, Dt::Float8_e4m3fn);
        return q8k_attention_prep_rows(cptr(t[0]), cptr(t[1]), cptr(t[2]), o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(),
                                       (int)B, (int)H, (int)t[0]->size(2), (int)t[1]->size(2), t[0]->stride(0), t[0]->stride(2),
                                       t[0]->stride(1), t[1]->stride(0), t[1]->stride(2), t[1]->stride(1), t[2]->stride(0),
                                       t[2]->stride(2), t[2]->stride(1), had, scale, c.stream());
    });
    if (!launched(rc, "attention_prep_rows")) return nullptr;
    return tuple_of(o);
    FAST_END
}

// The pre-passes of a projection's output.  Q, K and V (those that an op has) are column slices [B,S,H*64] of one tensor; the
// result is their e4m3 tensors.
struct Prep {
    const at::Tensor *q = nullptr, *k = nullptr, *v = nullptr, *wq = nullptr, *wk = nullptr;
    at::Tensor cos, sin;                                       // owned: a list may change while the lock is given up
    int64_t heads = 0;
    bool hadamard = false;
    float scale = 0.f;
    bool rotate = false;

    // freqs_cis: None or a (cos, sin) tuple or list; anything else is left as it is, an iterator unread
    void tables(Call& c, int i) {
        if (!c.ok || c.args[i] == Py_None) return;
        PyObject* f = c.args[i];
        if (!(PyTuple_CheckExact(f) || PyList_CheckExact(f)) || PySequence_Fast_GET_SIZE(f) != 2) { c.ok = false; return; }
        const at::Tensor* t[2] = {nullptr, nullptr};
        for (int k = 0; k < 2 && c.ok; ++k) t[k] = c.tensor_of(PySequence_Fast_GET_ITEM(f, k));
        c.need(c.ok && t[0]->scalar_type() == Dt::Float && t[1]->scalar_type() == Dt::Float);
        if (!c.ok) return;
        cos = *t[0];
        sin = *t[1];
        rotate = true;
    }
};

PyObject* prep(Call& c, const Prep& a, const char* op) {
    OR_NONE(c);
    const at::Tensor& k = *a.k;
    const at::Tensor* x[3] = {a.q, a.k, a.v};
    c.need(k.dim() == 3 && k.size(2) == a.heads * 64);
    OR_NONE(c);
    const int64_t B = k.size(0), S = k.size(1), C = a.heads * 64, rs = k.stride(1);
    for (const at::Tensor* t : x)
        c.need(t == nullptr || (t->sizes() == k.sizes() && t->strides() == k.strides() && (uintptr_t)cptr(t) % 16 == 0));
    c.need(k.stride(2) == 1 && k.stride(0) == S * rs && rs % 8 == 0 && int_sized(B) && int_sized(S) && int_sized(C) &&
           a.wk->numel() == C && (a.wq == nullptr || a.wq->numel() == C) &&
           (!a.rotate || (a.cos.numel() == S * C && a.sin.numel() == S * C)));
    OR_NONE(c);
    const float* co = a.rotate ? fptr(&a.cos) : nullptr;
    const float* si = a.rotate ? fptr(&a.sin) : nullptr;
    at::Tensor o[3];
    void* p[3] = {nullptr, nullptr, nullptr};
    const int rc = launch([&] {
        for (int i = 0; i < 3; ++i)
            if (x[i] != nullptr) {
                o[i] = c.empty({B, a.heads, S, 64}, Dt::Float8_e4m3fn);
                p[i] = o[i].data_ptr();
            }
        if (a.v != nullptr)
            return q8k_qkv_prep(cptr(a.q), cptr(a.k), cptr(a.v), rs, fptr(a.wq), fptr(a.wk), co, si, p[0], p[1], p[2], (int)B,
                                (int)S, (int)a.heads, a.hadamard, a.scale, c.stream());
        if (a.q != nullptr)
            return q8k_qk_norm_rope_prep_pair(cptr(a.q), cptr(a.k), rs, fptr(a.wq), fptr(a.wk), co, si, p[0], p[1], (int)B, (int)S,
                                              (int)a.heads, a.hadamard, a.scale, c.stream());
        return q8k_qk_norm_rope_prep(cptr(a.k), rs, fptr(a.wk), co, si, p[1], (int)B, (int)S, (int)a.heads, a.hadamard, a.scale,
                                     c.stream());
    });
    if (!launched(rc, op)) return nullptr;
    return a.q == nullptr && a.v == nullptr ? wrap(std::move(o[1])) : tuple_of(o);
}

// qk_norm_rope_prep(x, norm_w, freqs_cis, heads, apply_hadamard, scale)
PyObject* qk_norm_rope_prep(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 6);
    Prep a;
    a.k = c.tensor(0, Dt::BFloat16, true);
    a.wk = c.tensor(1, Dt::Float);
    a.tables(c, 2);
    a.heads = c.integer(3);
    a.hadamard = c.flag(4);
    a.scale = c.real(5);
    return prep(c, a, "qk_norm_rope_prep");
    FAST_END
}

// kv_prep(xk, xv, norm_wk, heads, apply_hadamard, scale)
PyObject* kv_prep(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 6);
    Prep a;
    a.k = c.tensor(0, Dt::BFloat16, true);
    a.v = c.tensor(1, Dt::BFloat16, true);
    a.wk = c.tensor(2, Dt::Float);
    a.heads = c.integer(3);
    a.hadamard = c.flag(4);
    a.scale = c.real(5);
    return prep(c, a, "qkv_prep");
    FAST_END
}

// qk_norm_rope_prep_pair(xq, xk, norm_wq, norm_wk, freqs_cis, heads, apply_hadamard, scale, xv | None)
PyObject* qk_norm_rope_prep_pair(PyObject*, PyObject* const* args, Py_ssize_t n) {
    FAST_BEGIN
    Call c(args, n, 9);
    Prep a;
    a.q = c.tensor(0, Dt::BFloat16, true);
    a.k = c.tensor(1, Dt::BFloat16, true);
    a.wq = c.tensor(2, Dt::Float);
    a.wk = c.tensor(3, Dt::Float);
    a.tables(c, 4);
    a.heads = c.integer(5);
    a.hadamard = c.flag(6);
    a.scale = c.real(7);
    if (c.ok && args[8] != Py_None) a.v = c.tensor(8, Dt::BFloat16, true);
    return prep(c, a, a.v == nullptr ? "qk_norm_rope_prep_pair" : "qkv_prep");
    FAST_END
}

// ---------------------------------------------------------------- module
PyObject* set_check(PyObject*, PyObject* f) {
    Py_INCREF(f);
    Py_XSETREF(g_check, f);
    Py_RETURN_NONE;
}
// set_status_word(tensor): the word that the launches on its device write when a wait is abandoned
PyObject* set_status_word(PyObject*, PyObject* o) {
    if (!THPVariable_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "set_status_word: a tensor is expected");
        return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.scalar_type() != Dt::Int || t.device().index() >= kMaxDevices) {
        PyErr_SetString(PyExc_TypeError, "set_status_word: an int32 CUDA tensor is expected");
        return nullptr;
    }
    at::Tensor*& slot = g_status[t.device().index()];
    if (slot == nullptr) slot = new at::Tensor(t);             // kept for the life of the process, as the device's context is
    else *slot = t;
    Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FAST(tokenwise_quant), FAST(hadamard_quant), FAST(fast_hadamard_transform), FAST(norm_modulate_quant), FAST(transpose_quant),
    FAST(dequant_hadamard), FAST(rms_norm), FAST(rms_norm_backward), FAST(rope), FAST(rope_backward), FAST(mm),
    FAST(mm_gate_residual), FAST(linear), FAST(flash_attention), FAST(attention_prep_rows), FAST(qk_norm_rope_prep),
    FAST(kv_prep), FAST(qk_norm_rope_prep_pair),
    {"set_check", set_check, METH_O, nullptr}, {"set_status_word", set_status_word, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
    PyObject* m = PyModule_Create(&module);
    if (m != nullptr && PyModule_AddStringConstant(m, "__torch_version__", TORCH_VERSION) != 0) Py_CLEAR(m);
    return m;
}
