// native_ops.cpp -- the tensor side of fluke_b200.ops: argument checks, output allocation and the
// call of the C entry point in one step per operator (extension module fluke_b200._native).
//
// A small launch costs the GPU two or three microseconds; the same call through ctypes costs the
// host eight to ten (attribute look-ups for the checks, one Python call per data pointer,
// torch.empty, conversion of up to eleven arguments). Here the arguments are read from the
// tensors directly and the output comes from the CUDA allocator without the dispatcher.
//
// The functions take exactly the positional arguments that ops.py passes. The entry points are those
// of the library that fluke_b200.lib has loaded: bind() receives their addresses, so both share one
// copy of its state (stream setting, last error, prepared weights). The interpreter lock is
// released around every entry point.
#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>

#include <fluke/fluke.h>

namespace {

#define FLUKE_NATIVE_FUNCTIONS(X) \
    X(fluke_rmsnorm_gpu) X(fluke_rmsnorm_quant_int8_gpu) X(fluke_rmsnorm_quant_fp8_gpu) X(fluke_quant_int8_gpu) \
    X(fluke_quant_fp8_gpu) X(fluke_dequant_fp8_transpose_gpu) X(fluke_dequant_int8_transpose_gpu) X(fluke_rotary_emb_gpu) \
    X(fluke_silu_mul_gpu) X(fluke_flstm_step_gpu) X(fluke_qkv_rotary_i8_gpu) X(fluke_gated_mlp_i8_gpu) \
    X(fluke_qkv_rotary_fp8_gpu) X(fluke_gated_mlp_fp8_gpu) X(fluke_qkv_rotary_fp8_plain_gpu) \
    X(fluke_gated_mlp_fp8_plain_gpu) X(fluke_gemm_i8_gpu) X(fluke_gemm_fp8_gpu) X(fluke_down_proj_i8_gpu) \
    X(fluke_down_proj_fp8_gpu) X(fluke_factored_lstm_step_i8_gpu) X(fluke_factored_lstm_step_fp8_gpu) X(fluke_last_error)

struct Entry {
#define X(name) decltype(&::name) name = nullptr;
    FLUKE_NATIVE_FUNCTIONS(X)
#undef X
} L;

struct Failed {};  // a Python error is set

const at::Tensor &tensor(PyObject *o) {
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "fluke_b200.ops needs torch tensors, got %s", Py_TYPE(o)->tp_name);
        throw Failed();
    }
    return THPVariable_Unpack(o);
}
// An input: on the GPU and contiguous, or None.
const at::Tensor *input(PyObject *o) {
    if (o == Py_None) return nullptr;
    const at::Tensor &t = tensor(o);
    if (!t.is_cuda()) {
        PyErr_SetString(PyExc_RuntimeError, "fluke_b200.ops needs CUDA tensors (there is no CPU fallback)");
        throw Failed();
    }
    if (!t.is_contiguous()) {
        PyErr_SetString(PyExc_RuntimeError, "fluke_b200.ops needs contiguous tensors");
        throw Failed();
    }
    return &t;
}
const at::Tensor &required(PyObject *o) {
    const at::Tensor *t = input(o);
    if (!t) tensor(o);  // raises
    return *t;
}
// The same with the dimensions that the operator's sizes are read from.
const at::Tensor &required(PyObject *o, int64_t dims) {
    const at::Tensor &t = required(o);
    if (t.dim() != dims) {
        PyErr_Format(PyExc_ValueError, "fluke_b200.ops: a tensor of %lld dimensions where %lld are needed", (long long)t.dim(), (long long)dims);
        throw Failed();
    }
    return t;
}
void *ptr(const at::Tensor *t) { return t ? t->data_ptr() : nullptr; }
void *ptr(const at::Tensor &t) { return t.data_ptr(); }
// Numbers and addresses are taken as ctypes takes them for the same C arguments: an int of any size
// by its low bits (the stride of a dimension of one element may be anything), a ctypes integer by its value,
// an address also as a ctypes pointer or array; a real number as float() converts it.
int integer(PyObject *o) {
    if (PyLong_Check(o)) return int(PyLong_AsUnsignedLongMask(o));
    PyObject *v = PyIndex_Check(o) ? PyNumber_Index(o) : PyObject_GetAttrString(o, "value");
    if (!v || !PyLong_Check(v)) {
        Py_XDECREF(v);
        PyErr_Format(PyExc_TypeError, "fluke_b200.ops: an integer is needed, got %s", Py_TYPE(o)->tp_name);
        throw Failed();
    }
    const int r = int(PyLong_AsUnsignedLongMask(v));
    Py_DECREF(v);
    return r;
}
void *address(PyObject *o) {
    if (o == Py_None) return nullptr;
    if (PyLong_Check(o)) return reinterpret_cast<void *>(uintptr_t(PyLong_AsUnsignedLongLongMask(o)));
    PyObject *ctypes = PyImport_ImportModule("ctypes");
    PyObject *type = ctypes ? PyObject_GetAttrString(ctypes, "c_void_p") : nullptr;
    PyObject *cast = type ? PyObject_CallMethod(ctypes, "cast", "OO", o, type) : nullptr;
    PyObject *v = cast ? PyObject_GetAttrString(cast, "value") : nullptr;
    void *p = v && v != Py_None ? PyLong_AsVoidPtr(v) : nullptr;
    const bool ok = v && !PyErr_Occurred();
    Py_XDECREF(v);
    Py_XDECREF(cast);
    Py_XDECREF(type);
    Py_XDECREF(ctypes);
    if (!ok) throw Failed();
    return p;
}
float real(PyObject *o) {
    if (PyFloat_Check(o)) return float(PyFloat_AS_DOUBLE(o));
    PyObject *v = PyNumber_Float(o);
    if (!v) throw Failed();
    const double r = PyFloat_AS_DOUBLE(v);
    Py_DECREF(v);
    return float(r);
}
bool truth(PyObject *o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw Failed();
    return v != 0;
}

// A new tensor on `like`'s device. On the current device (nearly always) without the device guard and the
// initialisation check of at::detail::empty_cuda: 0.40 instead of 0.53 us.
at::Tensor empty_on(const at::Tensor &like, at::IntArrayRef size, at::ScalarType type) {
    const at::Device device = like.device();
    if (device.index() != c10::cuda::current_device()) return at::detail::empty_cuda(size, type, device, c10::nullopt);
    return at::detail::empty_generic(size, c10::cuda::CUDACachingAllocator::get(), c10::DispatchKeySet(c10::DispatchKey::CUDA), type,
                                     c10::nullopt);
}
// `o` as the output tensor, or a new one when it is None.
at::Tensor output(PyObject *o, const at::Tensor &like, at::IntArrayRef size, at::ScalarType type) {
    return o == Py_None ? empty_on(like, size, type) : tensor(o);
}

template <typename F>
auto unlocked(F f) {
    struct Release {
        PyThreadState *s = PyEval_SaveThread();
        ~Release() { PyEval_RestoreThread(s); }
    } r;
    return f();
}
void check(int rc, const char *what) {
    if (rc == 0) return;
    PyErr_SetString(PyExc_RuntimeError, (std::string(what) + " failed: rc=" + std::to_string(rc) + " " + L.fluke_last_error()).c_str());
    throw Failed();
}

PyObject *wrap(const at::Tensor &t) { return THPVariable_Wrap(t); }
PyObject *wrap(const at::Tensor &a, const at::Tensor &b) {
    PyObject *x = wrap(a), *y = wrap(b), *r = x && y ? PyTuple_Pack(2, x, y) : nullptr;
    Py_XDECREF(x);
    Py_XDECREF(y);
    return r;
}

using Args = PyObject *const *;

// Turns C++ errors into Python ones and checks the argument count.
template <PyObject *(*F)(Args), int N>
PyObject *entry(PyObject *, Args a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != N) {
        PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
        return nullptr;
    }
    if (!L.fluke_last_error) {
        PyErr_SetString(PyExc_RuntimeError, "fluke_b200._native: no library bound");
        return nullptr;
    }
    try {
        return F(a);
    } catch (const Failed &) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

// ---- memory-bound kernels ------------------------------------------------------------------------

// x, residual, weight, alpha, eps, out
PyObject *rmsnorm(Args a) {
    const at::Tensor &x = required(a[0]);
    const at::Tensor *res = input(a[1]), *w = input(a[2]);
    const float alpha = real(a[3]), eps = real(a[4]);
    at::Tensor out = output(a[5], x, x.sizes(), x.scalar_type());
    unlocked([&] { L.fluke_rmsnorm_gpu(ptr(x), ptr(res), ptr(w), ptr(out), int(x.size(0)), int(x.size(1)), alpha, eps); });
    return wrap(out);
}

// x, weight, residual, residual_scale, alpha, eps, fp8
PyObject *rmsnorm_quant(Args a) {
    const at::Tensor &x = required(a[0]);
    const at::Tensor *w = input(a[1]), *res = input(a[2]), *scale = input(a[3]);
    const float alpha = real(a[4]), eps = real(a[5]);
    auto fn = truth(a[6]) ? L.fluke_rmsnorm_quant_fp8_gpu : L.fluke_rmsnorm_quant_int8_gpu;
    unlocked([&] { fn(ptr(x), ptr(w), ptr(res), ptr(scale), int(x.size(0)), int(x.size(1)), alpha, eps); });
    return PyTuple_Pack(2, a[2], a[3]);
}

// x, out, scale, fp8
PyObject *quant(Args a) {
    const at::Tensor &x = required(a[0]);
    const bool fp8 = truth(a[3]);
    at::Tensor out = output(a[1], x, x.sizes(), fp8 ? at::kByte : at::kChar);
    at::Tensor scale = output(a[2], x, {x.size(0)}, at::kFloat);
    auto fn = fp8 ? L.fluke_quant_fp8_gpu : L.fluke_quant_int8_gpu;
    unlocked([&] { fn(ptr(x), ptr(out), ptr(scale), int(x.size(0)), int(x.size(1))); });
    return wrap(out, scale);
}

// x, scale, fp8
PyObject *dequant_transpose(Args a) {
    const at::Tensor &x = required(a[0], 3);
    const float scale = real(a[1]);
    auto fn = truth(a[2]) ? L.fluke_dequant_fp8_transpose_gpu : L.fluke_dequant_int8_transpose_gpu;
    const int64_t t = x.size(0), n = x.size(1), c = x.size(2);
    at::Tensor out = empty_on(x, {n, t, c}, at::kHalf);
    unlocked([&] { fn(ptr(x), ptr(out), int(t), int(n), int(c), scale); });
    return wrap(out);
}

// x address, sin, cos, batch, seq_len, heads, head_dim, width, stride_batch, stride_seq, stride_head
PyObject *rotary_emb(Args a) {
    void *x = address(a[0]);
    const at::Tensor *sin = input(a[1]), *cos = input(a[2]);
    int v[8];
    for (int i = 0; i < 8; ++i) v[i] = integer(a[3 + i]);
    unlocked([&] { L.fluke_rotary_emb_gpu(x, ptr(sin), ptr(cos), v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]); });
    Py_RETURN_NONE;
}

// qkv, sin, cos, width
PyObject *rotary_qkv(Args a) {
    const at::Tensor &qkv = required(a[0], 5);
    const at::Tensor *sin = input(a[1]), *cos = input(a[2]);
    const int width = integer(a[3]);
    // The q and k heads lie side by side: one call rotates both. The strides follow from the sizes: those of
    // a contiguous tensor say nothing in a dimension of one element, and with one head q and k are two.
    const int64_t heads = qkv.size(3), head_dim = qkv.size(4), position = qkv.size(2) * heads * head_dim;
    unlocked([&] {
        L.fluke_rotary_emb_gpu(ptr(qkv), ptr(sin), ptr(cos), int(qkv.size(0)), int(qkv.size(1)), 2 * int(heads), int(head_dim),
                               width, int(qkv.size(1) * position), int(position), int(head_dim));
    });
    Py_INCREF(a[0]);
    return a[0];
}

// x
PyObject *silu_mul(Args a) {
    const at::Tensor &x = required(a[0]);
    const int64_t m = x.size(0), h = x.size(1) / 2;
    at::Tensor out = empty_on(x, {m, h}, x.scalar_type());
    unlocked([&] { L.fluke_silu_mul_gpu(ptr(x), ptr(out), int(m), int(h)); });
    return wrap(out);
}

// scratch, ih_t, cell, hh_next
PyObject *flstm_step(Args a) {
    const at::Tensor *scratch = input(a[0]), *ih = input(a[1]);
    const at::Tensor &cell = required(a[2]);
    at::Tensor out = output(a[3], cell, cell.sizes(), cell.scalar_type());
    unlocked([&] { L.fluke_flstm_step_gpu(ptr(scratch), ptr(ih), ptr(cell), ptr(out), int(cell.size(0)), int(cell.size(1))); });
    return wrap(out);
}

// ---- fused transformer kernels -------------------------------------------------------------------

// backend, a, w, scale_a, scale_b, sin, cos, seqlen, out, kind (0 int8, 1 fp8 pre-shuffled, 2 fp8 row-major), columns
PyObject *qkv_rotary(Args a) {
    void *backend = address(a[0]);
    const at::Tensor &x = required(a[1]);
    const at::Tensor *w = input(a[2]), *sa = input(a[3]), *sb = input(a[4]), *sin = input(a[5]), *cos = input(a[6]);
    const int seqlen = integer(a[7]), kind = integer(a[9]), m = int(x.size(0));
    at::Tensor out = output(a[8], x, {m, integer(a[10])}, at::kHalf);
    check(unlocked([&] {
              if (kind == 0)
                  return L.fluke_qkv_rotary_i8_gpu(static_cast<const fluke_int8_backend_t *>(backend), ptr(out), ptr(x), ptr(w),
                                                   ptr(sa), ptr(sb), ptr(sin), ptr(cos), m, seqlen);
              auto fn = kind == 1 ? L.fluke_qkv_rotary_fp8_gpu : L.fluke_qkv_rotary_fp8_plain_gpu;
              return fn(static_cast<const fluke_fp8_backend_t *>(backend), ptr(out), ptr(x), ptr(w), ptr(sa), ptr(sb), ptr(sin),
                        ptr(cos), m, seqlen);
          }),
          kind == 0 ? "fluke_qkv_rotary_i8_gpu" : "fluke_qkv_rotary_fp8_gpu");
    return wrap(out);
}

// backend, a, gate, up, scale_a, scale_gate, scale_up, out, kind (as above), columns
PyObject *gated_mlp(Args a) {
    void *backend = address(a[0]);
    const at::Tensor &x = required(a[1]);
    const at::Tensor *gate = input(a[2]), *up = input(a[3]), *sa = input(a[4]), *sg = input(a[5]), *su = input(a[6]);
    const int kind = integer(a[8]), m = int(x.size(0));
    at::Tensor out = output(a[7], x, {m, integer(a[9])}, at::kHalf);
    check(unlocked([&] {
              if (kind == 0)
                  return L.fluke_gated_mlp_i8_gpu(static_cast<const fluke_int8_backend_t *>(backend), ptr(out), ptr(x), ptr(gate),
                                                  ptr(up), ptr(sa), ptr(sg), ptr(su), m);
              auto fn = kind == 1 ? L.fluke_gated_mlp_fp8_gpu : L.fluke_gated_mlp_fp8_plain_gpu;
              return fn(static_cast<const fluke_fp8_backend_t *>(backend), ptr(out), ptr(x), ptr(gate), ptr(up), ptr(sa), ptr(sg),
                        ptr(su), m);
          }),
          kind == 0 ? "fluke_gated_mlp_i8_gpu" : "fluke_gated_mlp_fp8_gpu");
    return wrap(out);
}

// ---- plain GEMMs and the LSTM step ---------------------------------------------------------------

// a, b, scale_a, scale_b, const_scale_a
PyObject *gemm_i8(Args a) {
    const at::Tensor &x = required(a[0], 2), &w = required(a[1]);
    const at::Tensor *sa = input(a[2]), *sb = input(a[3]);
    const float csa = real(a[4]);
    const int m = int(x.size(0)), k = int(x.size(1)), n = int(w.size(0));
    at::Tensor out = empty_on(x, {m, n}, at::kHalf);
    check(unlocked([&] { return L.fluke_gemm_i8_gpu(ptr(out), ptr(x), ptr(w), ptr(sa), csa, ptr(sb), m, n, k); }), "fluke_gemm_i8_gpu");
    return wrap(out);
}

// a, b, scale_a, scale_b
PyObject *gemm_fp8(Args a) {
    const at::Tensor &x = required(a[0], 2), &w = required(a[1]);
    const at::Tensor *sa = input(a[2]), *sb = input(a[3]);
    const int m = int(x.size(0)), k = int(x.size(1)), n = int(w.size(0));
    at::Tensor out = empty_on(x, {m, n}, at::kHalf);
    check(unlocked([&] { return L.fluke_gemm_fp8_gpu(ptr(out), ptr(x), ptr(w), ptr(sa), ptr(sb), m, n, k); }), "fluke_gemm_fp8_gpu");
    return wrap(out);
}

// a, w, scale_a, scale_b, out, fp8
PyObject *down_proj(Args a) {
    const at::Tensor &x = required(a[0], 2), &w = required(a[1]);
    const at::Tensor *sa = input(a[2]), *sb = input(a[3]);
    const bool fp8 = truth(a[5]);
    const int m = int(x.size(0)), k = int(x.size(1)), n = int(w.size(0));
    at::Tensor out = output(a[4], x, {m, n}, at::kHalf);
    const int ld = int(out.stride(0));
    auto fn = fp8 ? L.fluke_down_proj_fp8_gpu : L.fluke_down_proj_i8_gpu;
    check(unlocked([&] { return fn(ptr(out), ld, ptr(x), ptr(w), ptr(sa), ptr(sb), m, n, k); }),
          fp8 ? "fluke_down_proj_fp8_gpu" : "fluke_down_proj_i8_gpu");
    return wrap(out);
}

// A, W4, bias4, c, h_out, fp8_export_name
PyObject *lstm_step(Args a) {
    const at::Tensor &x = required(a[0], 2), &w4 = required(a[1]), &b4 = required(a[2]), &c = required(a[3]);
    const int b = int(x.size(0)), kc = int(x.size(1)), h = int(c.size(1));
    at::Tensor out = output(a[4], x, {b, h}, at::kChar);
    const char *w = static_cast<const char *>(ptr(w4));
    const float *bias = static_cast<const float *>(ptr(b4));
    const size_t ws = size_t(h) * kc * 2;
    auto fn = truth(a[5]) ? L.fluke_factored_lstm_step_fp8_gpu : L.fluke_factored_lstm_step_i8_gpu;
    check(unlocked([&] {
              return fn(ptr(x), w, w + ws, w + 2 * ws, w + 3 * ws, bias, bias + h, bias + 2 * h, bias + 3 * h, ptr(c), ptr(out), b, h, kc);
          }),
          "fluke_factored_lstm_step_i8_gpu");
    return wrap(out);
}

// {name: address} of the loaded library's entry points
PyObject *bind(PyObject *, PyObject *dict) {
    Entry e;
    if (!PyDict_Check(dict)) return PyErr_Format(PyExc_TypeError, "bind() takes a dict of addresses");
#define X(name)                                                                                     \
    {                                                                                               \
        PyObject *v = PyDict_GetItemString(dict, #name);                                            \
        void *p = v ? PyLong_AsVoidPtr(v) : nullptr;                                                \
        if (!p) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_KeyError, "%s", #name);      \
        e.name = reinterpret_cast<decltype(e.name)>(p);                                             \
    }
    FLUKE_NATIVE_FUNCTIONS(X)
#undef X
    L = e;
    Py_RETURN_NONE;
}

PyObject *names(PyObject *, PyObject *) {
    PyObject *list = PyList_New(0);
#define X(name)                                         \
    if (list) {                                         \
        PyObject *s = PyUnicode_FromString(#name);      \
        if (s) PyList_Append(list, s);                  \
        Py_XDECREF(s);                                  \
    }
    FLUKE_NATIVE_FUNCTIONS(X)
#undef X
    return list;
}

#define FAST(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entry<name, n>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", bind, METH_O, nullptr}, {"names", names, METH_NOARGS, nullptr},
    FAST(rmsnorm, 6), FAST(rmsnorm_quant, 7), FAST(quant, 4), FAST(dequant_transpose, 3), FAST(rotary_emb, 11), FAST(rotary_qkv, 4),
    FAST(silu_mul, 1), FAST(flstm_step, 4), FAST(qkv_rotary, 11), FAST(gated_mlp, 10), FAST(gemm_i8, 5), FAST(gemm_fp8, 4),
    FAST(down_proj, 6), FAST(lstm_step, 6), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject *PyInit__native() { return PyModule_Create(&module); }
