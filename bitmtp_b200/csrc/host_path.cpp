// Host side of the two calls a program makes for single packed products, in one native function each: checks,
// output allocation and the call into libbitmtp_b200.so.
//
// A decode-width product is 2 to 10 us on the device, while the same steps written in Python (two dozen attribute reads,
// one to four allocations through the Python front end, a ctypes call per launch) took 10.5 us for
// t2g128_int8xint2_linear (1024 x 2048, one row: 4.1 us here) and 26 us for T2LinearKernel.forward.  Nothing is decided
// here that the Python code does not decide: a call that does not meet every condition returns None, and the Python path
// then serves it or raises its own error.
//
// Tensors are taken only where their data pointer is the plain answer: exact torch.Tensor / Parameter objects with dense
// CUDA storage, outside torch-function modes and transforms (tracing, vmap, forward-mode wrappers).
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <exception>

namespace {

typedef int (*QuantFn)(const void *, int, int, void *, void *, void *, void *, int, void *);
typedef int (*GemvFn)(const void *, const void *, void *, const void *, const void *, int, int, int, int, int, int, void *,
                      int, void *);
typedef int (*GemvPreparedFn)(const void *, const void *, const void *, void *, const void *, const void *, int, int, int,
                              int, int, int, void *);
typedef int (*GemmFn)(const void *, const void *, const void *, void *, const void *, const void *, int, int, int, int, int,
                      void *);

// Entry points of the library, set once by bind() before the first call.
QuantFn g_quant = nullptr;
GemvFn g_gemv = nullptr;
GemvPreparedFn g_gemv_prepared = nullptr;
GemmFn g_gemm = nullptr;

// The tensor behind `o` when its data pointer may be handed to a kernel, else null.  (Strided nested tensors are exact
// torch.Tensor objects too, without one size per dimension.)
const at::Tensor *plain_cuda(PyObject *o) {
    if (!THPVariable_CheckExact(o) && Py_TYPE(o) != reinterpret_cast<PyTypeObject *>(ParameterClass)) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.is_nested() || !t.has_storage()) return nullptr;
    constexpr c10::DispatchKeySet kWrapped({c10::DispatchKey::Python, c10::DispatchKey::Functionalize,
                                            c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                            c10::DispatchKey::Conjugate, c10::DispatchKey::Negative,
                                            c10::DispatchKey::ZeroTensor});
    if (t.key_set().has_any(kWrapped) || !t.is_contiguous()) return nullptr;
    return &t;
}

// The exception in flight as the Python error that torch's own calls raise for it (torch.OutOfMemoryError for an allocation
// that fails, an error that Python has already set as it is).
PyObject *raise_as_torch_does() {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
}

bool modes_active() {
    return at::impl::torch_function_mode_enabled() ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Python) ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

// An uninitialised bf16 tensor on `dev`.  The CUDA allocation behind at::empty is called by itself: the walk through the
// dispatcher is 0.25 of the 4.2 us of a call whose kernel takes 2.4 (1024 x 2048, one row: 4.14 to 4.54 us by process with it,
// 3.97 to 4.10 without; back to back the launches alone take 3.9).  A tracer wants to see the call.
at::Tensor empty_bf16(at::IntArrayRef shape, c10::Device dev) {
    if (c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Tracer))
        return at::empty(shape, at::TensorOptions().dtype(at::kBFloat16).device(dev));
    return at::Tensor(at::detail::empty_cuda(shape, at::kBFloat16, dev, std::nullopt));
}

PyObject *bind(PyObject *, PyObject *args) {
    unsigned long long f[4];
    if (!PyArg_ParseTuple(args, "KKKK", &f[0], &f[1], &f[2], &f[3])) return nullptr;
    g_quant = reinterpret_cast<QuantFn>(f[0]);
    g_gemv = reinterpret_cast<GemvFn>(f[1]);
    g_gemv_prepared = reinterpret_cast<GemvPreparedFn>(f[2]);
    g_gemm = reinterpret_cast<GemmFn>(f[3]);
    Py_RETURN_NONE;
}

// linear(a, b, s, ws): t2g128_int8xint2_linear without the registry check.
PyObject *linear(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 4 || g_gemv == nullptr || modes_active()) Py_RETURN_NONE;
    try {                                                  // sizes too: they throw for tensors without plain ones
        const at::Tensor *a = plain_cuda(args[0]), *b = plain_cuda(args[1]), *s = plain_cuda(args[2]), *ws = plain_cuda(args[3]);
        if (!a || !b || !s || !ws || (a->dim() != 2 && a->dim() != 3) || b->dim() != 2 || ws->dim() != 2 || s->dim() < 1)
            Py_RETURN_NONE;
        const int64_t k = a->size(-1), n = b->size(0);
        if (k < 128 || k % 128 || b->size(1) * 4 != k || n < 8 || n % 8 || k > INT32_MAX || n > INT32_MAX) Py_RETURN_NONE;
        const int64_t m = a->numel() / k;
        if (m < 1 || m > 32 || ws->size(0) != n || ws->size(1) != k / 128 || s->size(-1) != 1 || s->numel() != m) Py_RETURN_NONE;
        if (a->scalar_type() != at::kChar || b->scalar_type() != at::kChar || ws->scalar_type() != at::kBFloat16 ||
            s->scalar_type() != at::kFloat)
            Py_RETURN_NONE;
        const c10::Device dev = a->device();
        if (b->device() != dev || s->device() != dev || ws->device() != dev) Py_RETURN_NONE;
        const int64_t shape[3] = {a->size(0), a->dim() == 2 ? n : a->size(1), n};
        at::Tensor out = empty_bf16(at::IntArrayRef(shape, a->dim()), dev);
        void *stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
        const void *ap = a->const_data_ptr(), *bp = b->const_data_ptr(), *sp = s->const_data_ptr(), *wp = ws->const_data_ptr();
        void *op = out.mutable_data_ptr();
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = g_gemv(ap, bp, op, sp, wp, (int)m, (int)n, (int)k, (int)n, 0, 0, nullptr, 0, stream);
        Py_END_ALLOW_THREADS
        if (rc != 0) Py_RETURN_NONE;                       // the Python path reports it
        return THPVariable_Wrap(std::move(out));
    } catch (...) {
        return raise_as_torch_does();
    }
}

inline int64_t up16(int64_t v) { return (v + 15) & ~int64_t(15); }

// linear_rows(x, w, ws, route, wide_max): T2LinearKernel.forward on bf16 rows [..., K]; route(T, N, K) -> bool is
// ops.gemv_serves_rows, asked for 17 to 32 rows only.  The second launch may start under the first (it waits on the device
// for the rows' codes).
PyObject *linear_rows(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 5 || g_quant == nullptr || modes_active()) Py_RETURN_NONE;
    try {
        const at::Tensor *x = plain_cuda(args[0]), *w = plain_cuda(args[1]), *ws = plain_cuda(args[2]);
        if (!x || !w || !ws || x->dim() < 1 || w->dim() != 2 || ws->dim() != 2) Py_RETURN_NONE;
        const int64_t k = x->size(-1), n = w->size(0), wide_max = PyLong_AsLongLong(args[4]);
        if (k < 128 || k % 128 || w->size(1) * 4 != k || n < 8 || n % 8 || k > INT32_MAX || n > INT32_MAX) Py_RETURN_NONE;
        const int64_t t = x->numel() / k;
        if (t < 1 || t > wide_max || ws->size(0) != n || ws->size(1) != k / 128) Py_RETURN_NONE;
        if (x->scalar_type() != at::kBFloat16 || w->scalar_type() != at::kChar || ws->scalar_type() != at::kBFloat16)
            Py_RETURN_NONE;
        const c10::Device dev = x->device();
        const void *xp = x->const_data_ptr(), *bp = w->const_data_ptr(), *wp = ws->const_data_ptr();
        if (w->device() != dev || ws->device() != dev || (reinterpret_cast<uintptr_t>(wp) & 15)) Py_RETURN_NONE;
        bool gemv = t <= 16;
        if (t > 16 && t <= 32) {
            PyObject *r = PyObject_CallFunction(args[3], "LLL", (long long)t, (long long)n, (long long)k);
            if (r == nullptr) return nullptr;
            gemv = PyObject_IsTrue(r);
            Py_DECREF(r);
        }
        c10::DimVector shape(x->sizes());
        shape.back() = n;
        // codes, group sums and multipliers of the rows in one allocation
        const int64_t sums = up16(t * k), s = sums + up16(4 * t * (k / 128));
        at::Tensor tmp = at::empty({s + 4 * t}, x->options().dtype(at::kByte));
        at::Tensor out = at::empty(shape, x->options());
        void *stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
        char *q = static_cast<char *>(tmp.mutable_data_ptr());
        void *op = out.mutable_data_ptr();
        const int T = (int)t, N = (int)n, K = (int)k;
        int rc;
        Py_BEGIN_ALLOW_THREADS
        if (T <= 16 && K % 256) {
            rc = g_quant(xp, T, K, q, nullptr, nullptr, q + s, 0, stream);
            if (rc == 0) rc = g_gemv(q, bp, op, q + s, wp, T, N, K, N, 0, 0, nullptr, 1, stream);
        } else {
            rc = g_quant(xp, T, K, nullptr, q, q + sums, q + s, 0, stream);
            if (rc == 0)
                rc = gemv ? g_gemv_prepared(q, q + sums, bp, op, q + s, wp, T, N, K, N, 0, 1, stream)
                          : g_gemm(q, q + sums, bp, op, q + s, wp, T, N, K, N, 1, stream);
        }
        Py_END_ALLOW_THREADS
        if (rc != 0) Py_RETURN_NONE;                       // the Python path reports it
        return THPVariable_Wrap(std::move(out));
    } catch (...) {
        return raise_as_torch_does();
    }
}

PyMethodDef kMethods[] = {
    {"bind", bind, METH_VARARGS, "Addresses of the library's entry points."},
    {"linear", (PyCFunction)(void (*)(void))linear, METH_FASTCALL, "t2g128_int8xint2_linear, or None."},
    {"linear_rows", (PyCFunction)(void (*)(void))linear_rows, METH_FASTCALL, "T2LinearKernel.forward, or None."},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "Native host path of the packed products.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&kModule); }
