// The operators' calls as Python makes them, in native code: tensors in, tensor out, one call of the C ABI between them. A call of a small
// operator is bound by the host, and in Python its checks, its result's allocation and the ctypes call were most of it (classifier
// head, four operators on 32 images: 30.9 us for 13 of device time, 18.4 so).
//
// Every function here takes the ordinary call and nothing else: plain CUDA tensors of the right type, contiguous, in an ordinary state of
// the dispatcher. It returns the result, or None for whatever is not ordinary (ops.py then does the same step by step, with its errors),
// or the library's error code (which ops.py raises). Nothing is kept between calls but the addresses of the library's functions.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstring>

#include "kxc_b200.h"

namespace {

using Entry = int32_t (*)(void**, const void*, void*);           // (packed_args, descriptor, stream)
using CountEntry = int32_t (*)(void**, int64_t, void*);          // nn_relu, nn_flatten
using GapEntry = int32_t (*)(void**, int32_t, int32_t, int32_t, int32_t, void*);
using PlanEntry = int32_t (*)(void*, void**, void*);

struct {
    Entry conv2d, conv2d_s8, max_pool, avg_pool, chain, softmax, gemm;
    CountEntry relu, flatten;
    GapEntry gap;
    PlanEntry plan_run;
} lib = {};

// The dispatcher does nothing but run kernels: no modes, no transforms, no tracing.
bool ordinary_state() {
    static constexpr c10::DispatchKeySet special{c10::DispatchKey::Python,          c10::DispatchKey::PythonTLSSnapshot,
                                                 c10::DispatchKey::Functionalize,   c10::DispatchKey::FuncTorchDynamicLayerFrontMode,
                                                 c10::DispatchKey::FuncTorchVmapMode, c10::DispatchKey::Tracer, c10::DispatchKey::PreDispatch};
    return !c10::impl::tls_local_dispatch_key_set().included_.has_any(special) && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
           !at::impl::torch_function_mode_enabled();
}
// A plain tensor on a GPU (no subclass, wrapper or lazy view), of `type`, dense and in order; `rank` < 0: any.
const at::Tensor* plain(PyObject* o, at::ScalarType type, int rank) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    static constexpr c10::DispatchKeySet special{c10::DispatchKey::Python,       c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::Functionalize,
                                                 c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched,
                                                 c10::DispatchKey::Conjugate,    c10::DispatchKey::Negative,          c10::DispatchKey::ZeroTensor};
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.scalar_type() != type || t.key_set().has_any(special)) return nullptr;
    if (!t.unsafeGetTensorImpl()->has_storage() || (rank >= 0 && t.dim() != rank) || !t.is_contiguous() || t.numel() == 0) return nullptr;
    return &t;
}
void* address(const at::Tensor& t) { return const_cast<void*>(t.const_data_ptr()); }
void* result_address(const at::Tensor& t) { return t.mutable_data_ptr(); }  // (memory shared with a lazy clone becomes its own first)

// `n` plain whole numbers of a tuple or list.
bool numbers(PyObject* o, int n, int32_t* out) {
    const bool tuple = PyTuple_CheckExact(o);
    if ((!tuple && !PyList_CheckExact(o)) || Py_SIZE(o) != n) return false;
    for (int i = 0; i < n; ++i) {
        PyObject* e = tuple ? PyTuple_GET_ITEM(o, i) : PyList_GET_ITEM(o, i);
        if (!PyLong_CheckExact(e)) return false;
        int overflow = 0;
        const long v = PyLong_AsLongAndOverflow(e, &overflow);
        if (overflow != 0 || v < 0 || v > (1 << 24)) return false;
        out[i] = (int32_t)v;
    }
    return true;
}
bool flag(PyObject* o, bool* out) {
    *out = o == Py_True;
    return PyBool_Check(o);
}
bool small(const at::Tensor& t) {  // (the descriptors' extents have 32 bits)
    for (const int64_t d : t.sizes())
        if (d > INT32_MAX) return false;
    return true;
}

template <typename F>
PyObject* call(const at::Tensor& on, const at::Tensor& result, F&& f) {
    int32_t rc;
    void* stream = c10::cuda::getCurrentCUDAStream(on.get_device()).stream();
    Py_BEGIN_ALLOW_THREADS
    rc = f(stream);
    Py_END_ALLOW_THREADS
    return rc == 0 ? THPVariable_Wrap(result) : PyLong_FromLong(rc);
}

// (data, weight, bias or None, strides, padding, dilation, residual or None, relu, precision, out or None)
PyObject* conv2d(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 10 || !ordinary_state()) Py_RETURN_NONE;
    const at::Tensor *x = plain(a[0], at::kFloat, 4), *w = plain(a[1], at::kFloat, 4);
    int32_t s[2], p[2], d[2];
    if (x == nullptr || w == nullptr || !small(*x) || !small(*w) || !numbers(a[3], 2, s) || !numbers(a[4], 2, p) || !numbers(a[5], 2, d)) Py_RETURN_NONE;
    if (!PyLong_CheckExact(a[8]) || w->size(1) != x->size(1) || s[0] < 1 || s[1] < 1 || d[0] < 1 || d[1] < 1) Py_RETURN_NONE;
    const int64_t oh = (x->size(2) + 2 * p[0] - ((w->size(2) - 1) * d[0] + 1)) / s[0] + 1, ow = (x->size(3) + 2 * p[1] - ((w->size(3) - 1) * d[1] + 1)) / s[1] + 1;
    if (x->size(2) + 2 * p[0] < (w->size(2) - 1) * d[0] + 1 || x->size(3) + 2 * p[1] < (w->size(3) - 1) * d[1] + 1) Py_RETURN_NONE;
    const int64_t dims[4] = {x->size(0), w->size(0), oh, ow};
    void* ptrs[5] = {address(*x), address(*w)};
    bool relu;
    if (!flag(a[7], &relu)) Py_RETURN_NONE;
    int at = 2, flags = relu ? KXC_B200_RELU : 0;
    if (a[2] != Py_None) {
        const at::Tensor* b = plain(a[2], at::kFloat, 1);
        if (b == nullptr || b->size(0) != dims[1]) Py_RETURN_NONE;
        ptrs[at++] = address(*b);
        flags |= KXC_B200_BIAS;
    }
    if (a[6] != Py_None) {
        const at::Tensor* r = plain(a[6], at::kFloat, 4);
        if (r == nullptr || r->sizes() != at::IntArrayRef(dims, 4)) Py_RETURN_NONE;
        ptrs[at++] = address(*r);
        flags |= KXC_B200_RESIDUAL;
    }
    at::Tensor out;
    if (a[9] != Py_None) {
        const at::Tensor* o = plain(a[9], at::kFloat, -1);
        if (o == nullptr) Py_RETURN_NONE;
        out = *o;
    } else {
        out = at::empty(at::IntArrayRef(dims, 4), x->options().requires_grad(false));
    }
    ptrs[at] = result_address(out);
    const kxc_b200_conv2d_desc desc = {(int32_t)x->size(0), (int32_t)x->size(1), (int32_t)x->size(2), (int32_t)x->size(3), (int32_t)w->size(0),
                                       (int32_t)w->size(2), (int32_t)w->size(3), s[0], s[1], p[0], p[1], d[0], d[1], flags, (int32_t)PyLong_AsLong(a[8])};
    return call(*x, out, [&](void* stream) { return lib.conv2d(ptrs, &desc, stream); });
    END_HANDLE_TH_ERRORS
}

// (data, weight, bias, multiplier, shift, strides, padding, dilation, relu, simt, nhwc)
PyObject* conv2d_s8(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 11 || !ordinary_state()) Py_RETURN_NONE;
    const at::Tensor *x = plain(a[0], at::kChar, 4), *w = plain(a[1], at::kChar, 4), *q[3];
    for (int i = 0; i < 3; ++i)
        if ((q[i] = plain(a[2 + i], at::kInt, -1)) == nullptr) Py_RETURN_NONE;
    int32_t s[2], p[2], d[2];
    if (x == nullptr || w == nullptr || !small(*x) || !small(*w) || !numbers(a[5], 2, s) || !numbers(a[6], 2, p) || !numbers(a[7], 2, d)) Py_RETURN_NONE;
    if (s[0] < 1 || s[1] < 1 || d[0] < 1 || d[1] < 1) Py_RETURN_NONE;
    bool relu, simt, nhwc;
    if (!flag(a[8], &relu) || !flag(a[9], &simt) || !flag(a[10], &nhwc)) Py_RETURN_NONE;
    const int H = nhwc ? 1 : 2, C = nhwc ? 3 : 1;  // (of both tensors)
    const int64_t h = x->size(H), wd = x->size(H + 1), kh = w->size(H), kw = w->size(H + 1), o = w->size(0);
    if (h + 2 * p[0] < (kh - 1) * d[0] + 1 || wd + 2 * p[1] < (kw - 1) * d[1] + 1) Py_RETURN_NONE;
    const int64_t oh = (h + 2 * p[0] - ((kh - 1) * d[0] + 1)) / s[0] + 1, ow = (wd + 2 * p[1] - ((kw - 1) * d[1] + 1)) / s[1] + 1;
    const int64_t dims[4] = {x->size(0), nhwc ? oh : o, nhwc ? ow : oh, nhwc ? o : ow};
    const at::Tensor out = at::empty(at::IntArrayRef(dims, 4), x->options().requires_grad(false));
    void* ptrs[6] = {address(*x), address(*w), address(*q[0]), address(*q[1]), address(*q[2]), result_address(out)};
    const int32_t flags = KXC_B200_BIAS | (relu ? KXC_B200_RELU : 0) | (nhwc ? KXC_B200_NHWC : 0);
    const kxc_b200_conv2d_desc desc = {(int32_t)x->size(0), (int32_t)x->size(C), (int32_t)h, (int32_t)wd, (int32_t)o, (int32_t)kh, (int32_t)kw, s[0], s[1], p[0], p[1],
                                       d[0], d[1], flags, simt ? KXC_B200_PREC_SIMT : KXC_B200_PREC_FP32};
    return call(*x, out, [&](void* stream) { return lib.conv2d_s8(ptrs, &desc, stream); });
    END_HANDLE_TH_ERRORS
}

// (x, residual or None, pool_size, strides, padding, ceil_mode, out or None)
PyObject* pool(Entry entry, PyObject* const* a, Py_ssize_t n, bool chain) {
    HANDLE_TH_ERRORS
    if (n != 7 || !ordinary_state()) Py_RETURN_NONE;
    const at::Tensor* x = plain(a[0], at::kFloat, 4);
    int32_t k[2], s[2], p[4];
    if (x == nullptr || !small(*x) || !numbers(a[2], 2, k) || !numbers(a[3], 2, s) || !numbers(a[4], 4, p) || k[0] < 1 || k[1] < 1 || s[0] < 1 || s[1] < 1) Py_RETURN_NONE;
    bool ceil_mode;
    if (!flag(a[5], &ceil_mode)) Py_RETURN_NONE;
    const int64_t nh = x->size(2) + p[0] + p[2] - k[0], nw = x->size(3) + p[1] + p[3] - k[1];
    if (nh < 0 || nw < 0) Py_RETURN_NONE;
    const int64_t dims[4] = {x->size(0), x->size(1), (ceil_mode ? (nh + s[0] - 1) / s[0] : nh / s[0]) + 1, (ceil_mode ? (nw + s[1] - 1) / s[1] : nw / s[1]) + 1};
    void* ptrs[3] = {address(*x)};
    int at = 1;
    if (chain) {
        const at::Tensor* r = plain(a[1], at::kFloat, 4);
        if (r == nullptr || r->sizes() != at::IntArrayRef(dims, 4)) Py_RETURN_NONE;
        ptrs[at++] = address(*r);
    }
    at::Tensor out;
    if (a[6] != Py_None) {
        const at::Tensor* o = plain(a[6], at::kFloat, -1);
        if (o == nullptr) Py_RETURN_NONE;
        out = *o;
    } else {
        out = at::empty(at::IntArrayRef(dims, 4), x->options().requires_grad(false));
    }
    ptrs[at] = result_address(out);
    const kxc_b200_pool2d_desc desc = {(int32_t)x->size(0), (int32_t)x->size(1), (int32_t)x->size(2), (int32_t)x->size(3), k[0], k[1], s[0], s[1], p[0], p[1], p[2], p[3], ceil_mode ? 1 : 0};
    return call(*x, out, [&](void* stream) { return entry(ptrs, &desc, stream); });
    END_HANDLE_TH_ERRORS
}
PyObject* max_pool2d(PyObject*, PyObject* const* a, Py_ssize_t n) { return pool(lib.max_pool, a, n, false); }
PyObject* avg_pool2d(PyObject*, PyObject* const* a, Py_ssize_t n) { return pool(lib.avg_pool, a, n, false); }
PyObject* pool_add_relu(PyObject*, PyObject* const* a, Py_ssize_t n) { return pool(lib.chain, a, n, true); }

// (x)
PyObject* global_avg_pool2d(PyObject*, PyObject* o) {
    HANDLE_TH_ERRORS
    const at::Tensor* x = ordinary_state() ? plain(o, at::kFloat, 4) : nullptr;
    if (x == nullptr || !small(*x)) Py_RETURN_NONE;
    const int64_t dims[4] = {x->size(0), x->size(1), 1, 1};
    const at::Tensor out = at::empty(at::IntArrayRef(dims, 4), x->options().requires_grad(false));
    void* ptrs[2] = {address(*x), result_address(out)};
    return call(*x, out, [&](void* stream) {
        return lib.gap(ptrs, (int32_t)x->size(0), (int32_t)x->size(1), (int32_t)x->size(2), (int32_t)x->size(3), stream);
    });
    END_HANDLE_TH_ERRORS
}
PyObject* flatten(PyObject*, PyObject* o) {
    HANDLE_TH_ERRORS
    const at::Tensor* x = ordinary_state() ? plain(o, at::kFloat, -1) : nullptr;
    if (x == nullptr || x->dim() < 1) Py_RETURN_NONE;
    const int64_t dims[2] = {x->size(0), x->numel() / x->size(0)};
    const at::Tensor out = at::empty(at::IntArrayRef(dims, 2), x->options().requires_grad(false));
    void* ptrs[2] = {address(*x), result_address(out)};
    return call(*x, out, [&](void* stream) { return lib.flatten(ptrs, x->numel(), stream); });
    END_HANDLE_TH_ERRORS
}
PyObject* relu(PyObject*, PyObject* o) {
    HANDLE_TH_ERRORS
    const at::Tensor* x = ordinary_state() ? plain(o, at::kFloat, -1) : nullptr;
    if (x == nullptr) Py_RETURN_NONE;
    const at::Tensor out = at::empty(x->sizes(), x->options().requires_grad(false));
    void* ptrs[2] = {address(*x), result_address(out)};
    return call(*x, out, [&](void* stream) { return lib.relu(ptrs, x->numel(), stream); });
    END_HANDLE_TH_ERRORS
}
// (x, axis)
PyObject* softmax(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    const at::Tensor* x = n == 2 && ordinary_state() ? plain(a[0], at::kFloat, -1) : nullptr;
    int overflow = 0;
    const long axis = x != nullptr && PyLong_CheckExact(a[1]) ? PyLong_AsLongAndOverflow(a[1], &overflow) : 0;
    if (x == nullptr || x->dim() < 1 || x->dim() > 6 || !PyLong_CheckExact(a[1]) || overflow != 0 || axis < -64 || axis > 64) Py_RETURN_NONE;
    kxc_b200_softmax_desc desc = {};
    desc.rank = (int32_t)x->dim();
    for (int i = 0; i < desc.rank; ++i) desc.shape[i] = x->size(i);
    desc.axis = (int32_t)axis;
    const at::Tensor out = at::empty(x->sizes(), x->options().requires_grad(false));
    void* ptrs[2] = {address(*x), result_address(out)};
    return call(*x, out, [&](void* stream) { return lib.softmax(ptrs, &desc, stream); });
    END_HANDLE_TH_ERRORS
}
// (a, b, c or None, transB, precision): alpha = beta = 1
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 5 || !ordinary_state()) Py_RETURN_NONE;
    const at::Tensor *a = plain(args[0], at::kFloat, 2), *b = plain(args[1], at::kFloat, 2);
    if (a == nullptr || b == nullptr || !small(*a) || !small(*b) || !PyLong_CheckExact(args[4]) || !PyLong_Check(args[3])) Py_RETURN_NONE;
    const bool trans = PyObject_IsTrue(args[3]) == 1, has_c = args[2] != Py_None;
    if (b->size(trans ? 1 : 0) != a->size(1)) Py_RETURN_NONE;
    void* ptrs[4] = {address(*a), address(*b)};
    int at = 2;
    if (has_c) {
        const at::Tensor* c = plain(args[2], at::kFloat, -1);
        if (c == nullptr) Py_RETURN_NONE;
        ptrs[at++] = address(*c);
    }
    const int64_t dims[2] = {a->size(0), b->size(trans ? 0 : 1)};
    const at::Tensor out = at::empty(at::IntArrayRef(dims, 2), a->options().requires_grad(false));
    ptrs[at] = result_address(out);
    const kxc_b200_gemm_desc desc = {(int32_t)dims[0], (int32_t)dims[1], (int32_t)a->size(1), 1.0f, 1.0f, 0, trans ? 1 : 0, has_c ? 1 : 0, (int32_t)PyLong_AsLong(args[4])};
    return call(*a, out, [&](void* stream) { return lib.gemm(ptrs, &desc, stream); });
    END_HANDLE_TH_ERRORS
}

// (plan handle, addresses of the constants as bytes, input tensors as a tuple, out): the packed argument list inputs, constants, output
PyObject* plan_run(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    constexpr int kMost = 512;
    if (n != 4 || !PyBytes_CheckExact(a[1]) || !PyTuple_CheckExact(a[2]) || !ordinary_state()) Py_RETURN_NONE;
    const Py_ssize_t inputs = PyTuple_GET_SIZE(a[2]), constants = PyBytes_GET_SIZE(a[1]) / (Py_ssize_t)sizeof(void*);
    const at::Tensor* out = plain(a[3], at::kFloat, -1);
    if (out == nullptr || inputs < 1 || inputs + constants + 1 > kMost) Py_RETURN_NONE;
    void* args[kMost];
    const at::Tensor* first = nullptr;
    for (Py_ssize_t i = 0; i < inputs; ++i) {
        const at::Tensor* t = plain(PyTuple_GET_ITEM(a[2], i), at::kFloat, -1);
        if (t == nullptr) Py_RETURN_NONE;
        if (i == 0) first = t;
        args[i] = address(*t);
    }
    memcpy(args + inputs, PyBytes_AS_STRING(a[1]), (size_t)constants * sizeof(void*));
    args[inputs + constants] = result_address(*out);
    void* handle = PyLong_Check(a[0]) ? PyLong_AsVoidPtr(a[0]) : nullptr;
    if (handle == nullptr) {
        PyErr_Clear();
        Py_RETURN_NONE;
    }
    int32_t rc;
    void* stream = c10::cuda::getCurrentCUDAStream(first->get_device()).stream();
    Py_BEGIN_ALLOW_THREADS
    rc = lib.plan_run(handle, args, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

// (addresses of the library's functions, in the order of `lib`)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void* f[11];
    if (n != 11) {
        PyErr_SetString(PyExc_TypeError, "bind: eleven addresses");
        return nullptr;
    }
    for (int i = 0; i < 11; ++i)
        if ((f[i] = PyLong_AsVoidPtr(a[i])) == nullptr) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: null address");
            return nullptr;
        }
    Entry* entries[7] = {&lib.conv2d, &lib.conv2d_s8, &lib.max_pool, &lib.avg_pool, &lib.chain, &lib.softmax, &lib.gemm};
    for (int i = 0; i < 7; ++i) *entries[i] = reinterpret_cast<Entry>(f[i]);
    lib.relu = reinterpret_cast<CountEntry>(f[7]);
    lib.flatten = reinterpret_cast<CountEntry>(f[8]);
    lib.gap = reinterpret_cast<GapEntry>(f[9]);
    lib.plan_run = reinterpret_cast<PlanEntry>(f[10]);
    Py_RETURN_NONE;
}

template <typename F>
PyCFunction fast(F f) {
    return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}
PyMethodDef methods[] = {{"bind", fast(bind), METH_FASTCALL, nullptr},
                         {"conv2d", fast(conv2d), METH_FASTCALL, nullptr},
                         {"conv2d_s8", fast(conv2d_s8), METH_FASTCALL, nullptr},
                         {"max_pool2d", fast(max_pool2d), METH_FASTCALL, nullptr},
                         {"avg_pool2d", fast(avg_pool2d), METH_FASTCALL, nullptr},
                         {"pool_add_relu", fast(pool_add_relu), METH_FASTCALL, nullptr},
                         {"global_avg_pool2d", global_avg_pool2d, METH_O, nullptr},
                         {"flatten", flatten, METH_O, nullptr},
                         {"relu", relu, METH_O, nullptr},
                         {"softmax", fast(softmax), METH_FASTCALL, nullptr},
                         {"gemm", fast(gemm), METH_FASTCALL, nullptr},
                         {"plan_run", fast(plan_run), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Operator calls in native code (ops.py, plan.py).", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    const char* here = Py_GetVersion();  // "3.12.3 (...": the binary interface is that of the first two numbers
    const size_t minor = strcspn(strchr(PY_VERSION, '.') + 1, ".") + (size_t)(strchr(PY_VERSION, '.') + 1 - PY_VERSION);
    if (strncmp(here, PY_VERSION, minor) != 0 || (here[minor] >= '0' && here[minor] <= '9')) {
        PyErr_Format(PyExc_ImportError, "built for Python " PY_VERSION ", not %.10s", here);
        return nullptr;
    }
    PyObject* m = PyModule_Create(&module);
    if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", KXC_TORCH_VERSION) != 0) Py_CLEAR(m);
    return m;
}
