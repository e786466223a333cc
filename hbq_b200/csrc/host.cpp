// The library's hot entry points for torch tensors, as a CPython module (hbq_host): what a decode step calls tens of
// thousands of times a second.  A call through ctypes costs more than its kernel: building the argument objects, two
// trips through Python's allocator and torch.empty, the stream query -- 20 us of host time for a 3 us quantizer, 43 us
// for one linear layer (quantizer + product) whose kernels take 9 to 27 us; through this module 12 us for the layer.
//
// Each function takes the plain case -- exact torch.Tensor objects (or parameters) of ordinary dense CUDA storage,
// contiguous, of the dtypes and shapes the kernel reads -- and returns None for anything else: the caller then runs its
// general path, which also raises the errors.  A negative return code of the library comes back as an int.  The module
// does not load the library itself: bind() is given the entry points of the copy that the process uses.
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include "../../include/hbq_b200.h"

namespace {

// What this module was compiled for (build.py compares it with the process that is about to load it).
__attribute__((used)) const char built_for[] = HBQ_HOST_TAG;

decltype(&hbq_quantize) p_quantize = nullptr;
decltype(&hbq_gemm) p_gemm = nullptr;
decltype(&hbq_gemm_workspace_bytes) p_gemm_workspace_bytes = nullptr;
decltype(&hbq_gemm_w4) p_gemm_w4 = nullptr;

// The tensor behind `o` when it is a plain dense CUDA tensor: no Python subclass, no functorch wrapper, no fake or
// lazily conjugated / negated tensor (any of them brings a dispatch key of its own).
const at::Tensor* plain_cuda(PyObject* o)
{
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda()) return nullptr;
    const c10::DispatchKeySet ordinary = c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
                                         c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA) | c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView);
    if ((t.key_set().raw_repr() & ~ordinary.raw_repr()) != 0 || !t.has_storage() || !t.is_contiguous()) return nullptr;
    return &t;
}

bool to_i64(PyObject* o, int64_t* v)
{
    *v = PyLong_AsLongLong(o);
    return !(*v == -1 && PyErr_Occurred());
}

const hbq_format* to_format(PyObject* o)
{
    if (!PyBytes_CheckExact(o) || PyBytes_GET_SIZE(o) != (Py_ssize_t)sizeof(hbq_format)) {
        PyErr_SetString(PyExc_TypeError, "format must be the bytes of an hbq_format");
        return nullptr;
    }
    return reinterpret_cast<const hbq_format*>(PyBytes_AS_STRING(o));
}

// An optional fp16 vector of n elements beside `like`; false when it is something the general path has to convert.
bool plain_bias(PyObject* o, const at::Tensor& like, int64_t n, const void** p)
{
    *p = nullptr;
    if (o == Py_None) return true;
    const at::Tensor* b = plain_cuda(o);
    if (!b || b->scalar_type() != at::kHalf || b->numel() != n || b->device() != like.device()) return false;
    *p = b->data_ptr();
    return true;
}

// Library calls run without the interpreter lock, as through ctypes: a launch may wait for room in the launch queue.
template <class F>
int unlocked(F f)
{
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f();
    Py_END_ALLOW_THREADS
    return rc;
}

PyObject* result(int rc, const at::Tensor& t) { return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(t); }

// bind(quantize, gemm, gemm_workspace_bytes, gemm_w4): addresses of the library's entry points
PyObject* host_bind(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    int64_t a[4];
    if (n != 4) { PyErr_SetString(PyExc_TypeError, "bind takes four addresses"); return nullptr; }
    for (int i = 0; i < 4; ++i)
        if (!to_i64(args[i], &a[i])) return nullptr;
    p_quantize = reinterpret_cast<decltype(p_quantize)>(a[0]);
    p_gemm = reinterpret_cast<decltype(p_gemm)>(a[1]);
    p_gemm_workspace_bytes = reinterpret_cast<decltype(p_gemm_workspace_bytes)>(a[2]);
    p_gemm_w4 = reinterpret_cast<decltype(p_gemm_w4)>(a[3]);
    Py_RETURN_NONE;
}

// quantize(x, format, out_dtype): the fake-quantised tensor; out_dtype: -1 as x, 0 fp16, 1 bf16
PyObject* host_quantize(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    int64_t od;
    if (n != 3 || !to_i64(args[2], &od)) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "quantize(x, format, out_dtype)"); return nullptr; }
    const hbq_format* f = to_format(args[1]);
    if (!f) return nullptr;
    const at::Tensor* x = plain_cuda(args[0]);
    if (!x || x->dim() < 1 || x->numel() == 0 || (f->kind == HBQ_KIND_MXFP && f->per_tensor_scale)) Py_RETURN_NONE;
    const auto st = x->scalar_type();
    if (st != at::kHalf && st != at::kBFloat16) Py_RETURN_NONE;
    const int in = st == at::kHalf ? HBQ_DTYPE_F16 : HBQ_DTYPE_BF16, out = od < 0 ? in : (int)od;
    const c10::cuda::OptionalCUDAGuard guard(x->device());
    const at::Tensor deq = at::empty(x->sizes(), x->options().dtype(out == HBQ_DTYPE_F16 ? at::kHalf : at::kBFloat16));
    const int64_t K = x->size(-1), rows = x->numel() / K;
    const void* xp = x->data_ptr();
    void* dp = deq.data_ptr();
    void* stream = at::cuda::getCurrentCUDAStream(x->device().index()).stream();
    return result(unlocked([&] { return p_quantize(xp, in, rows, K, f, dp, out, nullptr, nullptr, stream); }), deq);
    END_HANDLE_TH_ERRORS
}

// gemm(a, b, mode, group_k, group_n, bias, b_is_nk): a [M, K] x b [N, K] or [K, N], fp16
PyObject* host_gemm(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    int64_t mode, gk, gn, nk;
    if (n != 7 || !to_i64(args[2], &mode) || !to_i64(args[3], &gk) || !to_i64(args[4], &gn) || !to_i64(args[6], &nk)) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "gemm(a, b, mode, group_k, group_n, bias, b_is_nk)");
        return nullptr;
    }
    const at::Tensor *a = plain_cuda(args[0]), *b = plain_cuda(args[1]);
    if (!a || !b || a->scalar_type() != at::kHalf || b->scalar_type() != at::kHalf || a->dim() != 2 || b->dim() != 2 ||
        a->device() != b->device())
        Py_RETURN_NONE;
    const int64_t M = a->size(0), K = a->size(1), N = b->size(nk ? 0 : 1);
    const void* bias;
    if (b->size(nk ? 1 : 0) != K || M == 0 || N == 0 || K == 0 || !plain_bias(args[5], *a, N, &bias)) Py_RETURN_NONE;
    const c10::cuda::OptionalCUDAGuard guard(a->device());
    const at::Tensor c = at::empty({M, N}, a->options());
    const int64_t wb = p_gemm_workspace_bytes(M, N, K, (int)nk, (int)mode, (int)gk, (int)gn);
    at::Tensor ws;
    if (wb > 0) ws = at::empty({wb}, a->options().dtype(at::kByte));
    const void *ap = a->data_ptr(), *bp = b->data_ptr();
    void *cp = c.data_ptr(), *wp = wb > 0 ? ws.data_ptr() : nullptr;
    void* stream = at::cuda::getCurrentCUDAStream(a->device().index()).stream();
    return result(unlocked([&] { return p_gemm(ap, bp, cp, M, N, K, (int)nk, (int)mode, (int)gk, (int)gn, bias, wp, wb, stream); }), c);
    END_HANDLE_TH_ERRORS
}

// gemm_w4(x, data, N, K, format, container_bits, bias, workspace): x [M, K] fp16 times a prepacked weight, into a new tensor
PyObject* host_gemm_w4(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    int64_t N, K, bits;
    if (n != 8 || !to_i64(args[2], &N) || !to_i64(args[3], &K) || !to_i64(args[5], &bits)) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "gemm_w4(x, data, N, K, format, container_bits, bias, workspace)");
        return nullptr;
    }
    const hbq_format* f = to_format(args[4]);
    if (!f) return nullptr;
    const at::Tensor *x = plain_cuda(args[0]), *d = plain_cuda(args[1]), *ws = plain_cuda(args[7]);
    const void* bias;
    if (!x || !d || !ws || x->scalar_type() != at::kHalf || x->dim() != 2 || x->size(1) != K || x->size(0) == 0 ||
        x->device() != d->device() || ws->device() != d->device() || !plain_bias(args[6], *x, N, &bias))
        Py_RETURN_NONE;
    const int64_t M = x->size(0);
    const c10::cuda::OptionalCUDAGuard guard(x->device());
    const at::Tensor c = at::empty({M, N}, x->options());
    const void *xp = x->data_ptr(), *dp = d->data_ptr();
    void *cp = c.data_ptr(), *wp = ws->data_ptr();
    const int64_t wb = ws->numel();
    void* stream = at::cuda::getCurrentCUDAStream(x->device().index()).stream();
    return result(unlocked([&] { return p_gemm_w4(xp, dp, cp, M, N, K, f, (int)bits, bias, wp, wb, stream); }), c);
    END_HANDLE_TH_ERRORS
}

// current_stream(device_index): the handle of torch's current stream there
PyObject* host_current_stream(PyObject*, PyObject* o)
{
    HANDLE_TH_ERRORS
    int64_t i;
    if (!to_i64(o, &i)) return nullptr;
    return PyLong_FromVoidPtr(at::cuda::getCurrentCUDAStream((c10::DeviceIndex)i).stream());
    END_HANDLE_TH_ERRORS
}

#define HBQ_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(host_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {HBQ_FAST(bind), HBQ_FAST(quantize), HBQ_FAST(gemm), HBQ_FAST(gemm_w4),
                         {"current_stream", host_current_stream, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "hbq_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_hbq_host() { return PyModule_Create(&module); }
