// native_calls.cpp - the short way from Python to the C entry points that programs call most: argument checks, result allocation
// and stream look-up in C++ instead of some ten Python and ctypes steps, which took longer than the kernels of small operands.
// us a call from Python, before / after: a GEMM of 200 x 136 x 72 9.0 / 4.8, an operator of 2048 floats 6.1 / 3.9.
//
// Every function returns None for whatever it does not know for certain (other devices, types, layouts, tensor subclasses, active
// function or dispatch modes, tensors of transforms): the caller then goes the general way, which also raises the errors.  A
// failed launch comes back as its HcclResult.  Entry points are handed over as addresses, so that they are those of the library
// that Python loaded.  The interpreter lock is released around them, since ranks of one process may wait for one another.
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include "hccl/hccl_types.h"
#include "released.h"

namespace {

using hcomm_torch::Released;
using AllReduceFn = int (*)(void *, void *, uint64_t, int, int, void *, void *);
using AllReduceScaledFn = int (*)(void *, void *, uint64_t, int, int, float, void *, void *);
using AllGatherFn = int (*)(void *, void *, uint64_t, int, void *, void *);
using AlltoAllFn = int (*)(const void *, uint64_t, int, const void *, uint64_t, int, void *, void *);
using GemmFn = int (*)(const void *, const void *, void *, int, int, int, int, int, int, void *);
using DispatchFn = int (*)(void *, const void *, const int32_t *, int, void *);
using CombineFn = int (*)(void *, const void *, uint64_t, const float *, void *, int, void *);

const c10::DispatchKeySet kPlain = c10::DispatchKeySet({c10::DispatchKey::Dense, c10::DispatchKey::AutogradFunctionality, c10::DispatchKey::ADInplaceOrView,
                                                        c10::DispatchKey::AutocastCUDA}) |
                                   c10::DispatchKeySet(c10::BackendComponent::CUDABit);

// A strided CUDA tensor with memory of its own on the current device, nothing wrapped around it; NULL otherwise.
const at::Tensor *Plain(PyObject *o, int device)
{
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.defined()) return nullptr;
    const c10::TensorImpl *impl = t.unsafeGetTensorImpl();
    if ((impl->key_set().raw_repr() & ~kPlain.raw_repr()) != 0 || !t.is_cuda() || t.get_device() != device || !impl->has_storage() || impl->layout() != c10::kStrided)
        return nullptr;
    return &t;
}
bool ModesActive()
{
    return at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
           (c10::impl::tls_local_dispatch_key_set().included_.raw_repr() & ~c10::default_included_set.raw_repr()) != 0;
}
// The device of this call, -1 where the general way has to be taken.
int Device() { return ModesActive() ? -1 : (int)c10::cuda::current_device(); }
void *StreamOf(int device) { return (void *)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }
// The address in a Python integer; false for anything else (the handle of a communicator that was destroyed is None).
bool Address(PyObject *o, void **p)
{
    if (!PyLong_Check(o)) return false;
    *p = PyLong_AsVoidPtr(o);
    if (!PyErr_Occurred()) return true;
    PyErr_Clear();
    return false;
}

int TypeCode(at::ScalarType t)
{
    switch (t) {
        case at::kChar: return HCCL_DATA_TYPE_INT8; case at::kShort: return HCCL_DATA_TYPE_INT16; case at::kInt: return HCCL_DATA_TYPE_INT32;
        case at::kLong: return HCCL_DATA_TYPE_INT64; case at::kByte: return HCCL_DATA_TYPE_UINT8; case at::kFloat: return HCCL_DATA_TYPE_FP32;
        case at::kHalf: return HCCL_DATA_TYPE_FP16; case at::kBFloat16: return HCCL_DATA_TYPE_BFP16; case at::kDouble: return HCCL_DATA_TYPE_FP64;
        default: return -1;
    }
}

// A matrix of bf16 whose rows are contiguous and whose sizes the entry points can take.
bool Matrix(const at::Tensor *t)
{
    const int64_t most = INT32_MAX;
    return t && t->scalar_type() == at::kBFloat16 && t->dim() == 2 && t->stride(1) == 1 && t->size(0) <= most && t->size(1) <= most && t->stride(0) >= 0 &&
           t->stride(0) <= most;
}

// gemm_bf16(entry, a, b, out or None) -> the result, an error code, or None
PyObject *Gemm(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    if (n != 4) Py_RETURN_NONE;
    const int dev = Device();
    const at::Tensor *a = dev < 0 ? nullptr : Plain(args[1], dev), *b = a ? Plain(args[2], dev) : nullptr;
    if (!Matrix(a) || !Matrix(b) || a->size(1) != b->size(1)) Py_RETURN_NONE;
    void *entry;
    if (!Address(args[0], &entry)) Py_RETURN_NONE;
    const int64_t m = a->size(0), k = a->size(1), w = b->size(0);
    at::Tensor made;
    const at::Tensor *out = &made;
    if (args[3] == Py_None) made = at::empty({m, w}, a->options());
    else if (!(out = Plain(args[3], dev)) || out->dim() != 2 || out->stride(0) > INT32_MAX) Py_RETURN_NONE;
    const auto fn = (GemmFn)entry;
    const void *pa = a->data_ptr(), *pb = b->data_ptr();
    void *pc = out->data_ptr(), *stream = StreamOf(dev);
    const int lda = (int)a->stride(0), ldb = (int)b->stride(0), ldc = (int)out->stride(0);
    const int rc = Released([=] { return fn(pa, pb, pc, (int)m, (int)w, (int)k, lda, ldb, ldc, stream); });
    if (rc) return PyLong_FromLong(rc);
    if (args[3] != Py_None) return Py_NewRef(args[3]);
    return THPVariable_Wrap(std::move(made));
    END_HANDLE_TH_ERRORS
}

// collective(entry, kind, send, recv, communicator, operator, scale, ranks) -> an error code (0: launched) or None
enum Kind { ALL_REDUCE, ALL_REDUCE_SCALED, REDUCE_SCATTER, ALL_GATHER, ALL_TO_ALL };
PyObject *Collective(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    if (n != 8) Py_RETURN_NONE;
    const int dev = Device();
    const at::Tensor *in = dev < 0 ? nullptr : Plain(args[2], dev), *out = in ? Plain(args[3], dev) : nullptr;
    if (!out || !in->is_contiguous() || !out->is_contiguous()) Py_RETURN_NONE;
    const int type = TypeCode(in->scalar_type()), outType = TypeCode(out->scalar_type());
    void *fn, *comm;
    if (type < 0 || outType < 0 || !Address(args[0], &fn) || !Address(args[4], &comm)) Py_RETURN_NONE;
    const int kind = (int)PyLong_AsLong(args[1]), op = (int)PyLong_AsLong(args[5]);
    const float scale = (float)PyFloat_AsDouble(args[6]);
    const uint64_t ranks = (uint64_t)PyLong_AsLong(args[7]), count = (uint64_t)in->numel(), outCount = (uint64_t)out->numel();
    if (PyErr_Occurred() || ranks == 0) { PyErr_Clear(); Py_RETURN_NONE; }
    void *src = in->data_ptr(), *dst = out->data_ptr(), *stream = StreamOf(dev);
    return PyLong_FromLong(Released([=]() -> int {
        switch (kind) {
            case ALL_REDUCE: return ((AllReduceFn)fn)(src, dst, count, type, op, comm, stream);
            case ALL_REDUCE_SCALED: return ((AllReduceScaledFn)fn)(src, dst, count, type, outType, scale, comm, stream);
            case REDUCE_SCATTER: return ((AllReduceFn)fn)(src, dst, outCount, type, op, comm, stream);
            case ALL_GATHER: return ((AllGatherFn)fn)(src, dst, count, type, comm, stream);
            default: return ((AlltoAllFn)fn)(src, count / ranks, type, dst, count / ranks, type, comm, stream);
        }
    }));
    END_HANDLE_TH_ERRORS
}

// moe_dispatch(entry, exchange, x, choices, hidden, topk) -> an error code (0: launched) or None
PyObject *MoeDispatch(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    if (n != 6) Py_RETURN_NONE;
    const int dev = Device();
    const at::Tensor *x = dev < 0 ? nullptr : Plain(args[2], dev), *idx = x ? Plain(args[3], dev) : nullptr;
    void *entry, *handle;
    if (!idx || !Address(args[0], &entry) || !Address(args[1], &handle)) Py_RETURN_NONE;
    const int64_t hidden = PyLong_AsLong(args[4]), topk = PyLong_AsLong(args[5]);
    if (x->scalar_type() != at::kBFloat16 || idx->scalar_type() != at::kInt || x->dim() != 2 || idx->dim() != 2 || x->size(1) != hidden ||
        idx->size(0) != x->size(0) || idx->size(1) != topk || !x->is_contiguous() || !idx->is_contiguous() || x->size(0) > INT32_MAX)
        Py_RETURN_NONE;
    const auto fn = (DispatchFn)entry;
    void *const px = x->data_ptr(), *const pi = idx->data_ptr(), *const stream = StreamOf(dev);
    const int tokens = (int)x->size(0);
    return PyLong_FromLong(Released([=] { return fn(handle, px, (const int32_t *)pi, tokens, stream); }));
    END_HANDLE_TH_ERRORS
}

// moe_combine(entry, exchange, y, gates, out or None, hidden) -> the result, an error code, or None
PyObject *MoeCombine(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    if (n != 6) Py_RETURN_NONE;
    const int dev = Device();
    const at::Tensor *y = dev < 0 ? nullptr : Plain(args[2], dev), *gates = y ? Plain(args[3], dev) : nullptr;
    void *entry, *handle;
    if (!gates || !Address(args[0], &entry) || !Address(args[1], &handle)) Py_RETURN_NONE;
    const int64_t hidden = PyLong_AsLong(args[5]);
    if (y->scalar_type() != at::kBFloat16 || gates->scalar_type() != at::kFloat || y->dim() != 2 || y->size(1) != hidden || gates->dim() < 1 ||
        !y->is_contiguous() || !gates->is_contiguous() || gates->size(0) > INT32_MAX)
        Py_RETURN_NONE;
    at::Tensor made;
    const at::Tensor *out = &made;
    if (args[4] == Py_None) made = at::empty({gates->size(0), hidden}, y->options());
    else if (!(out = Plain(args[4], dev))) Py_RETURN_NONE;
    const auto fn = (CombineFn)entry;
    void *const py = y->data_ptr(), *const pg = gates->data_ptr(), *const po = out->data_ptr(), *const stream = StreamOf(dev);
    const uint64_t rows = (uint64_t)y->size(0);
    const int tokens = (int)gates->size(0);
    const int rc = Released([=] { return fn(handle, py, rows, (const float *)pg, po, tokens, stream); });
    if (rc) return PyLong_FromLong(rc);
    if (args[4] != Py_None) return Py_NewRef(args[4]);
    return THPVariable_Wrap(std::move(made));
    END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"gemm_bf16", (PyCFunction)(void *)Gemm, METH_FASTCALL, nullptr},
    {"collective", (PyCFunction)(void *)Collective, METH_FASTCALL, nullptr},
    {"moe_dispatch", (PyCFunction)(void *)MoeDispatch, METH_FASTCALL, nullptr},
    {"moe_combine", (PyCFunction)(void *)MoeCombine, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

}  // namespace

namespace hcomm_torch {
bool AddNativeCalls(PyObject *module) { return PyModule_AddFunctions(module, kMethods) == 0; }
}  // namespace hcomm_torch
