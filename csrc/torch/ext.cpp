// The calls of the Python binding that are made often enough for their own cost to matter, as a CPython
// extension on PyTorch's C++ API.
//
// Measured per call (8 KiB AllReduce on one GPU, host time): 12.8 us through ctypes, of which 3.4 us were
// torch.cuda.current_stream(), 1.3 us the conversion of twelve ctypes arguments, 2 us attribute reads of
// the tensors and 5 us the library and the launch.  Here a tensor is unpacked in place and the library is
// called through the address that the ctypes binding has already loaded (bind()), so MINI_NCCL_LIB selects
// the library as before and nothing links against it.  Arguments that can be wrong are still checked here,
// with the messages and exception types of the Python layer they come from.
//
// The GIL is released around every library call: the network plane's AllReduce blocks, and the ranks of a
// program may be threads of one process.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "mini_nccl_api.h"

namespace {

struct Library {
  decltype(&mncclAllReduceEx) all_reduce_ex = nullptr;
  decltype(&mncclCommGetAsyncError) async_error = nullptr;
  int (*gemm)(const void*, const void*, void*, int, int, int, int, int, int, int, cudaStream_t) = nullptr;
  int (*gemm_rs)(const void*, const void*, void*, int, int, int, int, int, int, int, int, void* const*, void* const*, uint32_t*,
                 const void*, size_t, cudaStream_t) = nullptr;
  int (*ag_gemm)(void* const*, const void*, void*, int, int, int, int, int, int, int, int, void* const*, void* const*, uint32_t*, int,
                 int, const void*, size_t, cudaStream_t) = nullptr;
} lib;

// ncclDataType_t of a tensor's scalar type, -1 for a type the library does not have.
int type_code(at::ScalarType t) {
  switch (t) {
    case at::kChar: return ncclInt8;
    case at::kByte: return ncclUint8;
    case at::kInt: return ncclInt32;
    case at::kUInt32: return ncclUint32;
    case at::kLong: return ncclInt64;
    case at::kUInt64: return ncclUint64;
    case at::kHalf: return ncclFloat16;
    case at::kFloat: return ncclFloat;
    case at::kDouble: return ncclDouble;
    case at::kBFloat16: return ncclBfloat16;
    default: return -1;
  }
}

bool have_gpu() {
  static const bool have = c10::cuda::device_count() > 0;
  return have;
}

// None: the current stream (0 without a GPU); a stream object; or a raw handle.
bool stream_arg(PyObject* o, cudaStream_t* out) {
  if (o == Py_None) {
    *out = have_gpu() ? c10::cuda::getCurrentCUDAStream().stream() : nullptr;
    return true;
  }
  PyObject* raw = PyLong_Check(o) ? Py_NewRef(o) : PyObject_GetAttrString(o, "cuda_stream");
  if (!raw) {
    PyErr_Clear();
    raw = PyNumber_Long(o);
    if (!raw) return false;
  }
  *out = reinterpret_cast<cudaStream_t>(PyLong_AsUnsignedLongLongMask(raw));
  Py_DECREF(raw);
  return !PyErr_Occurred();
}

const at::Tensor* tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a torch tensor", name);
    return nullptr;
  }
  return &THPVariable_Unpack(o);
}

bool arg_count(Py_ssize_t n, Py_ssize_t want) {
  if (n != want) PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, n);
  return n == want;
}

// bind(all_reduce_ex, async_error, gemm, gemm_rs, ag_gemm): addresses in the library that ctypes has loaded (the
// last three may be 0)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (!arg_count(n, 5)) return nullptr;
  lib.all_reduce_ex = reinterpret_cast<decltype(lib.all_reduce_ex)>(PyLong_AsVoidPtr(args[0]));
  lib.async_error = reinterpret_cast<decltype(lib.async_error)>(PyLong_AsVoidPtr(args[1]));
  lib.gemm = reinterpret_cast<decltype(lib.gemm)>(PyLong_AsVoidPtr(args[2]));
  lib.gemm_rs = reinterpret_cast<decltype(lib.gemm_rs)>(PyLong_AsVoidPtr(args[3]));
  lib.ag_gemm = reinterpret_cast<decltype(lib.ag_gemm)>(PyLong_AsVoidPtr(args[4]));
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

// all_reduce(comm, tensor, out | None, wire_dtype | None, op, scale, algo, stream | None) -> ncclResult_t
PyObject* all_reduce(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 8)) return nullptr;
  void* comm = PyLong_AsVoidPtr(args[0]);
  const at::Tensor* in = tensor_arg(args[1], "tensor");
  const at::Tensor* out = args[2] == Py_None ? in : tensor_arg(args[2], "out");
  if (!in || !out) return nullptr;
  if (!in->is_contiguous() || !out->is_contiguous()) {
    PyErr_SetString(PyExc_ValueError, "all_reduce needs contiguous tensors");
    return nullptr;
  }
  const int64_t count = in->numel();
  if (out->numel() != count) {
    PyErr_SetString(PyExc_ValueError, "size mismatch");
    return nullptr;
  }
  const int send_type = type_code(in->scalar_type()), recv_type = type_code(out->scalar_type());
  int wire_type = send_type == recv_type ? recv_type : static_cast<int>(ncclBfloat16);
  if (args[3] != Py_None) {
    if (!THPDtype_Check(args[3])) {
      PyErr_SetString(PyExc_TypeError, "wire_dtype must be a torch dtype");
      return nullptr;
    }
    wire_type = type_code(reinterpret_cast<THPDtype*>(args[3])->scalar_type);
  }
  if (send_type < 0 || recv_type < 0 || wire_type < 0) {
    PyErr_SetString(PyExc_TypeError, "unsupported dtype");
    return nullptr;
  }
  const long op = PyLong_AsLong(args[4]);
  const double scale = PyFloat_AsDouble(args[5]);
  const long algo = PyLong_AsLong(args[6]);
  cudaStream_t stream = nullptr;
  if (PyErr_Occurred() || !stream_arg(args[7], &stream)) return nullptr;
  const void* send = in->data_ptr();
  void* recv = out->data_ptr();
  ncclResult_t rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.all_reduce_ex(send, static_cast<ncclDataType_t>(send_type), recv, static_cast<ncclDataType_t>(recv_type),
                         static_cast<ncclDataType_t>(wire_type), static_cast<size_t>(count), static_cast<ncclRedOp_t>(op), scale,
                         static_cast<mncclAlgo_t>(algo), static_cast<ncclComm_t>(comm), stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

// gemm(a, b, out | None, out_dtype | None, stream | None) -> out; see ops/gemm.py
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 5)) return nullptr;
  const at::Tensor* a = tensor_arg(args[0], "a");
  const at::Tensor* b = tensor_arg(args[1], "b");
  if (!a || !b) return nullptr;
  if (a->scalar_type() != at::kBFloat16 || b->scalar_type() != at::kBFloat16) {
    PyErr_SetString(PyExc_TypeError, "gemm_bf16 needs bf16 operands");
    return nullptr;
  }
  if (a->dim() != 2 || b->dim() != 2 || a->size(1) != b->size(1)) {
    PyErr_SetString(PyExc_ValueError, "shapes: a [M, K], b [N, K]");
    return nullptr;
  }
  if (a->stride(1) != 1 || b->stride(1) != 1) {
    PyErr_SetString(PyExc_ValueError, "operands need a unit inner stride");
    return nullptr;
  }
  const int64_t M = a->size(0), K = a->size(1), N = b->size(0);
  at::Tensor fresh;
  const at::Tensor* out = nullptr;
  if (args[2] != Py_None) {
    out = tensor_arg(args[2], "out");
    if (!out) return nullptr;
  } else {
    at::ScalarType t = at::kBFloat16;
    if (args[3] != Py_None) {
      if (!THPDtype_Check(args[3])) {
        PyErr_SetString(PyExc_TypeError, "out_dtype must be a torch dtype");
        return nullptr;
      }
      t = reinterpret_cast<THPDtype*>(args[3])->scalar_type;
    }
    fresh = at::empty({M, N}, a->options().dtype(t));
    out = &fresh;
  }
  const at::ScalarType ot = out->scalar_type();
  if ((ot != at::kBFloat16 && ot != at::kFloat) || out->dim() != 2 || out->size(0) != M || out->size(1) != N || out->stride(1) != 1) {
    PyErr_SetString(PyExc_ValueError, "out must be [M, N] bf16 or fp32 with a unit inner stride");
    return nullptr;
  }
  cudaStream_t stream = nullptr;
  if (!stream_arg(args[4], &stream)) return nullptr;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.gemm(a->data_ptr(), b->data_ptr(), out->data_ptr(), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K),
                static_cast<int>(a->stride(0)), static_cast<int>(b->stride(0)), static_cast<int>(out->stride(0)),
                ot == at::kFloat ? 1 : 0, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) {
    PyErr_Format(PyExc_RuntimeError, "mncclGemmBf16 failed with code %d", rc);
    return nullptr;
  }
  return fresh.defined() ? THPVariable_Wrap(fresh) : Py_NewRef(args[2]);
  END_HANDLE_TH_ERRORS
}

// What a fused kernel's Python object keeps for its calls, as a tuple of integers: (M, N or K, rank, ranks, address of
// the first and of the second array of peers' buffers, of the state words, address and length of the
// communicator's device handle, ...)
bool workspace_arg(PyObject* t, Py_ssize_t want, uintptr_t (&v)[10]) {
  if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != want) {
    PyErr_SetString(PyExc_TypeError, "bad workspace tuple");
    return false;
  }
  for (Py_ssize_t i = 0; i < want; ++i) v[i] = PyLong_AsUnsignedLongLongMask(PyTuple_GET_ITEM(t, i));
  return !PyErr_Occurred();
}

// A communicator that has failed takes no more work: its error code, 0 when it is usable.
int comm_error(PyObject* comm) {
  ncclResult_t e = ncclSuccess;
  const ncclResult_t rc = lib.async_error(static_cast<ncclComm_t>(PyLong_AsVoidPtr(comm)), &e);
  return rc != ncclSuccess ? rc : e;
}

// gemm_rs(comm, a, b, out | None, stream | None, workspace) -> out, or the communicator's error code; see ops/fused.py
PyObject* gemm_rs(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  uintptr_t w[10];
  if (!arg_count(n, 6) || !workspace_arg(args[5], 9, w)) return nullptr;
  const at::Tensor* a = tensor_arg(args[1], "a");
  const at::Tensor* b = tensor_arg(args[2], "b");
  if (!a || !b) return nullptr;
  const int64_t M = static_cast<int64_t>(w[0]), N = static_cast<int64_t>(w[1]), ranks = static_cast<int64_t>(w[3]);
  if (a->dim() != 2 || b->dim() != 2 || a->size(0) != M || b->size(0) != N || a->size(1) != b->size(1)) {
    PyErr_SetString(PyExc_ValueError, "shape mismatch");
    return nullptr;
  }
  if (a->scalar_type() != at::kBFloat16 || b->scalar_type() != at::kBFloat16 || a->stride(1) != 1 || b->stride(1) != 1) {
    PyErr_SetString(PyExc_TypeError, "bf16 operands with a unit inner stride");
    return nullptr;
  }
  at::Tensor fresh;
  if (args[3] == Py_None) fresh = at::empty({M / ranks, N}, a->options());
  const at::Tensor* out = args[3] == Py_None ? &fresh : tensor_arg(args[3], "out");
  cudaStream_t stream = nullptr;
  if (!out || !stream_arg(args[4], &stream)) return nullptr;
  if (const int e = comm_error(args[0])) return PyLong_FromLong(e);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.gemm_rs(a->data_ptr(), b->data_ptr(), out->data_ptr(), static_cast<int>(M), static_cast<int>(N), static_cast<int>(a->size(1)),
                   static_cast<int>(a->stride(0)), static_cast<int>(b->stride(0)), static_cast<int>(out->stride(0)), static_cast<int>(w[2]),
                   static_cast<int>(ranks), reinterpret_cast<void* const*>(w[4]), reinterpret_cast<void* const*>(w[5]),
                   reinterpret_cast<uint32_t*>(w[6]), reinterpret_cast<const void*>(w[7]), w[8], stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) {
    PyErr_Format(PyExc_RuntimeError, "mncclGemmReduceScatterBf16 failed with code %d", rc);
    return nullptr;
  }
  return fresh.defined() ? THPVariable_Wrap(fresh) : Py_NewRef(args[3]);
  END_HANDLE_TH_ERRORS
}

// ag_gemm(comm, n_comm_ctas, b, out | None, stream | None, swiglu, workspace) -> out, or the communicator's error code
PyObject* ag_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  uintptr_t w[10];
  if (!arg_count(n, 7) || !workspace_arg(args[6], 10, w)) return nullptr;
  const at::Tensor* b = tensor_arg(args[2], "b");
  if (!b) return nullptr;
  const int64_t M = static_cast<int64_t>(w[0]), K = static_cast<int64_t>(w[1]);
  if (b->scalar_type() != at::kBFloat16 || b->dim() != 2 || b->size(1) != K || b->stride(1) != 1) {
    PyErr_SetString(PyExc_TypeError, "b must be bf16 [N, K] with a unit inner stride");
    return nullptr;
  }
  const int64_t N = b->size(0);
  const int swiglu = PyObject_IsTrue(args[5]), n_comm_ctas = static_cast<int>(PyLong_AsLong(args[1]));
  if (swiglu < 0 || PyErr_Occurred()) return nullptr;
  if (swiglu && N % 32 != 0) {
    PyErr_SetString(PyExc_ValueError, "SwiGLU in the epilogue needs N a multiple of 32");
    return nullptr;
  }
  const int64_t n_out = swiglu ? N / 2 : N;
  at::Tensor fresh;
  if (args[3] == Py_None) fresh = at::empty({M, n_out}, b->options());
  const at::Tensor* out = args[3] == Py_None ? &fresh : tensor_arg(args[3], "out");
  if (!out) return nullptr;
  if (out->dim() != 2 || out->size(0) != M || out->size(1) != n_out || out->scalar_type() != at::kBFloat16 || out->stride(1) != 1) {
    PyErr_Format(PyExc_ValueError, "out must be bf16 [%lld, %lld] with a unit inner stride", static_cast<long long>(M), static_cast<long long>(n_out));
    return nullptr;
  }
  cudaStream_t stream = nullptr;
  if (!stream_arg(args[4], &stream)) return nullptr;
  if (const int e = comm_error(args[0])) return PyLong_FromLong(e);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.ag_gemm(reinterpret_cast<void* const*>(w[4]), b->data_ptr(), out->data_ptr(), static_cast<int>(M), static_cast<int>(N),
                   static_cast<int>(K), static_cast<int>(K), static_cast<int>(b->stride(0)), static_cast<int>(out->stride(0)),
                   static_cast<int>(w[2]), static_cast<int>(w[3]), reinterpret_cast<void* const*>(w[5]),
                   reinterpret_cast<void* const*>(w[6]), reinterpret_cast<uint32_t*>(w[7]), n_comm_ctas, swiglu,
                   reinterpret_cast<const void*>(w[8]), w[9], stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) {
    PyErr_Format(PyExc_RuntimeError, "all-gather->GEMM kernel failed with code %d", rc);
    return nullptr;
  }
  return fresh.defined() ? THPVariable_Wrap(fresh) : Py_NewRef(args[3]);
  END_HANDLE_TH_ERRORS
}

// async_error(comm) -> ncclResult_t
PyObject* async_error(PyObject*, PyObject* comm) {
  const int e = comm_error(comm);
  return PyErr_Occurred() ? nullptr : PyLong_FromLong(e);
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(bind)), METH_FASTCALL, nullptr},
    {"all_reduce", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(all_reduce)), METH_FASTCALL, nullptr},
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(gemm)), METH_FASTCALL, nullptr},
    {"gemm_rs", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(gemm_rs)), METH_FASTCALL, nullptr},
    {"ag_gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(ag_gemm)), METH_FASTCALL, nullptr},
    {"async_error", async_error, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_ext", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_ext(void) { return PyModule_Create(&module); }
