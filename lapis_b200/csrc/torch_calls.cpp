// CPython entry points of the device-resident layer: tensor checks, address and stream lookup and the call into
// liblapis_b200.so in native code.
//
// A small call is bound by the host: at 10,000 rows the SpMV kernel takes 2-3 us and the launch 2 us, while the same
// checks written in Python with a ctypes call took 11 us (3.5 us of it torch.cuda.current_stream()).
// Every function returns the library's status, or -1 when an operand is not the kind of tensor it takes; the caller
// (lapis_b200/device.py) then names the operand in the exception it raises.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/Exception.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/lapis_b200.h"

namespace {

const at::Tensor *tensor(PyObject *o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }
bool is(const at::Tensor *t, at::ScalarType st) {
  return t != nullptr && t->is_cuda() && t->scalar_type() == st && t->is_contiguous();
}
// Two extents, further ones being 1: a row-major matrix.
bool is_matrix(const at::Tensor *t) {
  for (int64_t d = 2; d < t->dim(); ++d)
    if (t->size(d) != 1) return false;
  return t->dim() >= 2;
}
bool is_index(const at::Tensor *t) {
  return t != nullptr && t->is_cuda() && (t->scalar_type() == at::kInt || t->scalar_type() == at::kLong) && t->is_contiguous();
}
void *addr(const at::Tensor *t) { return t->numel() == 0 ? nullptr : t->data_ptr(); }
template <typename T>
T *addr_of(const at::Tensor *t) {
  return static_cast<T *>(addr(t));
}
void *stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
lapis_b200_csr_t handle(PyObject *o) { return static_cast<lapis_b200_csr_t>(PyLong_AsVoidPtr(o)); }
PyObject *status(int code) { return PyLong_FromLong(code); }
// Calls the library without the interpreter lock: a launch waits where the stream's queue is full.
template <typename... P, typename... A>
PyObject *call(int (*fn)(P...), A... args) {
  int code;
  Py_BEGIN_ALLOW_THREADS
  code = fn(static_cast<P>(args)...);
  Py_END_ALLOW_THREADS
  return status(code);
}

// What Python calls.  torch reports some operands by a C++ exception (a tensor without storage has no address, a sparse
// one no contiguity), which must not leave a C function; an argument that is no integer leaves a Python one.
template <PyObject *(*CALL)(PyObject *const *), Py_ssize_t ARGS>
PyObject *entry(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  if (nargs != ARGS) {
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");
    return nullptr;
  }
  try {
    PyObject *result = CALL(a);
    if (PyErr_Occurred() == nullptr) return result;
    Py_XDECREF(result);
  } catch (const c10::Error &e) {
    if (PyErr_Occurred() == nullptr) PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception &e) {
    if (PyErr_Occurred() == nullptr) PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// spmv(handle, nrows, ncols, x, y, accumulate)
PyObject *py_spmv(PyObject *const *a) {
  const int accumulate = PyObject_IsTrue(a[5]);
  if (accumulate < 0) return nullptr;
  const at::Tensor *x = tensor(a[3]), *y = tensor(a[4]);
  if (!is(x, at::kDouble) || !is(y, at::kDouble)) return status(-1);
  if (y->numel() != PyLong_AsLongLong(a[1]) || x->numel() != PyLong_AsLongLong(a[2])) return status(-1);
  return call(lapis_b200_spmv_f64, handle(a[0]), addr_of<double>(x), addr_of<double>(y), accumulate, stream());
}

// spmm(handle, nrows, ncols, B, C, accumulate)
PyObject *py_spmm(PyObject *const *a) {
  const int accumulate = PyObject_IsTrue(a[5]);
  if (accumulate < 0) return nullptr;
  const at::Tensor *B = tensor(a[3]), *C = tensor(a[4]);
  if (!is(B, at::kDouble) || !is(C, at::kDouble) || !is_matrix(B) || !is_matrix(C)) return status(-1);
  if (C->size(0) != PyLong_AsLongLong(a[1]) || B->size(0) != PyLong_AsLongLong(a[2]) || B->size(1) != C->size(1)) return status(-1);
  return call(lapis_b200_spmm_f64, handle(a[0]), B->size(1), addr_of<double>(B), addr_of<double>(C), accumulate, stream());
}

// spmm_dcsr(i1, p2, i2, val, B, C, ncols)
PyObject *py_spmm_dcsr(PyObject *const *a) {
  const at::Tensor *i1 = tensor(a[0]), *p2 = tensor(a[1]), *i2 = tensor(a[2]), *val = tensor(a[3]), *B = tensor(a[4]), *C = tensor(a[5]);
  const long long ncols = PyLong_AsLongLong(a[6]);
  if (!is_index(i1) || !is_index(p2) || !is_index(i2) || i1->scalar_type() != p2->scalar_type() ||
      i2->scalar_type() != p2->scalar_type() || !is(val, at::kDouble) || !is(B, at::kDouble) || !is(C, at::kDouble))
    return status(-1);
  if (B->dim() != 2 || C->dim() != 2 || B->size(0) != ncols || B->size(1) != C->size(1) || p2->numel() != i1->numel() + 1)
    return status(-1);
  return call(lapis_b200_spmm_dcsr_f64, (int)p2->element_size(), C->size(0), ncols, i1->numel(), B->size(1), addr(i1), addr(p2),
              addr(i2), addr_of<double>(val), addr_of<double>(B), addr_of<double>(C), stream());
}

// bspmm(pos, crd, val, B, C, n2, accumulate)
PyObject *py_bspmm(PyObject *const *a) {
  const int accumulate = PyObject_IsTrue(a[6]);
  if (accumulate < 0) return nullptr;
  const at::Tensor *pos = tensor(a[0]), *crd = tensor(a[1]), *val = tensor(a[2]), *B = tensor(a[3]), *C = tensor(a[4]);
  const long long n2 = PyLong_AsLongLong(a[5]);
  if (!is_index(pos) || !is_index(crd) || pos->scalar_type() != crd->scalar_type() || !is(val, at::kFloat) || !is(B, at::kFloat) ||
      !is(C, at::kFloat) || B->dim() != 3 || C->dim() != 3)
    return status(-1);
  const int64_t n1 = pos->numel() - 1, dh = B->size(1), nh = B->size(2);
  if (B->size(0) != n2 || val->numel() != crd->numel() * nh || C->size(0) != n1 || C->size(1) != dh || C->size(2) != nh) return status(-1);
  return call(lapis_b200_bspmm_csrv_f32, (int)pos->element_size(), n1, n2, nh, dh, addr(pos), addr(crd), addr_of<float>(val),
              addr_of<float>(B), addr_of<float>(C), accumulate, stream());
}

// bgemm(A, B, C): [M,K]x[K,N] or [b,M,K]x[b,K,N]
PyObject *py_bgemm(PyObject *const *a) {
  const at::Tensor *A = tensor(a[0]), *B = tensor(a[1]), *C = tensor(a[2]);
  if (!is(A, at::kFloat) || !is(B, at::kFloat) || !is(C, at::kFloat)) return status(-1);
  const int64_t d = A->dim();
  if ((d != 2 && d != 3) || B->dim() != d || C->dim() != d) return status(-1);
  const int64_t batch = d == 3 ? A->size(0) : 1, M = A->size(d - 2), K = A->size(d - 1), N = B->size(d - 1);
  if (B->size(d - 2) != K || C->size(d - 2) != M || C->size(d - 1) != N || (d == 3 && (B->size(0) != batch || C->size(0) != batch)))
    return status(-1);
  return call(lapis_b200_bgemm_f32, batch, M, N, K, addr_of<float>(A), addr_of<float>(B), addr_of<float>(C), stream());
}

template <PyObject *(*CALL)(PyObject *const *), Py_ssize_t ARGS>
PyMethodDef method(const char *name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entry<CALL, ARGS>)), METH_FASTCALL, nullptr};
}
PyMethodDef methods[] = {method<py_spmv, 6>("spmv"),   method<py_spmm, 6>("spmm"),   method<py_spmm_dcsr, 7>("spmm_dcsr"),
                         method<py_bspmm, 7>("bspmm"), method<py_bgemm, 3>("bgemm"), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) { return PyModule_Create(&module); }
