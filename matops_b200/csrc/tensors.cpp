// Python extension: torch tensors to the mo_matrix views of the C ABI, in native code.
//
// A view made in Python (dim, dtype, device, shape and two strides read one by one, a ctypes
// structure per matrix) costs about 1.5 us; a batch of 4096 systems paid for 12 000 of them,
// 9 ms per call beside 5 ms of device time, and a small product for three, most of its 10 us.
// The checks and messages are those of api.view.
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>

#include "../../include/matops_b200.h"

namespace {

// fills m from a column-major CUDA float64 matrix; false with a Python error set otherwise
bool as_view(PyObject *o, mo_matrix *m) {
  if (!THPVariable_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "expected a 2-D float64 CUDA tensor");
    return false;
  }
  const at::Tensor &t = THPVariable_Unpack(o);
  if (t.dim() != 2 || t.scalar_type() != at::kDouble || !t.is_cuda()) {
    PyErr_SetString(PyExc_TypeError, "expected a 2-D float64 CUDA tensor");
    return false;
  }
  const int64_t r = t.size(0), c = t.size(1);
  if (r > 1 && t.stride(0) != 1) {
    PyErr_SetString(PyExc_TypeError, "matrix view must be column-major (stride(0) == 1)");
    return false;
  }
  m->data = static_cast<double *>(t.data_ptr());
  m->rows = r;
  m->cols = c;
  m->ld = std::max<int64_t>({t.stride(1), r, 1});
  return true;
}

// a C++ exception (a tensor without storage, say) becomes a Python one
template <typename F>
PyObject *guarded(F &&f) {
  try {
    return f();
  } catch (const std::exception &e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

int (*set_stream)(mo_ctx *, void *) = nullptr;  // mo_set_stream (bind)

// the C function at `fn` on the context, with its work on `stream`; called without the GIL
template <typename... A>
PyObject *invoke(PyObject *fn, PyObject *ctx, unsigned long long stream, A... args) {
  auto f = reinterpret_cast<int (*)(mo_ctx *, A...)>(PyLong_AsVoidPtr(fn));
  auto c = static_cast<mo_ctx *>(PyLong_AsVoidPtr(ctx));
  if (!f || !c || !set_stream) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "the library is not bound");
    return nullptr;
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS set_stream(c, reinterpret_cast<void *>(stream));
  rc = f(c, args...);
  Py_END_ALLOW_THREADS return PyLong_FromLong(rc);
}

// bind(address of mo_set_stream)
PyObject *bind(PyObject *, PyObject *addr) {
  set_stream = reinterpret_cast<int (*)(mo_ctx *, void *)>(PyLong_AsVoidPtr(addr));
  if (!set_stream && PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

// call3(fn, ctx, stream, C, A, B, alpha, beta, flags) -> status
PyObject *call3(PyObject *, PyObject *args) {
  PyObject *fn, *ctx, *c, *a, *b;
  double alpha, beta;
  int flags;
  unsigned long long st;
  if (!PyArg_ParseTuple(args, "OOKOOOddi", &fn, &ctx, &st, &c, &a, &b, &alpha, &beta, &flags)) return nullptr;
  return guarded([&]() -> PyObject * {
    mo_matrix C, A, B;
    if (!as_view(c, &C) || !as_view(a, &A) || !as_view(b, &B)) return nullptr;
    return invoke(fn, ctx, st, C, A, B, alpha, beta, flags);
  });
}

// call2(fn, ctx, stream, C, A, alpha, beta, flags) -> status
PyObject *call2(PyObject *, PyObject *args) {
  PyObject *fn, *ctx, *c, *a;
  double alpha, beta;
  int flags;
  unsigned long long st;
  if (!PyArg_ParseTuple(args, "OOKOOddi", &fn, &ctx, &st, &c, &a, &alpha, &beta, &flags)) return nullptr;
  return guarded([&]() -> PyObject * {
    mo_matrix C, A;
    if (!as_view(c, &C) || !as_view(a, &A)) return nullptr;
    return invoke(fn, ctx, st, C, A, alpha, beta, flags);
  });
}

// call2a(fn, ctx, stream, B, A, alpha, flags) -> status
PyObject *call2a(PyObject *, PyObject *args) {
  PyObject *fn, *ctx, *b, *a;
  double alpha;
  int flags;
  unsigned long long st;
  if (!PyArg_ParseTuple(args, "OOKOOdi", &fn, &ctx, &st, &b, &a, &alpha, &flags)) return nullptr;
  return guarded([&]() -> PyObject * {
    mo_matrix B, A;
    if (!as_view(b, &B) || !as_view(a, &A)) return nullptr;
    return invoke(fn, ctx, st, B, A, alpha, flags);
  });
}

// views(sequence of tensors, address of as many mo_matrix)
PyObject *views(PyObject *, PyObject *args) {
  PyObject *seq;
  unsigned long long addr;
  if (!PyArg_ParseTuple(args, "OK", &seq, &addr)) return nullptr;
  PyObject *fast = PySequence_Fast(seq, "expected a sequence of tensors");
  if (!fast) return nullptr;
  PyObject *res = guarded([&]() -> PyObject * {
    mo_matrix *out = reinterpret_cast<mo_matrix *>(addr);
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
    for (Py_ssize_t i = 0; i < n; ++i)
      if (!as_view(PySequence_Fast_GET_ITEM(fast, i), out + i)) return nullptr;
    Py_RETURN_NONE;
  });
  Py_DECREF(fast);
  return res;
}

// batch_pack(As, Bs or None, pivs or None, orders, count, nrhs, table) -> whether the table
// changed.  orders: address of count int32; table: address of 5 x count int64 that receive
// the addresses and leading dimensions of A, those of B and the addresses of the pivots
// (zeros where not given).  Raises ValueError for shapes that do not match the orders.
PyObject *batch_pack(PyObject *, PyObject *args) {
  PyObject *list[3];
  unsigned long long orders, table;
  Py_ssize_t count;
  long long nrhs;
  if (!PyArg_ParseTuple(args, "OOOKnLK", &list[0], &list[1], &list[2], &orders, &count, &nrhs, &table))
    return nullptr;
  PyObject *fast[3] = {nullptr, nullptr, nullptr};
  PyObject *res = guarded([&]() -> PyObject * {
    for (int l = 0; l < 3; ++l) {
      if (list[l] == Py_None) continue;
      if (!(fast[l] = PySequence_Fast(list[l], "expected a sequence of tensors"))) return nullptr;
      if (PySequence_Fast_GET_SIZE(fast[l]) < count) {
        PyErr_SetString(PyExc_ValueError, "number of matrices does not match the plan");
        return nullptr;
      }
    }
    const int32_t *n = reinterpret_cast<const int32_t *>(orders);
    int64_t *t = reinterpret_cast<int64_t *>(table);
    bool changed = false;
    auto put = [&](Py_ssize_t at, int64_t v) {
      changed |= t[at] != v;
      t[at] = v;
    };
    for (Py_ssize_t i = 0; i < count; ++i) {
      mo_matrix A;
      if (!as_view(PySequence_Fast_GET_ITEM(fast[0], i), &A)) return nullptr;
      if (A.rows != n[i] || A.cols != n[i]) {
        PyErr_SetString(PyExc_ValueError, "matrix shape does not match the plan's order");
        return nullptr;
      }
      put(i, reinterpret_cast<int64_t>(A.data));
      put(count + i, A.ld);
    }
    for (Py_ssize_t i = 0; i < count; ++i) {
      mo_matrix B{nullptr, 0, 0, 0};
      if (fast[1]) {
        if (!as_view(PySequence_Fast_GET_ITEM(fast[1], i), &B)) return nullptr;
        if (B.rows != n[i] || B.cols != nrhs) {
          PyErr_SetString(PyExc_ValueError, "right-hand side shape does not match the plan");
          return nullptr;
        }
      }
      put(2 * count + i, reinterpret_cast<int64_t>(B.data));
      put(3 * count + i, B.ld);
    }
    for (Py_ssize_t i = 0; i < count; ++i) {
      int64_t p = 0;
      if (fast[2]) {
        PyObject *o = PySequence_Fast_GET_ITEM(fast[2], i);
        if (!THPVariable_Check(o)) {
          PyErr_SetString(PyExc_TypeError, "pivots must be tensors");
          return nullptr;
        }
        p = reinterpret_cast<int64_t>(THPVariable_Unpack(o).data_ptr());
      }
      put(4 * count + i, p);
    }
    return PyBool_FromLong(changed);
  });
  for (PyObject *f : fast) Py_XDECREF(f);
  return res;
}

PyMethodDef methods[] = {{"bind", bind, METH_O, nullptr},
                         {"call3", call3, METH_VARARGS, nullptr},
                         {"call2", call2, METH_VARARGS, nullptr},
                         {"call2a", call2a, METH_VARARGS, nullptr},
                         {"views", views, METH_VARARGS, nullptr},
                         {"batch_pack", batch_pack, METH_VARARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_tensors", nullptr, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tensors() { return PyModule_Create(&module); }
