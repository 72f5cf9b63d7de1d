// CPython module over the launch entry points of the library.
//
// A launch costs about 2.2 us in the driver; through ctypes the conversion of 13
// to 21 arguments cost another 3 to 6 us per call, which bounded every call on a
// small vector (a select of 1 M elements and its sparse update: 23 us of host
// work for 16 us of kernels).  Here each entry point is a METH_FASTCALL function
// whose arguments are converted straight from the C signature: pointers and
// handles from int or None, numbers from int or float, about 15 ns each.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <type_traits>
#include <utility>
#include <vector>
#include "host_api.h"

namespace {

template <typename T>
inline T convert(PyObject* o) {
  if constexpr (std::is_same_v<T, gtk_addresses>) {  // a list of int
    static thread_local std::vector<unsigned long long> words;
    if (!PyList_Check(o)) {
      PyErr_SetString(PyExc_TypeError, "expected a list of addresses");
      return gtk_addresses{nullptr, 0};
    }
    const Py_ssize_t n = PyList_GET_SIZE(o);
    words.resize(n);
    for (Py_ssize_t i = 0; i < n; ++i) words[i] = PyLong_AsUnsignedLongLong(PyList_GET_ITEM(o, i));
    return gtk_addresses{words.data(), static_cast<unsigned int>(n)};
  } else if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) return nullptr;
    return reinterpret_cast<T>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLong(o)));
  } else if constexpr (std::is_floating_point_v<T>) {
    return static_cast<T>(PyFloat_AsDouble(o));
  } else if constexpr (std::is_signed_v<T>) {
    return static_cast<T>(PyLong_AsLongLong(o));
  } else {
    return static_cast<T>(PyLong_AsUnsignedLongLong(o));
  }
}

template <auto F>
struct Call;

template <typename... A, int (*F)(A...)>
struct Call<F> {
  template <size_t... I>
  static PyObject* apply(PyObject* const* args, std::index_sequence<I...>) {
    const int code = call(convert<A>(args[I])...);
    return code == kRaised ? nullptr : PyLong_FromLong(code);
  }
  static PyObject* fast(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != static_cast<Py_ssize_t>(sizeof...(A))) {
      PyErr_Format(PyExc_TypeError, "expected %zu arguments, got %zd", sizeof...(A), n);
      return nullptr;
    }
    return apply(args, std::index_sequence_for<A...>{});
  }

 private:
  static constexpr int kRaised = -1000;
  static int call(A... a) {
    if (PyErr_Occurred()) return kRaised;
    int code;
    Py_BEGIN_ALLOW_THREADS  // a full launch queue makes the driver wait
    code = F(a...);
    Py_END_ALLOW_THREADS
    return code;
  }
};

// ---- p.grad of many parameters -----------------------------------------------------------------------------
// One iteration looks at every parameter's gradient; from Python that is 1 us each, here a quarter of that.
PyObject *kGrad, *kDataPtr, *kDtype, *kIsContiguous;

// clear_grads(params): p.grad = None
PyObject* clear_grads(PyObject*, PyObject* params) {
  PyObject* seq = PySequence_Fast(params, "expected a sequence of parameters");
  if (!seq) return nullptr;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i)
    if (PyObject_SetAttr(PySequence_Fast_GET_ITEM(seq, i), kGrad, Py_None) < 0) {
      Py_DECREF(seq);
      return nullptr;
    }
  Py_DECREF(seq);
  Py_RETURN_NONE;
}

// grad_addresses(params, dtype): [p.grad.data_ptr() or 0 where there is none]; None if a gradient is not contiguous
// or not of that dtype.
PyObject* grad_addresses(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2) {
    PyErr_SetString(PyExc_TypeError, "grad_addresses(params, dtype)");
    return nullptr;
  }
  PyObject* seq = PySequence_Fast(args[0], "expected a sequence of parameters");
  if (!seq) return nullptr;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
  PyObject* out = PyList_New(n);
  bool usable = out != nullptr;
  for (Py_ssize_t i = 0; usable && i < n; ++i) {
    PyObject* g = PyObject_GetAttr(PySequence_Fast_GET_ITEM(seq, i), kGrad);
    PyObject* at = nullptr;
    if (g == Py_None) {
      at = PyLong_FromLong(0);
    } else if (g) {
      PyObject* dtype = PyObject_GetAttr(g, kDtype);
      PyObject* dense = dtype == args[1] ? PyObject_CallMethodNoArgs(g, kIsContiguous) : nullptr;
      if (dense == Py_True) at = PyObject_CallMethodNoArgs(g, kDataPtr);
      Py_XDECREF(dense);
      Py_XDECREF(dtype);
    }
    Py_XDECREF(g);
    if (at) PyList_SET_ITEM(out, i, at);
    else usable = false;
  }
  Py_DECREF(seq);
  if (usable) return out;
  Py_XDECREF(out);
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

#define GTK_METHOD(name) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Call<name>::fast)), METH_FASTCALL, nullptr}

PyMethodDef kMethods[] = {
    GTK_METHOD(gtk_k1_select),        GTK_METHOD(gtk_k1_select_segments),
    GTK_METHOD(gtk_k1_compress),      GTK_METHOD(gtk_k2_exchange),      GTK_METHOD(gtk_k2t_allgather),
    GTK_METHOD(gtk_k3_dense),         GTK_METHOD(gtk_k3_sparse),      GTK_METHOD(gtk_k3_scatter_dense),
    GTK_METHOD(gtk_k3_momentum_correct), GTK_METHOD(gtk_k4_sumsq_dense), GTK_METHOD(gtk_k4_sumsq_pairs),
    GTK_METHOD(gtk_k4_finalize),      GTK_METHOD(gtk_k5_top1),
    {"clear_grads", clear_grads, METH_O, nullptr},
    {"grad_addresses", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&grad_addresses)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_gtk_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__gtk_calls(void) {
  kGrad = PyUnicode_InternFromString("grad");
  kDataPtr = PyUnicode_InternFromString("data_ptr");
  kDtype = PyUnicode_InternFromString("dtype");
  kIsContiguous = PyUnicode_InternFromString("is_contiguous");
  return PyModule_Create(&kModule);
}
