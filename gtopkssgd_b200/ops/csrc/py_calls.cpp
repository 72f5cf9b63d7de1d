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

#define GTK_METHOD(name) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Call<name>::fast)), METH_FASTCALL, nullptr}

PyMethodDef kMethods[] = {
    GTK_METHOD(gtk_k1_select),        GTK_METHOD(gtk_k1_select_segments),
    GTK_METHOD(gtk_k1_compress),      GTK_METHOD(gtk_k2_exchange),      GTK_METHOD(gtk_k2t_allgather),
    GTK_METHOD(gtk_k3_dense),         GTK_METHOD(gtk_k3_sparse),      GTK_METHOD(gtk_k3_scatter_dense),
    GTK_METHOD(gtk_k3_momentum_correct), GTK_METHOD(gtk_k4_sumsq_dense), GTK_METHOD(gtk_k4_sumsq_pairs),
    GTK_METHOD(gtk_k4_finalize),      GTK_METHOD(gtk_k5_top1),          {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_gtk_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__gtk_calls(void) { return PyModule_Create(&kModule); }
