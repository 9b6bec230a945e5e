// Whether an ensemble's models still hold the very tensors that a table of their addresses was made from, and these still
// lie where they did.  A prediction asks it before every launch: with attribute getters, comparisons and data_ptr() from Python the
// answer for 100 trees took 28 us of the 46 of a prediction of 16 rows (500 trees: 136 of 153), here 5 of 22 (22 of 47).
#include <Python.h>

#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstring>
#include <exception>

namespace {

PyObject* g_names[3];  // leaf_value, feature, split_value

// 1: model `m` holds source[0 .. 2] at addresses[0 .. 2], 0: it does not, -1: a Python error is set
int HoldsArrays(PyObject* m, PyObject* const* source, const char* addresses)
{
  for (int i = 0; i < 3; ++i) {
    PyObject* t = PyObject_GetAttr(m, g_names[i]);
    if (t == nullptr) return -1;
    int same = t == source[i] && THPVariable_Check(t) ? 1 : 0;
    if (same) {
      try {
        const auto at = static_cast<int64_t>(reinterpret_cast<intptr_t>(THPVariable_Unpack(t).const_data_ptr()));
        same          = std::memcmp(&at, addresses + 8 * i, 8) == 0 ? 1 : 0;
      } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        same = -1;
      } catch (...) {
        PyErr_SetString(PyExc_RuntimeError, "the address of a tensor could not be had");
        same = -1;
      }
    }
    Py_DECREF(t);
    if (same != 1) return same;
  }
  return 1;
}

// holds(models: list, source: tuple of 3 tensors per model, addresses: bytes, 8 of each) -> bool
PyObject* Holds(PyObject*, PyObject* const* args, Py_ssize_t n_args)
{
  if (n_args != 3 || !PyList_Check(args[0]) || !PyTuple_Check(args[1]) || !PyBytes_Check(args[2])) {
    PyErr_SetString(PyExc_TypeError, "holds(models: list, source: tuple, addresses: bytes)");
    return nullptr;
  }
  PyObject *models = args[0], *source = args[1];
  const Py_ssize_t n = PyTuple_GET_SIZE(source);
  if (n % 3 != 0 || PyBytes_GET_SIZE(args[2]) != 8 * n) {
    PyErr_SetString(PyExc_ValueError, "three tensors per model, eight bytes per tensor");
    return nullptr;
  }
  if (PyList_GET_SIZE(models) != n / 3) Py_RETURN_FALSE;
  const char* addresses = PyBytes_AS_STRING(args[2]);
  for (Py_ssize_t i = 0; i < n / 3; ++i) {
    if (i >= PyList_GET_SIZE(models)) Py_RETURN_FALSE;  // (an attribute of the user's own may have changed the list)
    PyObject* m = PyList_GET_ITEM(models, i);
    Py_INCREF(m);
    const int same = HoldsArrays(m, &PyTuple_GET_ITEM(source, 3 * i), addresses + 24 * i);
    Py_DECREF(m);
    if (same < 0) return nullptr;
    if (same == 0) Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
}

PyMethodDef g_methods[] = {
  {"holds", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(Holds)), METH_FASTCALL,
   "Whether the models hold the source's tensors, at these addresses."},
  {nullptr, nullptr, 0, nullptr}};
// LBK_MODULE: the module's name, which tells the torch it is compiled for (build.py)
#define LBK_TEXT_(x) #x
#define LBK_TEXT(x) LBK_TEXT_(x)
#define LBK_JOIN_(a, b) a##b
#define LBK_JOIN(a, b) LBK_JOIN_(a, b)

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, LBK_TEXT(LBK_MODULE), nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC LBK_JOIN(PyInit_, LBK_MODULE)()
{
  const char* names[3] = {"leaf_value", "feature", "split_value"};
  for (int i = 0; i < 3; ++i) {
    g_names[i] = PyUnicode_InternFromString(names[i]);
    if (g_names[i] == nullptr) return nullptr;
  }
  return PyModule_Create(&g_module);
}
