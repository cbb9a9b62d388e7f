// The Python module beside the ops, a library of its own: gnb200_torch.so is loaded by libtorch programs without Python too.
//
// plain_call(x, weight, bias, num_groups, eps, act, num_channels) -> tensor, or None where the module's Python code has
// to look at the call: anything but exact tensors and parameters, a torch-function mode, other argument types, a shape that it
// refuses.  Called without torch.ops' argument matching, which took 3 us.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <utility>

#include "gn_torch.h"

namespace {

const at::Tensor* exact_tensor(PyObject* o) {
  if (Py_TYPE(o) != (PyTypeObject*)THPVariableClass && Py_TYPE(o) != (PyTypeObject*)ParameterClass) return nullptr;
  return &THPVariable_Unpack(o);
}

PyObject* plain_call(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 7 || !PyLong_CheckExact(args[3]) || !PyFloat_CheckExact(args[4]) || !PyLong_CheckExact(args[5]) ||
      !PyLong_CheckExact(args[6]) || at::impl::torch_function_mode_enabled())
    Py_RETURN_NONE;
  const at::Tensor *x = exact_tensor(args[0]), *w = exact_tensor(args[1]), *b = exact_tensor(args[2]);
  if (!x || !w || !b) Py_RETURN_NONE;
  const long long G = PyLong_AsLongLong(args[3]), act = PyLong_AsLongLong(args[5]), C = PyLong_AsLongLong(args[6]);
  if (PyErr_Occurred()) return nullptr;
  if (!x->is_cuda() || x->dim() < 3 || x->size(1) != C) Py_RETURN_NONE;
  const double eps = PyFloat_AS_DOUBLE(args[4]);
  at::Tensor y;
  {
    pybind11::gil_scoped_release no_gil;
    y = gnb200_ops::group_norm_act_direct(*x, *w, *b, G, eps, act);
  }
  if (!y.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {{"plain_call", (PyCFunction)(void (*)())plain_call, METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "gnb200_python", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_gnb200_python(void) { return PyModule_Create(&kModule); }
