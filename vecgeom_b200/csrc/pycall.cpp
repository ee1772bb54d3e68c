// pycall.cpp -- the Python side of one vgb_batch call on torch tensors.
//
// A batch call on a few thousand points takes the GPU 2 to 5 us.  Taking its arrays
// apart in Python (contiguity, addresses, lengths, types of up to nine tensors),
// converting sixteen ctypes arguments and asking the driver what kind of memory two of
// them are took the host 9.6 (four Python calls a tensor, 1 us a driver query; now 3.8,
// of which the launch is more than half).  batch() does the first two here, from the tensors'
// own fields, and calls vgb_batch_device where the tensors say that they are all on one GPU.
//
// It handles the plain case only: every array a torch.Tensor itself, contiguous, with
// the lengths and types the call needs, and all of them on one device.  For anything
// else (numpy arrays, subclasses, tensors without storage, a wrong length, a mix of
// devices, an empty batch) it returns None without calling, and the caller's general
// path does the call or raises its errors.  Nothing is kept between calls.
//
// The module is only good for the torch and the Python it was built with: it names the
// one (torch_version) for its loader to compare and refuses to load in another of the other.
#include <Python.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <string>

#include "../../include/vgb.h"

#define VGB_TEXT(x) #x
#define VGB_TEXT_OF(x) VGB_TEXT(x)

namespace {

using BatchFn = decltype(&vgb_batch);

// A contiguous tensor of n rows (at_least: or more) and, when type is given, of that
// type; nullptr where it is anything else.
const at::Tensor *plain(PyObject *o, int64_t n, bool at_least, const at::ScalarType *type) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor &t = THPVariable_Unpack(o);
  if (!t.has_storage() || t.layout() != at::kStrided || t.dim() < 1) return nullptr;
  const int64_t len = t.size(0);
  if (at_least ? len < n : len != n) return nullptr;
  if (type && t.scalar_type() != *type) return nullptr;
  return t.is_contiguous() ? &t : nullptr;
}

// batch(vgb_batch, vgb_batch_device, geometry, placed, op, x, y, z, dx, dy, dz, step_max,
// out, aux, daughter, precision, stream): the status, or None.  The functions and the
// geometry are addresses; dx, step_max and aux may be None.
PyObject *batch(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
  if (nargs != 17) {
    PyErr_SetString(PyExc_TypeError, "batch takes 17 arguments");
    return nullptr;
  }
  if (!THPVariable_CheckExact(a[5])) Py_RETURN_NONE;
  try {
    const at::ScalarType f8 = at::kDouble, i4 = at::kInt;
    const at::Tensor &x = THPVariable_Unpack(a[5]);
    const int64_t n = x.dim() > 0 ? x.size(0) : 0;
    const at::Tensor *t[9] = {};
    bool ok = n > 0;
    for (int k = 0; k < 3 && ok; ++k) ok = (t[k] = plain(a[5 + k], n, false, &f8));
    if (a[8] != Py_None)
      for (int k = 3; k < 6 && ok; ++k) ok = (t[k] = plain(a[5 + k], n, false, &f8));
    if (a[11] != Py_None && ok) ok = (t[6] = plain(a[11], n, true, &f8));
    if (ok) ok = (t[7] = plain(a[12], n, true, nullptr));
    if (a[13] != Py_None && ok) ok = (t[8] = plain(a[13], n, true, &i4));
    for (int k = 1; k < 9 && ok; ++k) ok = !t[k] || t[k]->device() == t[0]->device();
    if (!ok) Py_RETURN_NONE;
    const bool device = t[0]->is_cuda();
    const auto fn = reinterpret_cast<BatchFn>(PyLong_AsVoidPtr(a[device ? 1 : 0]));
    const auto g = static_cast<const vgb_geometry *>(PyLong_AsVoidPtr(a[2]));
    const long placed = PyLong_AsLong(a[3]), op = PyLong_AsLong(a[4]);
    const long daughter = PyLong_AsLong(a[14]), precision = PyLong_AsLong(a[15]);
    void *stream = a[16] == Py_None ? nullptr : PyLong_AsVoidPtr(a[16]);
    if (PyErr_Occurred() || placed != (int32_t)placed || op != (int32_t)op ||
        daughter != (int32_t)daughter || precision != (int32_t)precision) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    void *p[9];
    for (int k = 0; k < 9; ++k) p[k] = t[k] ? t[k]->data_ptr() : nullptr;
    auto d = [&](int k) { return static_cast<const double *>(p[k]); };
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = fn(g, (int32_t)placed, (int32_t)op, n, d(0), d(1), d(2), d(3), d(4), d(5), d(6), p[7],
                static_cast<int32_t *>(p[8]), (int32_t)daughter, (int32_t)precision, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
  } catch (const std::exception &) {  // a tensor whose data may not be asked for
    Py_RETURN_NONE;
  }
}

PyMethodDef methods[] = {{"batch", reinterpret_cast<PyCFunction>(
                                       reinterpret_cast<void (*)()>(batch)),
                          METH_FASTCALL, "one vgb_batch call, or None"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pycall", nullptr, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pycall() {
  const std::string built = std::to_string(PY_MAJOR_VERSION) + "." + std::to_string(PY_MINOR_VERSION);
  if (std::string(Py_GetVersion()).rfind(built + ".", 0) != 0) {
    PyErr_SetString(PyExc_ImportError, ("built for Python " + built).c_str());
    return nullptr;
  }
  PyObject *m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "torch_version", VGB_TEXT_OF(VGB_TORCH_VERSION)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
