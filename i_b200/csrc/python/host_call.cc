// Native half of Component.into / exec_numpy for NumPy arrays (ilang.py): the counterpart of
// cuda_call.cc for host buffers, with no dependency beyond Python's own C API.  It handles the
// common case, every argument a C-contiguous float32 ndarray, and returns None before doing
// anything otherwise; the caller then takes the general route, which also converts and words the
// errors.  Through ctypes the same marshalling took 25-30 us a call (exec_numpy describes its
// inputs twice).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstring>

#include "i.h"

namespace {

struct Library {
  decltype(&i_exec_into) exec_into = nullptr;
  decltype(&i_output_count) output_count = nullptr;
  decltype(&i_output_ranks) output_ranks = nullptr;
  decltype(&i_output_shapes) output_shapes = nullptr;
  decltype(&i_error) error = nullptr;
} g_lib;
PyObject* g_ndarray = nullptr;     // numpy.ndarray, numpy.empty, numpy.float32: held for good
PyObject* g_empty = nullptr;
PyObject* g_float32 = nullptr;

constexpr int kMostTensors = 16, kMostRank = 8;

// Up to kMostTensors arrays as the runtime takes them, their buffers held until destruction.
struct Described {
  i_tensor tensors[kMostTensors];
  size_t extents[kMostTensors][kMostRank];
  Py_buffer views[kMostTensors];
  int count = 0;

  ~Described() {
    for (int i = 0; i < count; ++i) PyBuffer_Release(&views[i]);
  }
  bool add(PyObject* o, bool writable) {
    if (count == kMostTensors || reinterpret_cast<PyObject*>(Py_TYPE(o)) != g_ndarray) return false;
    Py_buffer& v = views[count];
    if (PyObject_GetBuffer(o, &v, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT | (writable ? PyBUF_WRITABLE : 0))) {
      PyErr_Clear();
      return false;
    }
    if (v.ndim > kMostRank || v.itemsize != 4 || !v.format || std::strcmp(v.format, "f") != 0) {
      PyBuffer_Release(&v);
      return false;
    }
    for (int d = 0; d < v.ndim; ++d) extents[count][d] = static_cast<size_t>(v.shape[d]);
    tensors[count] = i_tensor{static_cast<const float*>(v.buf), extents[count], static_cast<size_t>(v.ndim)};
    ++count;
    return true;
  }
};

bool describe_all(PyObject* tuple, Described* out, bool writable) {
  const Py_ssize_t n = PyTuple_GET_SIZE(tuple);
  for (Py_ssize_t i = 0; i < n; ++i)
    if (!out->add(PyTuple_GET_ITEM(tuple, i), writable)) return false;
  return true;
}

PyObject* fail() {
  const char* message = g_lib.error();
  PyErr_SetString(PyExc_RuntimeError, message ? message : "i-core error");
  return nullptr;
}

int run(const i_program* program, const Described& in, const Described& out) {
  i_tensor_mut outputs[kMostTensors];
  for (int o = 0; o < out.count; ++o)
    outputs[o] = i_tensor_mut{const_cast<float*>(out.tensors[o].data), out.tensors[o].shape, out.tensors[o].rank};
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_lib.exec_into(program, in.tensors, static_cast<size_t>(in.count), outputs, static_cast<size_t>(out.count));
  Py_END_ALLOW_THREADS
  return rc;
}

// bind(exec_into, output_count, output_ranks, output_shapes, error, ndarray, empty, float32)
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long p[5];
  PyObject *nd, *empty, *f32;
  if (!PyArg_ParseTuple(args, "KKKKKOOO", &p[0], &p[1], &p[2], &p[3], &p[4], &nd, &empty, &f32)) return nullptr;
  g_lib.exec_into = reinterpret_cast<decltype(g_lib.exec_into)>(p[0]);
  g_lib.output_count = reinterpret_cast<decltype(g_lib.output_count)>(p[1]);
  g_lib.output_ranks = reinterpret_cast<decltype(g_lib.output_ranks)>(p[2]);
  g_lib.output_shapes = reinterpret_cast<decltype(g_lib.output_shapes)>(p[3]);
  g_lib.error = reinterpret_cast<decltype(g_lib.error)>(p[4]);
  g_ndarray = Py_NewRef(nd);
  g_empty = Py_NewRef(empty);
  g_float32 = Py_NewRef(f32);
  Py_RETURN_NONE;
}

const i_program* program_of(PyObject* o) { return static_cast<const i_program*>(PyLong_AsVoidPtr(o)); }

// into(program, outputs, inputs): as in cuda_call.cc.
PyObject* into(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3 || !g_ndarray || !PyTuple_Check(args[2])) Py_RETURN_NONE;
  PyObject* given = args[1];
  Described in, out;
  if (!describe_all(args[2], &in, false)) Py_RETURN_NONE;
  PyObject* many = nullptr;
  if (PyTuple_Check(given) || PyList_Check(given)) {
    many = PySequence_Tuple(given);
    if (!many) return nullptr;
  }
  if (!(many ? describe_all(many, &out, true) : out.add(given, true)) || in.count + out.count == 0) {
    Py_XDECREF(many);
    Py_RETURN_NONE;
  }
  if (run(program_of(args[0]), in, out)) {
    Py_XDECREF(many);
    return fail();
  }
  if (!many) return Py_NewRef(given);
  if (PyTuple_GET_SIZE(many) != 1) return many;
  PyObject* only = Py_NewRef(PyTuple_GET_ITEM(many, 0));
  Py_DECREF(many);
  return only;
}

// exec(program, inputs): allocates the outputs and runs; what exec_numpy returns.
PyObject* exec(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2 || !g_ndarray || !PyTuple_Check(args[1])) Py_RETURN_NONE;
  Described in, out;
  if (!describe_all(args[1], &in, false) || in.count == 0) Py_RETURN_NONE;
  const i_program* program = program_of(args[0]);
  const size_t count = g_lib.output_count(program);
  if (count == 0 || count > kMostTensors) Py_RETURN_NONE;
  size_t ranks[kMostTensors], shapes[kMostTensors][kMostRank];
  size_t* rows[kMostTensors];
  if (g_lib.output_ranks(program, ranks)) return fail();
  for (size_t o = 0; o < count; ++o) {
    if (ranks[o] > kMostRank) Py_RETURN_NONE;
    rows[o] = shapes[o];
  }
  if (g_lib.output_shapes(program, in.tensors, static_cast<size_t>(in.count), rows)) return fail();
  PyObject* made = PyTuple_New(static_cast<Py_ssize_t>(count));
  if (!made) return nullptr;
  for (size_t o = 0; o < count; ++o) {
    PyObject* dims = PyTuple_New(static_cast<Py_ssize_t>(ranks[o]));
    for (size_t d = 0; dims && d < ranks[o]; ++d)
      PyTuple_SET_ITEM(dims, static_cast<Py_ssize_t>(d), PyLong_FromSize_t(shapes[o][d]));
    PyObject* array = dims ? PyObject_CallFunctionObjArgs(g_empty, dims, g_float32, nullptr) : nullptr;
    Py_XDECREF(dims);
    if (array) PyTuple_SET_ITEM(made, static_cast<Py_ssize_t>(o), array);
    if (!array || !out.add(array, true)) {
      Py_DECREF(made);
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "numpy.empty did not return a float32 array");
      return nullptr;
    }
  }
  if (run(program, in, out)) {
    Py_DECREF(made);
    return fail();
  }
  if (count != 1) return made;
  PyObject* only = Py_NewRef(PyTuple_GET_ITEM(made, 0));
  Py_DECREF(made);
  return only;
}

PyMethodDef kMethods[] = {
    {"bind", bind, METH_VARARGS, "Addresses of the runtime's entry points, and what of NumPy is used."},
    {"into", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(into)), METH_FASTCALL,
     "Run into given NumPy arrays."},
    {"exec", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(exec)), METH_FASTCALL,
     "Run into new NumPy arrays."},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host_call", "Calls with NumPy arrays, without ctypes.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_call(void) { return PyModule_Create(&kModule); }
