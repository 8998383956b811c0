// Native half of Component.into / exec_torch for CUDA tensors (ilang.py).
//
// What bounds a small call is the host: describing four tensors through ctypes (a shape array, a
// struct and a few attribute look-ups each) took 14-18 us of Python where the launch itself takes
// two.  Here the tensors are read through torch's own C++ type, so a call costs about 1 us besides
// the runtime's.  The functions handle the common case only: every argument a dense, contiguous float32
// CUDA tensor with memory of its own, on one device.  For anything else (sparse layouts, fake tensors and
// other subclasses that dispatch in Python, functorch's wrappers under vmap or grad) they return None
// before doing anything, and the caller takes the general route, which also words the errors.  What torch
// throws on the way becomes the Python exception it stands for: nothing may leave a C function.
//
// The library is reached through function addresses handed over once (bind), so it stays the one
// ilang.py loaded.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include "i_b200.h"

namespace {

struct Library {
  decltype(&i_b200_exec_into) exec_into = nullptr;
  decltype(&i_output_count) output_count = nullptr;
  decltype(&i_output_ranks) output_ranks = nullptr;
  decltype(&i_output_shapes) output_shapes = nullptr;
  decltype(&i_error) error = nullptr;
} g_lib;

constexpr int kMostTensors = 16, kMostRank = 8;

// Up to kMostTensors tensors as the runtime takes them; the extents live here.
struct Described {
  i_tensor tensors[kMostTensors];
  size_t extents[kMostTensors][kMostRank];
  int count = 0;

  // False when `t` is not what this file handles; `device` is the first tensor's, or -1.
  // The address of an output is asked for as one to write to: a lazy clone then gets memory of its own.
  bool add(const at::Tensor& t, int* device, bool output) {
    if (count == kMostTensors || !t.defined() || !t.is_cuda() || t.scalar_type() != at::kFloat) return false;
    // Before anything that needs a storage: wrappers have none, fake tensors dispatch in Python.
    if (t.layout() != at::kStrided || !t.has_storage() || t.key_set().has(c10::DispatchKey::Python)) return false;
    if (t.dim() > kMostRank || !t.is_contiguous()) return false;
    if (*device < 0) *device = t.get_device();
    if (t.get_device() != *device) return false;
    const auto sizes = t.sizes();
    for (size_t d = 0; d < sizes.size(); ++d) extents[count][d] = static_cast<size_t>(sizes[d]);
    tensors[count] = i_tensor{static_cast<const float*>(output ? t.mutable_data_ptr() : t.const_data_ptr()), extents[count],
                              sizes.size()};
    ++count;
    return true;
  }
  bool add(PyObject* o, int* device, bool output) {
    return THPVariable_Check(o) && add(THPVariable_Unpack(o), device, output);
  }
};

bool describe_all(PyObject* tuple, Described* out, int* device, bool outputs) {
  const Py_ssize_t n = PyTuple_GET_SIZE(tuple);
  for (Py_ssize_t i = 0; i < n; ++i)
    if (!out->add(PyTuple_GET_ITEM(tuple, i), device, outputs)) return false;
  return true;
}

PyObject* fail() {
  const char* message = g_lib.error();
  PyErr_SetString(PyExc_RuntimeError, message ? message : "i-core error");
  return nullptr;
}

// Queues the program on torch's current stream of `device`; 0, or -1 with the library's message set.
int launch(const i_program* program, const Described& in, const Described& out, int device) {
  i_tensor_mut outputs[kMostTensors];
  for (int o = 0; o < out.count; ++o)
    outputs[o] = i_tensor_mut{const_cast<float*>(out.tensors[o].data), out.tensors[o].shape, out.tensors[o].rank};
  const c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device)));
  void* stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_lib.exec_into(program, in.tensors, static_cast<size_t>(in.count), outputs,
                       static_cast<size_t>(out.count), stream);
  Py_END_ALLOW_THREADS
  return rc;
}

// bind(exec_into, output_count, output_ranks, output_shapes, error): addresses in the loaded library.
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long p[5];
  if (!PyArg_ParseTuple(args, "KKKKK", &p[0], &p[1], &p[2], &p[3], &p[4])) return nullptr;
  g_lib.exec_into = reinterpret_cast<decltype(g_lib.exec_into)>(p[0]);
  g_lib.output_count = reinterpret_cast<decltype(g_lib.output_count)>(p[1]);
  g_lib.output_ranks = reinterpret_cast<decltype(g_lib.output_ranks)>(p[2]);
  g_lib.output_shapes = reinterpret_cast<decltype(g_lib.output_shapes)>(p[3]);
  g_lib.error = reinterpret_cast<decltype(g_lib.error)>(p[4]);
  Py_RETURN_NONE;
}

const i_program* program_of(PyObject* o) { return static_cast<const i_program*>(PyLong_AsVoidPtr(o)); }

// into(program, outputs, inputs): outputs is a tensor, or a tuple or list of tensors; inputs a tuple.
// Returns what Component.into returns, or None when the call is not of this file's kind.
PyObject* into(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3 || !PyTuple_Check(args[2])) Py_RETURN_NONE;
  try {
    PyObject* given = args[1];
    int device = -1;
    Described in, out;
    if (!describe_all(args[2], &in, &device, false)) Py_RETURN_NONE;
    THPObjectPtr many;                   // the outputs as a tuple
    if (PyTuple_Check(given) || PyList_Check(given)) {
      many = PySequence_Tuple(given);
      if (!many) return nullptr;
    }
    const bool described = many ? describe_all(many, &out, &device, true) : out.add(given, &device, true);
    if (!described || device < 0) Py_RETURN_NONE;
    if (launch(program_of(args[0]), in, out, device)) return fail();
    if (!many) return Py_NewRef(given);
    return PyTuple_GET_SIZE(many.get()) == 1 ? Py_NewRef(PyTuple_GET_ITEM(many.get(), 0)) : many.release();
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

// exec(program, inputs): allocates the outputs and runs; what exec_torch returns, or None when the
// call is not of this file's kind.
PyObject* exec(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2 || !PyTuple_Check(args[1])) Py_RETURN_NONE;
  try {
    int device = -1;
    Described in, out;
    if (!describe_all(args[1], &in, &device, false) || device < 0) Py_RETURN_NONE;
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
    THPObjectPtr made;                   // several outputs as a tuple
    if (count != 1 && !(made = PyTuple_New(static_cast<Py_ssize_t>(count)))) return nullptr;
    at::Tensor first;
    const auto options = at::TensorOptions().dtype(at::kFloat).device(at::kCUDA, static_cast<c10::DeviceIndex>(device));
    for (size_t o = 0; o < count; ++o) {
      int64_t dims[kMostRank];
      for (size_t d = 0; d < ranks[o]; ++d) dims[d] = static_cast<int64_t>(shapes[o][d]);
      at::Tensor t = at::empty(at::IntArrayRef(dims, ranks[o]), options);
      if (!out.add(t, &device, true)) Py_RETURN_NONE;      // a dispatch mode made something else of it
      if (made) {
        PyObject* wrapped = THPVariable_Wrap(t);
        if (!wrapped) return nullptr;
        PyTuple_SET_ITEM(made.get(), static_cast<Py_ssize_t>(o), wrapped);
      } else {
        first = std::move(t);
      }
    }
    if (launch(program, in, out, device)) return fail();
    return made ? made.release() : THPVariable_Wrap(first);
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

PyMethodDef kMethods[] = {
    {"bind", bind, METH_VARARGS, "Addresses of the runtime's entry points."},
    {"into", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(into)), METH_FASTCALL,
     "Run into given CUDA tensors."},
    {"exec", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(exec)), METH_FASTCALL,
     "Run into new CUDA tensors."},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_cuda_call", "Calls with CUDA tensors, without ctypes.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__cuda_call(void) { return PyModule_Create(&kModule); }
