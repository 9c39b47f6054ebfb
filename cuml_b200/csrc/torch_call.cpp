// Native call path for device tensors: `DeviceCall(X, preds, kind, chunk_size, threshold)`.
//
// A prediction of a small batch takes a few microseconds on the GPU, so what its caller waits for
// is host work: attribute look-ups, shape checks, `torch.empty`, the current stream and a ctypes
// call cost about 8 us from Python, as much as all kernel launches together.  This object does the
// same with torch's C++ interface in under 2 us.  It handles the common call only - a CUDA tensor
// of the forest's own dtype on the forest's device with unit column stride, results to a new
// tensor or to a fitting `preds` - and returns None for everything else, which the Python code
// then converts or rejects with its usual messages.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/b2fil.h"

namespace {

using PredictFn = int (*)(const b2fil_forest*, int, const void*, int64_t, int64_t, void*, int,
                          double, void*);

struct DeviceCall {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  PredictFn predict;            // b2fil_predict of the library that owns the forest
  const b2fil_forest* forest;
  int64_t n_features, n_trees, n_outputs;
  int device;
  bool f64, vector_leaves;
};

// Shape and element type of an output kind.
struct OutSpec {
  int ndim;
  int64_t dims[3];
  at::ScalarType dtype;
};

bool out_spec(const DeviceCall* c, int64_t kind, int64_t n, OutSpec& s)
{
  s.dtype = c->f64 ? at::kDouble : at::kFloat;
  s.ndim  = 2;
  s.dims[0] = n;
  switch (kind) {
    case B2FIL_INFER_DEFAULT: s.dims[1] = c->n_outputs; return true;
    case B2FIL_INFER_PROBA2: s.dims[1] = 2; return true;
    case B2FIL_INFER_CLASS:
      s.ndim  = 1;
      s.dtype = at::kInt;
      return true;
    case B2FIL_INFER_LEAF_ID:
      s.dims[1] = c->n_trees;
      s.dtype   = at::kInt;
      return true;
    case B2FIL_INFER_PER_TREE:
      s.dims[1] = c->n_trees;
      if (c->vector_leaves) {
        s.ndim    = 3;
        s.dims[2] = c->n_outputs;
      }
      return true;
    default: return false;
  }
}

// X, preds (tensor or None), kind, chunk_size, threshold.  Returns the output tensor, None when
// the call is not one of the common ones, or the library's error code as an int.  Any of torch's
// functions may throw (a tensor subclass answers even size() in Python): the macros turn what they
// throw into the Python exception.
PyObject* device_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject*)
{
  HANDLE_TH_ERRORS
  const DeviceCall* c = reinterpret_cast<const DeviceCall*>(self);
  if (PyVectorcall_NARGS(nargsf) != 5) {
    PyErr_SetString(PyExc_TypeError, "DeviceCall takes X, preds, kind, chunk_size, threshold");
    return nullptr;
  }
  if (!THPVariable_Check(args[0])) Py_RETURN_NONE;
  const at::Tensor& X = THPVariable_Unpack(args[0]);
  const auto want     = c->f64 ? at::kDouble : at::kFloat;
  if (!X.is_cuda() || X.layout() != at::kStrided || X.dim() != 2 || X.scalar_type() != want ||
      X.get_device() != c->device || X.size(1) != c->n_features || X.stride(1) != 1)
    Py_RETURN_NONE;
  const int64_t kind  = PyLong_AsLongLong(args[2]);
  const int64_t chunk = PyLong_AsLongLong(args[3]);
  const double thr    = PyFloat_AsDouble(args[4]);
  if (PyErr_Occurred()) return nullptr;
  const int64_t n = X.size(0);
  OutSpec s;
  if (!out_spec(c, kind, n, s)) Py_RETURN_NONE;
  const at::IntArrayRef dims(s.dims, s.ndim);
  const void* from      = X.const_data_ptr();
  const int64_t stride  = X.stride(0);
  at::TensorBase made;
  const bool given = args[1] != Py_None;
  if (given) {
    if (!THPVariable_Check(args[1])) Py_RETURN_NONE;
    const at::Tensor& out = THPVariable_Unpack(args[1]);
    if (out.sizes() != dims || out.scalar_type() != s.dtype || !out.is_cuda() ||
        !out.is_contiguous())
      Py_RETURN_NONE;
    made = out;
  } else {
    made = at::detail::empty_cuda(dims, s.dtype, X.device(), std::nullopt);
  }
  void* to     = made.mutable_data_ptr();
  void* stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(c->device)).stream();
  int rc;
  // (nothing in here throws: the lock has to come back)
  Py_BEGIN_ALLOW_THREADS;
  rc = c->predict(c->forest, static_cast<int>(kind), from, n, stride, to, static_cast<int>(chunk), thr,
                  stream);
  Py_END_ALLOW_THREADS;
  if (rc != B2FIL_OK) return PyLong_FromLong(rc);
  if (given) return Py_NewRef(args[1]);
  return THPVariable_Wrap(std::move(made));
  END_HANDLE_TH_ERRORS
}

// DeviceCall(predict_address, forest_address, n_features, n_trees, n_outputs, device, f64, vector)
PyObject* device_call_new(PyTypeObject* type, PyObject* args, PyObject*)
{
  unsigned long long predict = 0, forest = 0;
  long long nf = 0, nt = 0, no = 0;
  int device = 0, f64 = 0, vec = 0;
  if (!PyArg_ParseTuple(args, "KKLLLipp", &predict, &forest, &nf, &nt, &no, &device, &f64, &vec))
    return nullptr;
  DeviceCall* c = reinterpret_cast<DeviceCall*>(type->tp_alloc(type, 0));
  if (!c) return nullptr;
  c->vectorcall    = device_call;
  c->predict       = reinterpret_cast<PredictFn>(static_cast<uintptr_t>(predict));
  c->forest        = reinterpret_cast<const b2fil_forest*>(static_cast<uintptr_t>(forest));
  c->n_features    = nf;
  c->n_trees       = nt;
  c->n_outputs     = no;
  c->device        = device;
  c->f64           = f64 != 0;
  c->vector_leaves = vec != 0;
  return reinterpret_cast<PyObject*>(c);
}

PyTypeObject device_call_type = [] {
  PyTypeObject t         = {PyVarObject_HEAD_INIT(nullptr, 0)};
  t.tp_name              = "b2fil_torch.DeviceCall";
  t.tp_basicsize         = sizeof(DeviceCall);
  t.tp_flags             = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  t.tp_vectorcall_offset = offsetof(DeviceCall, vectorcall);
  t.tp_call              = PyVectorcall_Call;
  t.tp_new               = device_call_new;
  t.tp_doc               = "Predict call of one forest on CUDA tensors.";
  return t;
}();

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "b2fil_torch",
                          "Native call path of libb2fil for torch tensors.", -1, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_b2fil_torch()
{
  if (PyType_Ready(&device_call_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module_def);
  if (!m) return nullptr;
  if (PyModule_AddObjectRef(m, "DeviceCall", reinterpret_cast<PyObject*>(&device_call_type)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
