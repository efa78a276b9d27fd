// Small calls from Python without the interpreter between the check of the arguments and the launch: lm2exp and lt2exp on
// ordinary CUDA tensors, for the sizes that one launch of the direct kernels takes.  A call of 4 us on the device took 17 us
// of Python (shape and stride objects, ctypes conversions); here 5.
//
// Both functions return None, having done nothing, for every call that is not such a one: other tensor types and modes,
// wrong shapes, larger problems.  The Python code behind them then does what it would have done without them.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/triturus_b200.h"

namespace {

// No tracing, no transform (vmap, grad, functionalisation) and no Python mode that would want to see the operations.
bool plain_mode() {
  using c10::DispatchKey;
  const c10::DispatchKeySet inc = c10::impl::tls_local_dispatch_key_set().included_;
  return !inc.has(DispatchKey::Python) && !inc.has(DispatchKey::Tracer) && !inc.has(DispatchKey::Functionalize) &&
         !inc.has(DispatchKey::FuncTorchDynamicLayerFrontMode) && !inc.has(DispatchKey::FuncTorchDynamicLayerBackMode) &&
         !at::impl::torch_function_mode_enabled();
}

// A float32 CUDA tensor that is nothing but its storage, shape and strides: the dispatch keys are those of an ordinary (or an
// inference) tensor, so no wrapper, lazy conjugation or negation, quantisation, subclass.
const at::Tensor* plain_tensor(PyObject* o, int64_t dim) {
  using c10::DispatchKey;
  static const c10::DispatchKeySet ordinary(
      {DispatchKey::CUDA, DispatchKey::AutogradCUDA, DispatchKey::ADInplaceOrView, DispatchKey::AutocastCUDA});
  static const c10::DispatchKeySet inference({DispatchKey::CUDA, DispatchKey::AutocastCUDA});
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  const c10::DispatchKeySet ks = t.key_set();
  if (ks != ordinary && ks != inference) return nullptr;
  if (t.scalar_type() != at::kFloat || t.layout() != at::kStrided || t.dim() != dim || t.numel() == 0) return nullptr;
  return &t;
}

bool int_arg(PyObject* o, int* v) {
  const long x = PyLong_AsLong(o);
  if (x == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  *v = static_cast<int>(x);
  return *v == x;
}

struct ThreadsRun {  // without the interpreter lock, for the time of a launch: it waits where the queue of the stream is full
  PyThreadState* state = PyEval_SaveThread();
  ~ThreadsRun() { PyEval_RestoreThread(state); }
};

PyObject* none() { Py_RETURN_NONE; }

at::Tensor new_result(const at::Tensor& like, int64_t r, int64_t i, int64_t k) {
  return at::empty({r, i, k}, at::TensorOptions().dtype(at::kFloat).device(like.device()));
}

// Set by the Python side.
PyObject* error_class = nullptr;  // what it raises for a code of the library
double copy_flop_rows = 0.0;      // problems of more operations than this get a padded copy of an operand that no tensor map
double copy_flop_strided = 0.0;   // describes: of rows of consecutive floats, and of other views

PyObject* failed(const char* what, int rc) {
  PyErr_Format(error_class != nullptr ? error_class : PyExc_RuntimeError, "%s failed with code %d: %s", what, rc, triturus_b200_strerror(rc));
  return nullptr;
}

// lm2exp(a, b, precision, variant)
PyObject* lm2exp(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  int precision, variant;
  if (nargs != 4 || !int_arg(args[2], &precision) || !int_arg(args[3], &variant) || variant != 0 || !plain_mode()) return none();
  const at::Tensor* a = plain_tensor(args[0], 3);
  const at::Tensor* b = a != nullptr ? plain_tensor(args[1], 3) : nullptr;
  if (b == nullptr || a->device() != b->device() || a->get_device() != c10::cuda::current_device()) return none();
  const int64_t R = a->size(0), I = a->size(1), J = a->size(2), K = b->size(2);
  if (b->size(0) != R || b->size(1) != J) return none();
  const int64_t* as = a->strides().data();
  const int64_t* bs = b->strides().data();
  const float* ap = a->const_data_ptr<float>();
  const float* bp = b->const_data_ptr<float>();
  const int small = triturus_b200_lm2exp_small_f32(ap, bp, nullptr, R, I, J, K, as, bs, nullptr, precision, nullptr);
  if (small <= 0) return none();
  // (the copies are the Python side's; with them the call is one of the large kernels)
  const double flop = 2.0 * static_cast<double>(R) * static_cast<double>(I) * static_cast<double>(J) * static_cast<double>(K);
  if ((small & 2) != 0 && flop > (as[2] == 1 ? copy_flop_rows : copy_flop_strided)) return none();
  if ((small & 4) != 0 && flop > (bs[2] == 1 ? copy_flop_rows : copy_flop_strided)) return none();
  at::Tensor out = new_result(*a, R, I, K);
  float* op = out.mutable_data_ptr<float>();
  const auto stream = c10::cuda::getCurrentCUDAStream(a->get_device()).stream();
  int rc;
  {
    ThreadsRun unlocked;
    rc = triturus_b200_lm2exp_small_f32(ap, bp, op, R, I, J, K, as, bs, out.strides().data(), precision, stream);
  }
  if (rc != TRITURUS_B200_OK) return failed("triturus_b200_lm2exp_small_f32", rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// lt2exp(w, a, b, precision, variant)
PyObject* lt2exp(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  int precision, variant;
  if (nargs != 5 || !int_arg(args[3], &precision) || !int_arg(args[4], &variant) || !plain_mode()) return none();
  const at::Tensor* w = plain_tensor(args[0], 4);
  const at::Tensor* a = w != nullptr ? plain_tensor(args[1], 3) : nullptr;
  const at::Tensor* b = a != nullptr ? plain_tensor(args[2], 3) : nullptr;
  if (b == nullptr || w->device() != a->device() || a->device() != b->device() || a->get_device() != c10::cuda::current_device())
    return none();
  const int64_t R = w->size(0), S = w->size(1), I = w->size(2), J = w->size(3), K = a->size(2);
  if (a->size(0) != R || a->size(1) != I || b->size(0) != R || b->size(1) != J || b->size(2) != K) return none();
  const int64_t* ws = w->strides().data();
  if (I > 1 && J > 1 && ws[2] != J * ws[3]) return none();  // (I and J are not one dimension: refused, as the reference's view does)
  const float* wp = w->const_data_ptr<float>();
  const uint64_t bits = (reinterpret_cast<uintptr_t>(wp) >> 2) | static_cast<uint64_t>(J | ws[0] | ws[1] | ws[2]);
  const int odd = ws[3] != 1 || (bits & 1) != 0;
  if (triturus_b200_lt2exp_direct(R, S, I, J, K, precision, variant, odd) != 1) return none();
  at::Tensor out = new_result(*a, R, S, K);
  const float *ap = a->const_data_ptr<float>(), *bp = b->const_data_ptr<float>();
  float* op = out.mutable_data_ptr<float>();
  const auto stream = c10::cuda::getCurrentCUDAStream(a->get_device()).stream();
  int rc;
  {
    ThreadsRun unlocked;
    rc = triturus_b200_lt2exp_direct_f32(wp, ap, bp, op, R, S, I, J, K, ws, a->strides().data(), b->strides().data(), out.strides().data(),
                                         precision, nullptr, nullptr, nullptr, stream);
  }
  if (rc != TRITURUS_B200_OK) return failed("triturus_b200_lt2exp_direct_f32", rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// set_up(error_class, copy_flop_rows, copy_flop_strided)
PyObject* set_up(PyObject*, PyObject* args) {
  PyObject* cls;
  if (!PyArg_ParseTuple(args, "Odd", &cls, &copy_flop_rows, &copy_flop_strided)) return nullptr;
  Py_XDECREF(error_class);
  error_class = Py_NewRef(cls);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"set_up", set_up, METH_VARARGS, "set_up(error_class, copy_flop_rows, copy_flop_strided)"},
    {"lm2exp", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(lm2exp)), METH_FASTCALL, "lm2exp(a, b, precision, variant) -> Tensor or None"},
    {"lt2exp", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(lt2exp)), METH_FASTCALL, "lt2exp(w, a, b, precision, variant) -> Tensor or None"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Small calls of triturus_b200 from C++.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
