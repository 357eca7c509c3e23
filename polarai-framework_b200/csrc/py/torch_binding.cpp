// The builtins called with torch tensors, in native code: what DeviceBuiltins and DeviceExecutor do per
// call - check the tensors, find their pointers and torch's current stream, call the C ABI - without
// the interpreter.  Through ctypes a call spent 3 to 5 us on that beside 2 us for the launch itself; here it
// is about 0.3 us, 0.1 of it for the interpreter's lock.
//
// Every function returns True when it has launched.  Anything out of the ordinary - an argument that is no
// contiguous float32 CUDA tensor, sizes that do not agree, a status other than 0 - makes it return
// False without an exception, and the caller takes its checked Python path, which raises, or launches what it can read and
// write within its tensors.  That goes for what torch throws as well (a tensor without storage, as tracing makes them, has
// no data pointer): a C++ exception must not reach the interpreter, where it would end the process.
//
// The C ABI is called without the interpreter's lock, as through ctypes: a launch waits when the GPU's queue is full,
// which may take until another thread has launched what the kernels at its head wait for.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <polar_b200.h>

#include <algorithm>
#include <exception>
#include <vector>

namespace {

// The tensors of one call: contiguous float32 on one CUDA device.
class Call {
public:
  Call(PyObject* const* args, Py_ssize_t given, Py_ssize_t expected) : args_(args), ok_(given == expected) {}
  const at::Tensor* tensor(int i) {
    if (!ok_) return nullptr;
    if (!THPVariable_Check(args_[i])) {
      ok_ = false;
      return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(args_[i]);
    if (!t.defined() || !t.is_cuda() || t.scalar_type() != at::kFloat || !t.is_contiguous() ||
        (device_ >= 0 && t.get_device() != device_)) {
      ok_ = false;
      return nullptr;
    }
    device_ = t.get_device();
    return &t;
  }
  float scalar(int i) {
    if (!ok_) return 0.f;
    const double v = PyFloat_AsDouble(args_[i]);
    if (v == -1.0 && PyErr_Occurred()) {
      PyErr_Clear();
      ok_ = false;
    }
    return (float)v;
  }
  uint64_t whole(int i) {
    if (!ok_) return 0;
    const long long v = PyLong_AsLongLong(args_[i]);
    if (v < 0) {                                           // negative, or not a whole number
      PyErr_Clear();
      ok_ = false;
      return 0;
    }
    return (uint64_t)v;
  }
  void require(bool condition) { ok_ = ok_ && condition; }
  bool ok() const { return ok_; }
  void* stream() const { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device_).stream(); }

private:
  PyObject* const* args_;
  bool ok_;
  int device_ = -1;
};

// Runs f without the interpreter's lock.  What f needs of Python objects is looked up before.
template <class F>
auto unlocked(F f) {
  PyThreadState* state = PyEval_SaveThread();
  auto r = f();
  PyEval_RestoreThread(state);
  return r;
}

float* data(const at::Tensor* t) { return static_cast<float*>(t->data_ptr()); }
uint64_t numel(const at::Tensor* t) { return (uint64_t)t->numel(); }
PyObject* answer(bool launched) { return PyBool_FromLong(launched); }
template <class F, class... A>
PyObject* launched(F f, A... args) {
  return answer(unlocked([&] { return f(args...); }) == 0);
}

using Function = PyObject* (*)(PyObject*, PyObject* const*, Py_ssize_t);
template <Function F>
PyObject* declining(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  try {
    return F(self, args, n);
  } catch (const std::exception&) {
    return answer(false);
  }
}
template <Function F>
PyObject* raising(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  try {
    return F(self, args, n);
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

#define BUILTIN(name) PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t n)

BUILTIN(ffill) {
  Call c(args, n, 2);
  const float v = c.scalar(0);
  const at::Tensor* out = c.tensor(1);
  return c.ok() ? launched(polar_b200_ffill, v, data(out), numel(out), c.stream()) : answer(false);
}
BUILTIN(fadd) {
  Call c(args, n, 5);
  const at::Tensor* a = c.tensor(0);
  const float sa = c.scalar(1);
  const at::Tensor* b = c.tensor(2);
  const float sb = c.scalar(3);
  const at::Tensor* out = c.tensor(4);
  if (c.ok()) c.require(numel(a) == numel(out) && numel(b) == numel(out));
  return c.ok() ? launched(polar_b200_fadd, data(a), sa, data(b), sb, data(out), numel(out), c.stream()) : answer(false);
}
template <int (*F)(const float*, float*, uint64_t, void*)>
BUILTIN(unary) {
  Call c(args, n, 2);
  const at::Tensor *a = c.tensor(0), *out = c.tensor(1);
  if (c.ok()) c.require(numel(a) == numel(out));
  return c.ok() ? launched(F, data(a), data(out), numel(out), c.stream()) : answer(false);
}
template <int (*F)(const float*, const float*, float*, uint64_t, void*)>
BUILTIN(binary) {
  Call c(args, n, 3);
  const at::Tensor *a = c.tensor(0), *b = c.tensor(1), *out = c.tensor(2);
  if (c.ok()) c.require(numel(a) == numel(out) && numel(b) == numel(out));
  return c.ok() ? launched(F, data(a), data(b), data(out), numel(out), c.stream()) : answer(false);
}
BUILTIN(fmulconcat) {
  Call c(args, n, 3);
  const at::Tensor *g = c.tensor(0), *l = c.tensor(1), *out = c.tensor(2);
  if (c.ok()) c.require(numel(g) >= 1 && numel(l) == numel(out));
  return c.ok() ? launched(polar_b200_fmulconcat, data(g), data(l), data(out), numel(out), c.stream()) : answer(false);
}
BUILTIN(fsoftmax) {
  Call c(args, n, 2);
  const at::Tensor *a = c.tensor(0), *out = c.tensor(1);
  if (c.ok()) c.require(numel(a) == numel(out));
  return c.ok() ? launched(polar_b200_fsoftmax, data(a), data(out), numel(out), nullptr, 0, c.stream()) : answer(false);
}
BUILTIN(fpool) {
  Call c(args, n, 6);
  const at::Tensor* a = c.tensor(0);
  const uint64_t wh = c.whole(1), ww = c.whole(2), sh = c.whole(3), sw = c.whole(4);
  const at::Tensor* out = c.tensor(5);
  if (c.ok()) c.require(a->dim() == 2);
  if (!c.ok()) return answer(false);
  const uint64_t h = (uint64_t)a->size(0), w = (uint64_t)a->size(1);
  if (wh && ww && sh && sw && wh <= h && ww <= w && numel(out) < ((h - wh) / sh + 1) * ((w - ww) / sw + 1)) return answer(false);
  return launched(polar_b200_fpool, data(a), h, w, wh, ww, sh, sw, data(out), c.stream());
}
BUILTIN(fconv2d) {
  Call c(args, n, 3);
  const at::Tensor *a = c.tensor(0), *k = c.tensor(1), *out = c.tensor(2);
  if (c.ok()) c.require(a->dim() == 2 && k->dim() == 2);
  if (!c.ok()) return answer(false);
  const int64_t oh = a->size(0) - k->size(0) + 1, ow = a->size(1) - k->size(1) + 1;
  if (oh > 0 && ow > 0 && out->numel() < oh * ow) return answer(false);
  return launched(polar_b200_fconv2d, data(a), (uint64_t)a->size(0), (uint64_t)a->size(1), data(k), (uint64_t)k->size(0),
                  (uint64_t)k->size(1), data(out), c.stream());
}
BUILTIN(ftranspose) {
  Call c(args, n, 2);
  const at::Tensor *a = c.tensor(0), *out = c.tensor(1);
  if (c.ok()) c.require(a->dim() == 2 && numel(a) <= numel(out));
  if (!c.ok()) return answer(false);
  return launched(polar_b200_ftranspose, data(a), (uint64_t)a->size(0), (uint64_t)a->size(1), data(out), c.stream());
}
BUILTIN(fmatmul) {
  Call c(args, n, 5);
  const uint64_t tl = c.whole(0), tr = c.whole(1);
  const at::Tensor *l = c.tensor(2), *r = c.tensor(3), *out = c.tensor(4);
  if (c.ok()) c.require(tl <= 1 && tr <= 1 && l->dim() == 2 && r->dim() == 2 && out->dim() == 2);
  if (!c.ok()) return answer(false);
  const int64_t m = l->size(tl ? 1 : 0), k = l->size(tl ? 0 : 1), cols = r->size(tr ? 0 : 1);
  if (r->size(tr ? 1 : 0) != k || out->size(0) != m || out->size(1) != cols) return answer(false);
  return launched(polar_b200_fmatmul, (int)tl, (int)tr, (uint64_t)m, (uint64_t)cols, (uint64_t)k, data(l), data(r), data(out),
                  nullptr, 0, c.stream());
}

// A program's operations as Python has them: a list of (native name, address of the argument structs, their count).
bool operations(PyObject* list, std::vector<polar_b200_op>* ops) {
  if (!PyList_Check(list)) {
    PyErr_SetString(PyExc_TypeError, "expected a list of (name, address, count)");
    return false;
  }
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) {
    const char* name;
    unsigned long long address, count;
    if (!PyArg_ParseTuple(PyList_GET_ITEM(list, i), "yKK", &name, &address, &count)) return false;
    ops->push_back({name, reinterpret_cast<const polar_b200_arg*>(address), count});
  }
  return true;
}
// workspace_bytes(operations): what the most demanding one asks for.
BUILTIN(workspace_bytes) {
  std::vector<polar_b200_op> ops;
  if (n != 1 || !operations(args[0], &ops)) return nullptr;
  uint64_t need = 0;
  for (const polar_b200_op& o : ops) need = std::max<uint64_t>(need, polar_b200_launch_workspace_bytes(o.name, o.args, o.argc));
  return PyLong_FromUnsignedLongLong(need);
}
// create_program(operations, workspace address, its bytes): (status, handle).
BUILTIN(create_program) {
  std::vector<polar_b200_op> ops;
  if (n != 3 || !operations(args[0], &ops)) return nullptr;
  void* workspace = PyLong_AsVoidPtr(args[1]);
  const uint64_t bytes = PyLong_AsUnsignedLongLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  void* program = nullptr;
  const int status = polar_b200_program_create(ops.data(), ops.size(), workspace, bytes, &program);
  return Py_BuildValue("iK", status, (unsigned long long)(uintptr_t)program);
}
// run_program(handle, device index): one pass of a polar_b200_program on the device's current stream; the status.
BUILTIN(run_program) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "run_program(handle, device)");
    return nullptr;
  }
  void* handle = PyLong_AsVoidPtr(args[0]);
  const long device = PyLong_AsLong(args[1]);
  if (PyErr_Occurred()) return nullptr;
  void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
  return PyLong_FromLong(unlocked([&] { return polar_b200_program_run(handle, stream); }));
}

#define ENTRY(name, ...) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(__VA_ARGS__)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    ENTRY("ffill", declining<ffill>),
    ENTRY("fcopy", declining<unary<polar_b200_fcopy>>),
    ENTRY("fadd", declining<fadd>),
    ENTRY("fmul", declining<binary<polar_b200_fmul>>),
    ENTRY("fdivide", declining<binary<polar_b200_fdivide>>),
    ENTRY("fsigmoid", declining<unary<polar_b200_fsigmoid>>),
    ENTRY("fsigmoid_unclamped", declining<unary<polar_b200_fsigmoid_unclamped>>),
    ENTRY("flogloss", declining<binary<polar_b200_flogloss>>),
    ENTRY("fmulconcat", declining<fmulconcat>),
    ENTRY("frelu", declining<unary<polar_b200_frelu>>),
    ENTRY("fsoftmax", declining<fsoftmax>),
    ENTRY("fpool", declining<fpool>),
    ENTRY("fconv2d", declining<fconv2d>),
    ENTRY("ftranspose", declining<ftranspose>),
    ENTRY("fmatmul", declining<fmatmul>),
    ENTRY("workspace_bytes", raising<workspace_bytes>),
    ENTRY("create_program", raising<create_program>),
    ENTRY("run_program", raising<run_program>),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "polar_b200_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_polar_b200_torch(void) { return PyModule_Create(&module); }
