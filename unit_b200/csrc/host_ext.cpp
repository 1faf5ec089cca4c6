// CPython extension unit_b200._host: the host side of repeated operator calls.
//
// An operator call on a small problem is bound by the host: argument checks, the output's allocation,
// tile selection, the tensor map and the ctypes crossing took 19-27 us in Python against 3-6 us of GPU
// time.  A Launcher (one per packed weight tensor) keeps the launch plan of every geometry it has seen
// (unit_conv_plan, made once by the Python operator through the C ABI); a later call with the same
// geometry checks its tensors, allocates the output unless the call names one, points the plan at the
// buffers (unit_plan_rebind) and launches it without returning to Python.  Whatever a Launcher does not
// recognise (another device, a host tensor, a strided view, an unseen geometry, a stream that has not
// waited for the weights) it leaves to the operator's Python code by returning None, so that every
// check and every error message lives there.
//
// Calls run under the GIL up to the launch itself, which works on a copy of the plan with the GIL
// released: threads may share a Launcher.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <memory>
#include <new>
#include <vector>

#include "../../include/unit_b200.h"

namespace {

// The library's entry points, handed over by Python (which chooses the library file).
using RunFn = int (*)(const unit_conv_plan *, void *);
using RebindFn = int (*)(unit_conv_plan *, const void *, const int32_t *, const void *, void *, void *);
using LayoutFn = int (*)(const void *, void *, int32_t, int32_t, int32_t, int32_t, int32_t, int32_t, void *);
RunFn g_run = nullptr;
RebindFn g_rebind = nullptr;
LayoutFn g_pack = nullptr, g_unpack = nullptr;
int64_t g_table_version = 0;   // plans made under another tile table are not used

constexpr int64_t kNone = INT64_MIN;
constexpr int kKeyLen = 22;
constexpr size_t kMaxEntries = 64, kMaxScratch = 32;

struct Key {
  int64_t v[kKeyLen] = {};
  int n = 0;
  void push(int64_t x) { v[n++] = x; }
  bool operator==(const Key &o) const { return n == o.n && memcmp(v, o.v, sizeof(int64_t) * n) == 0; }
};

// The pointers of one call.
struct Ptrs {
  const void *x = nullptr, *bias = nullptr, *residual = nullptr;
  void *out = nullptr, *workspace = nullptr;
  bool operator==(const Ptrs &o) const {
    return x == o.x && bias == o.bias && residual == o.residual && out == o.out && workspace == o.workspace;
  }
};

struct Entry {
  Key key;
  unit_conv_plan plan;
  Ptrs at;                       // what `plan` points at; every call points it at its own buffers
  std::vector<int64_t> out_sizes;
  at::ScalarType out_type;
  int64_t c_out = 0;
  // plans that need scratch: the buffer of each stream that has called (the operators keep one per stream and never
  // free one that was handed out)
  struct Scratch { cudaStream_t stream; void *buffer; };
  bool needs_scratch = false;
  std::vector<Scratch> scratch;
  size_t next_scratch = 0;
  void *scratch_of(cudaStream_t st) const {
    for (const Scratch &s : scratch)
      if (s.stream == st) return s.buffer;
    return nullptr;
  }
  void set_scratch(cudaStream_t st, void *buffer) {
    for (Scratch &s : scratch)
      if (s.stream == st) { s.buffer = buffer; return; }
    if (scratch.size() < kMaxScratch) scratch.push_back({st, buffer});
    else scratch[next_scratch++ % kMaxScratch] = {st, buffer};
  }
};

struct Launcher {
  PyObject_HEAD
  int device;
  std::vector<cudaStream_t> *streams;               // streams that have waited for the packed weights
  std::vector<std::shared_ptr<Entry>> *entries;   // (a call keeps its entry while others evict)
};

// The current C++ exception as the Python exception that torch gives it: a failed allocation is a
// torch.OutOfMemoryError here as it is in the operators' own checks.
PyObject *raise_in_python() {
  torch::translate_exception_to_python(std::current_exception());
  return nullptr;
}

bool get_int(PyObject *o, int64_t *v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}
bool get_int_or_none(PyObject *o, int64_t *v) {
  if (o == Py_None) { *v = kNone; return true; }
  return get_int(o, v);
}
// an int, or a tuple of `n` ints
bool push_ints(Key &k, PyObject *o, int n) {
  int64_t v;
  if (get_int(o, &v)) {
    for (int i = 0; i < n; ++i) k.push(v);
    return true;
  }
  if (!PyTuple_CheckExact(o) || PyTuple_GET_SIZE(o) != n) return false;
  for (int i = 0; i < n; ++i) {
    if (!get_int(PyTuple_GET_ITEM(o, i), &v)) return false;
    k.push(v);
  }
  return true;
}
bool str_is(PyObject *o, const char *s) { return PyUnicode_CheckExact(o) && PyUnicode_CompareWithASCIIString(o, s) == 0; }

// A plain contiguous CUDA tensor of this device, or nullptr.
const at::Tensor *cuda_tensor(PyObject *o, int device) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor &t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.get_device() != device || !t.is_contiguous()) return nullptr;
  return &t;
}

// ---- geometry of each operator's call; false: not for the launcher ----
bool push_tensor(Key &k, const at::Tensor &t, int dims) {
  if (t.dim() != dims) return false;
  k.push((int64_t)t.scalar_type());
  for (int i = 0; i < dims; ++i) k.push(t.size(i));
  return true;
}
bool push_out_dtype(Key &k, PyObject *o) {
  if (str_is(o, "int32")) k.push(0);
  else if (str_is(o, "uint8")) k.push(1);
  else return false;
  return true;
}

enum Op : int64_t { OP_CONV2D = 1, OP_DENSE, OP_GEMM, OP_CONV_F16 };

// Positions of a call's arguments: every operator passes (data, bias, residual, out, options ...).
constexpr Py_ssize_t kArgData = 0, kArgBias = 1, kArgResidual = 2, kArgOut = 3, kArgOptions = 4;

bool make_key(Key &k, int64_t op, PyObject *const *a, Py_ssize_t n, const at::Tensor &x) {
  k.push(op);
  k.push(g_table_version);
  k.push(a[kArgBias] != Py_None);
  k.push(a[kArgResidual] != Py_None);
  PyObject *const *o = a + kArgOptions;
  const Py_ssize_t no = n - kArgOptions;
  int64_t v;
  switch (op) {
    case OP_CONV2D:  // stride, padding, dilation, out_layout, out_dtype, requant_shift, mul
      if (no != 7 || !push_tensor(k, x, 5) || !push_ints(k, o[0], 2) || !push_ints(k, o[1], 2) || !push_ints(k, o[2], 2)) return false;
      if (!str_is(o[3], "NCHW16c") || !push_out_dtype(k, o[4])) return false;
      if (!get_int_or_none(o[5], &v)) return false;
      k.push(v);
      if (!get_int(o[6], &v)) return false;
      k.push(v);
      return true;
    case OP_DENSE:
    case OP_GEMM:
      return no == 0 && push_tensor(k, x, 2);
    case OP_CONV_F16:  // stride_h, stride_w, out_type, padding
      if (no != 4 || !push_tensor(k, x, 5)) return false;
      if (!get_int(o[0], &v)) return false;
      k.push(v);
      if (!get_int(o[1], &v)) return false;
      k.push(v);
      return str_is(o[2], "float32") && push_ints(k, o[3], 2);
    default: return false;
  }
}

// The optional tensors of a call; false: something the operator's own checks should see.
bool optional_ptrs(const Entry &e, PyObject *const *a, int device, Ptrs &p) {
  if (a[kArgBias] != Py_None) {
    const at::Tensor *t = cuda_tensor(a[kArgBias], device);
    if (!t || t->scalar_type() != at::kInt || t->numel() != e.c_out) return false;
    p.bias = t->data_ptr();
  }
  if (a[kArgResidual] != Py_None) {
    const at::Tensor *t = cuda_tensor(a[kArgResidual], device);
    if (!t || t->scalar_type() != at::kByte || t->sizes() != at::IntArrayRef(e.out_sizes)) return false;
    p.residual = t->data_ptr();
  }
  return true;
}

std::shared_ptr<Entry> find_entry(Launcher *self, const Key &k) {
  for (const std::shared_ptr<Entry> &e : *self->entries)
    if (e->key == k) return e;
  return nullptr;
}

int launch(const unit_conv_plan &plan, cudaStream_t st) {
  unit_conv_plan mine;
  memcpy(&mine, &plan, sizeof(mine));  // (another thread may rebind the entry's plan once the GIL is released)
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_run(&mine, st);
  Py_END_ALLOW_THREADS
  return rc;
}

// call(op, data, bias, residual, out, options...) -> result tensor, None (not for the launcher) or an int
// (the status of a failed launch)
PyObject *launcher_call(Launcher *self, PyObject *const *args, Py_ssize_t nargs) {
  int64_t op;
  if (nargs < 5 || !get_int(args[0], &op)) Py_RETURN_NONE;
  PyObject *const *a = args + 1;
  const Py_ssize_t n = nargs - 1;
  try {
    if (c10::cuda::current_device() != self->device) Py_RETURN_NONE;
    const at::Tensor *x = cuda_tensor(a[kArgData], self->device);
    Key k;
    if (!x || !make_key(k, op, a, n, *x)) Py_RETURN_NONE;
    const std::shared_ptr<Entry> e = find_entry(self, k);
    if (!e) Py_RETURN_NONE;
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(self->device).stream();
    bool known = false;
    for (cudaStream_t s : *self->streams) known = known || s == st;
    if (!known) Py_RETURN_NONE;
    Ptrs p;
    p.x = x->data_ptr();
    if (e->needs_scratch && !(p.workspace = e->scratch_of(st))) Py_RETURN_NONE;
    if (!optional_ptrs(*e, a, self->device, p)) Py_RETURN_NONE;
    const bool named = a[kArgOut] != Py_None;
    at::Tensor out;
    if (named) {
      const at::Tensor *t = cuda_tensor(a[kArgOut], self->device);
      if (!t || t->scalar_type() != e->out_type || t->sizes() != at::IntArrayRef(e->out_sizes)) Py_RETURN_NONE;
      p.out = t->data_ptr();
    } else {
      out = at::Tensor(at::detail::empty_cuda(e->out_sizes, e->out_type, x->device(), std::nullopt));
      p.out = out.data_ptr();
    }
    if (!(e->at == p)) {
      if (g_rebind(&e->plan, p.x, static_cast<const int32_t *>(p.bias), p.residual, p.out, p.workspace)) Py_RETURN_NONE;
      e->at = p;
    }
    const int rc = launch(e->plan, st);
    if (rc) return PyLong_FromLong(rc);
    return named ? Py_NewRef(a[kArgOut]) : THPVariable_Wrap(std::move(out));
  } catch (...) {
    return raise_in_python();
  }
}

// Keeps the plan of the call `a` (its operator number and arguments); `result` is the tensor it writes.
void keep(Launcher *self, int64_t plan_addr, PyObject *result_obj, void *workspace, int64_t c_out, int64_t op, PyObject *const *a,
          Py_ssize_t n, cudaStream_t st) {
  const at::Tensor *x = cuda_tensor(a[kArgData], self->device);
  const at::Tensor *result = cuda_tensor(result_obj, self->device);
  Key k;
  if (!x || !result || c10::cuda::current_device() != self->device || !make_key(k, op, a, n, *x)) return;
  if (const std::shared_ptr<Entry> e = find_entry(self, k)) {  // known, but not on this stream
    if (e->needs_scratch && workspace) e->set_scratch(st, workspace);
    return;
  }
  auto fresh = std::make_shared<Entry>();
  fresh->key = k;
  fresh->c_out = c_out;
  fresh->out_sizes = result->sizes().vec();
  fresh->out_type = result->scalar_type();
  Ptrs p;
  p.x = x->data_ptr();
  p.out = result->data_ptr();
  p.workspace = workspace;
  if (!optional_ptrs(*fresh, a, self->device, p)) return;
  memcpy(&fresh->plan, reinterpret_cast<const void *>(plan_addr), sizeof(unit_conv_plan));
  fresh->at = p;
  fresh->needs_scratch = workspace != nullptr;
  if (workspace) fresh->set_scratch(st, workspace);
  auto &es = *self->entries;
  if (es.size() >= kMaxEntries) es.erase(es.begin());
  es.push_back(std::move(fresh));
}

// run(plan_address, result, workspace_address, c_out, op, data, bias, residual, out, options...): launches the plan
// that the operator made for this call and keeps it (`result` is the tensor it writes) -> None or an int
PyObject *launcher_run(Launcher *self, PyObject *const *args, Py_ssize_t nargs) {
  int64_t plan_addr, ws_addr, c_out, op;
  if (nargs < 9 || !get_int(args[0], &plan_addr) || !get_int(args[2], &ws_addr) || !get_int(args[3], &c_out) || !get_int(args[4], &op)) {
    PyErr_SetString(PyExc_TypeError, "run(plan, result, workspace, c_out, op, data, bias, residual, out, options...)");
    return nullptr;
  }
  try {
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream().stream();
    const int rc = launch(*reinterpret_cast<const unit_conv_plan *>(plan_addr), st);
    if (rc) return PyLong_FromLong(rc);
    keep(self, plan_addr, args[1], reinterpret_cast<void *>(ws_addr), c_out, op, args + 5, nargs - 5, st);
    Py_RETURN_NONE;
  } catch (...) {
    return raise_in_python();
  }
}

// The weights are ready on this stream (a cudaStream_t as an integer).
PyObject *launcher_add_stream(Launcher *self, PyObject *o) {
  int64_t v;
  if (!get_int(o, &v)) {
    PyErr_SetString(PyExc_TypeError, "a stream handle is an int");
    return nullptr;
  }
  try {
    self->streams->push_back(reinterpret_cast<cudaStream_t>(v));
  } catch (...) {
    return raise_in_python();
  }
  Py_RETURN_NONE;
}

PyObject *launcher_new(PyTypeObject *type, PyObject *args, PyObject *) {
  int device;
  if (!PyArg_ParseTuple(args, "i", &device)) return nullptr;
  Launcher *self = reinterpret_cast<Launcher *>(type->tp_alloc(type, 0));
  if (!self) return nullptr;
  self->device = device;
  try {   // (the object's memory starts as zeros, so a half-made one can be dropped)
    self->streams = new std::vector<cudaStream_t>();
    self->entries = new std::vector<std::shared_ptr<Entry>>();
  } catch (...) {
    Py_DECREF(self);
    return raise_in_python();
  }
  return reinterpret_cast<PyObject *>(self);
}
void launcher_dealloc(Launcher *self) {
  delete self->streams;
  delete self->entries;
  Py_TYPE(self)->tp_free(reinterpret_cast<PyObject *>(self));
}

PyMethodDef launcher_methods[] = {
    {"call", (PyCFunction)(void (*)())launcher_call, METH_FASTCALL, "call(op, data, bias, residual, out, options...)"},
    {"run", (PyCFunction)(void (*)())launcher_run, METH_FASTCALL, "run(plan, result, workspace, c_out, op, data, bias, residual, out, options...)"},
    {"add_stream", (PyCFunction)launcher_add_stream, METH_O, "the packed weights are ready on this stream"},
    {nullptr, nullptr, 0, nullptr}};
PyTypeObject LauncherType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- Runner: one plan with its buffers (ConvPlan.run) ----
struct Runner {
  PyObject_HEAD
  unit_conv_plan plan;
  PyObject *out;
};
PyObject *runner_new(PyTypeObject *type, PyObject *args, PyObject *) {
  long long addr;
  PyObject *out;
  if (!PyArg_ParseTuple(args, "LO", &addr, &out)) return nullptr;
  Runner *self = reinterpret_cast<Runner *>(type->tp_alloc(type, 0));
  if (!self) return nullptr;
  memcpy(&self->plan, reinterpret_cast<const void *>(addr), sizeof(self->plan));
  self->out = Py_NewRef(out);
  return reinterpret_cast<PyObject *>(self);
}
void runner_dealloc(Runner *self) {
  Py_XDECREF(self->out);
  Py_TYPE(self)->tp_free(reinterpret_cast<PyObject *>(self));
}
PyObject *runner_run(Runner *self, PyObject *) {
  try {
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream().stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_run(&self->plan, st);
    Py_END_ALLOW_THREADS
    return rc ? PyLong_FromLong(rc) : Py_NewRef(self->out);
  } catch (...) {
    return raise_in_python();
  }
}
PyMethodDef runner_methods[] = {{"run", (PyCFunction)runner_run, METH_NOARGS, "launch the plan on the current stream"},
                                {nullptr, nullptr, 0, nullptr}};
PyTypeObject RunnerType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- layout transforms: pack(x, c_block) / unpack(x, channels) -> tensor, None or an int ----
PyObject *layout_call(LayoutFn fn, PyObject *const *args, Py_ssize_t nargs, bool pack) {
  int64_t arg;
  if (nargs != 2 || !THPVariable_CheckExact(args[0])) Py_RETURN_NONE;
  try {
    const at::Tensor *x = cuda_tensor(args[0], c10::cuda::current_device());
    if (!x || x->dim() != (pack ? 4 : 5) || x->numel() == 0) Py_RETURN_NONE;
    int64_t sizes[5], n, c, h, w, cb;
    if (pack) {
      if (!get_int(args[1], &arg) || arg < 1) Py_RETURN_NONE;
      n = x->size(0); c = x->size(1); h = x->size(2); w = x->size(3); cb = arg;
      sizes[0] = n; sizes[1] = (c + cb - 1) / cb; sizes[2] = h; sizes[3] = w; sizes[4] = cb;
    } else {
      const int64_t cc = x->size(1);
      n = x->size(0); h = x->size(2); w = x->size(3); cb = x->size(4);
      if (!get_int_or_none(args[1], &arg)) Py_RETURN_NONE;
      c = arg == kNone ? cc * cb : arg;
      if (c < 1 || c > cc * cb || (c + cb - 1) / cb != cc) Py_RETURN_NONE;
      sizes[0] = n; sizes[1] = c; sizes[2] = h; sizes[3] = w;
    }
    if (n > INT32_MAX || c > INT32_MAX || h > INT32_MAX || w > INT32_MAX || cb > INT32_MAX) Py_RETURN_NONE;
    at::Tensor out(at::detail::empty_cuda(at::IntArrayRef(sizes, pack ? 5 : 4), x->scalar_type(), x->device(), std::nullopt));
    const void *src = x->data_ptr();
    void *dst = out.data_ptr();
    const int32_t eb = (int32_t)x->element_size();
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream().stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fn(src, dst, (int32_t)n, (int32_t)c, (int32_t)h, (int32_t)w, (int32_t)cb, eb, st);
    Py_END_ALLOW_THREADS
    return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(std::move(out));
  } catch (...) {
    return raise_in_python();
  }
}
PyObject *host_pack(PyObject *, PyObject *const *args, Py_ssize_t n) { return layout_call(g_pack, args, n, true); }
PyObject *host_unpack(PyObject *, PyObject *const *args, Py_ssize_t n) { return layout_call(g_unpack, args, n, false); }

// ---- module ----
PyObject *host_bind(PyObject *, PyObject *args) {
  unsigned long long run, rebind, pack, unpack;
  if (!PyArg_ParseTuple(args, "KKKK", &run, &rebind, &pack, &unpack)) return nullptr;
  g_run = reinterpret_cast<RunFn>(run);
  g_rebind = reinterpret_cast<RebindFn>(rebind);
  g_pack = reinterpret_cast<LayoutFn>(pack);
  g_unpack = reinterpret_cast<LayoutFn>(unpack);
  Py_RETURN_NONE;
}
PyObject *host_set_table_version(PyObject *, PyObject *o) {
  if (!get_int(o, &g_table_version)) {
    PyErr_SetString(PyExc_TypeError, "a version is an int");
    return nullptr;
  }
  Py_RETURN_NONE;
}

PyMethodDef host_methods[] = {
    {"bind", host_bind, METH_VARARGS, "addresses of unit_conv2d_run, unit_plan_rebind and the two layout transforms"},
    {"set_table_version", host_set_table_version, METH_O, "plans made under another tile table are no longer used"},
    {"pack", (PyCFunction)(void (*)())host_pack, METH_FASTCALL, "pack(x, c_block)"},
    {"unpack", (PyCFunction)(void (*)())host_unpack, METH_FASTCALL, "unpack(x, channels)"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef host_module = {PyModuleDef_HEAD_INIT, "_host", "Host side of repeated operator calls.", -1, host_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  LauncherType.tp_name = "unit_b200._host.Launcher";
  LauncherType.tp_basicsize = sizeof(Launcher);
  LauncherType.tp_flags = Py_TPFLAGS_DEFAULT;
  LauncherType.tp_new = launcher_new;
  LauncherType.tp_dealloc = (destructor)launcher_dealloc;
  LauncherType.tp_methods = launcher_methods;
  RunnerType.tp_name = "unit_b200._host.Runner";
  RunnerType.tp_basicsize = sizeof(Runner);
  RunnerType.tp_flags = Py_TPFLAGS_DEFAULT;
  RunnerType.tp_new = runner_new;
  RunnerType.tp_dealloc = (destructor)runner_dealloc;
  RunnerType.tp_methods = runner_methods;
  if (PyType_Ready(&LauncherType) < 0 || PyType_Ready(&RunnerType) < 0) return nullptr;
  PyObject *m = PyModule_Create(&host_module);
  if (!m) return nullptr;
  if (PyModule_AddObjectRef(m, "Launcher", (PyObject *)&LauncherType) < 0 || PyModule_AddObjectRef(m, "Runner", (PyObject *)&RunnerType) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
