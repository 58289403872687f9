// The host side of an eager call on a prepared launch, as a Python extension.
//
// One token's Linear is 3 to 6 us on the device, so what an eager caller waits for is the host: in Python the checks of a
// call, the look-ups of its scratch and stream and the conversions of seven ctypes arguments took 5 us around the launch.
// Here they take a few hundred nanoseconds.  Three types of work, all on objects that belong to the
// Python side (its dictionaries stay the only record of scratches and of the launch ahead):
//   Call    runs a prepared launch on (x, out); `fits` first checks that the operands are what it was prepared for
//   Bound   the prepared decode of a module: checks x, runs a Call into the module's output, returns its view
//   holds   whether a layout's tensors are those, unchanged, that a record was made for
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstring>

namespace {

using RunFn = int (*)(const void* launch, const void* x, void* out, void* scratch, size_t scratch_bytes, unsigned flags, void* stream);

struct Call {
  PyObject_HEAD
  RunFn run;
  const void* handle;
  int64_t rows, in_features, out_features;
  int index;
  c10::ScalarType dtype;
  unsigned flags, follow_flags;  // of every launch; of one that reads the activations of the launch ahead
  bool follows;                  // a launch that may follow another on the same activations, or be followed
  size_t need;
  PyObject* dtype_object;
  PyObject* families;    // scratch families: the one, or the three that rotate
  PyObject* scratch;     // dict (index, stream, family) -> tensor
  PyObject* ahead;       // dict (index, stream) -> (Row, launches in it)
  PyObject* scratch_for; // (device index, bytes, family) -> tensor
  PyObject* capturing;   // () -> bool
  PyObject* failed;      // raises the error of a refused launch
};

PyObject* key_of(PyObject* index, PyObject* stream, PyObject* family) {
  return family ? PyTuple_Pack(3, index, stream, family) : PyTuple_Pack(2, index, stream);
}

// Borrowed reference, or null without an error when absent.
PyObject* scratch_at(Call* self, PyObject* index, PyObject* stream, PyObject* family) {
  PyObject* key = key_of(index, stream, family);
  if (!key) return nullptr;
  PyObject* found = PyDict_GetItemWithError(self->scratch, key);
  Py_DECREF(key);
  return found;
}

constexpr int kMostInARow = 3;

// Launches one after the other on the same activations: which, and where each of them writes; all captured or all eager,
// since one kind is not ahead of the other.  Kept as bytes: a call on a
// prepared launch compares and makes one, and as Python objects that took 0.3 us.
struct Row {
  uint64_t x = 0, k = 0, dtype = 0, captured = 0, launches = 0, outputs[kMostInARow][2] = {};

  // Which place a launch takes in the row; 0: it does not belong to it.  Launches of a row overlap and may not write to one place:
  // the older one could be the last to do so.
  long place(uint64_t x_, uint64_t k_, c10::ScalarType dtype_, bool captured_, uint64_t begin, uint64_t end) const {
    if (launches >= kMostInARow || x != x_ || k != k_ || dtype != static_cast<uint64_t>(dtype_) || captured != captured_) return 0;
    for (uint64_t i = 0; i < launches; ++i)
      if (begin < outputs[i][1] && outputs[i][0] < end) return 0;
    return static_cast<long>(launches);
  }
  // ... and the row with it; place 0 begins one.
  Row with(long place, uint64_t x_, uint64_t k_, c10::ScalarType dtype_, bool captured_, uint64_t begin, uint64_t end) const {
    Row row = place ? *this : Row();
    row.x = x_, row.k = k_, row.dtype = static_cast<uint64_t>(dtype_), row.captured = captured_;
    row.outputs[row.launches][0] = begin, row.outputs[row.launches][1] = end, ++row.launches;
    return row;
  }
  // of an entry of `ahead` (null, or None: an empty one)
  static Row of(PyObject* entry) {
    Row row;
    if (entry && entry != Py_None) memcpy(&row, PyBytes_AS_STRING(PyTuple_GET_ITEM(entry, 0)), sizeof row);
    return row;
  }
  PyObject* entry() const {
    PyObject *bytes = PyBytes_FromStringAndSize(reinterpret_cast<const char*>(this), sizeof *this), *count = PyLong_FromLong(static_cast<long>(launches));
    PyObject* made = bytes && count ? PyTuple_Pack(2, bytes, count) : nullptr;
    Py_XDECREF(count), Py_XDECREF(bytes);
    return made;
  }
};

// Launches under way, and how many there have been, under the GIL (a launch gives it up): one may follow the launch ahead, and be
// remembered as that, only if no other thread's came between the look at `ahead` and the note in it.
long under_way = 0;
unsigned long long turns = 0;

bool run_call(Call* self, const at::Tensor& x, const at::Tensor& out) {
  const c10::cuda::OptionalCUDAGuard guard(c10::cuda::current_device() == self->index ? c10::optional<c10::DeviceIndex>() : c10::optional<c10::DeviceIndex>(self->index));
  void* const stream = c10::cuda::getCurrentCUDAStream(self->index).stream();
  const void* const x_ptr = x.const_data_ptr();
  void* const out_ptr = out.data_ptr();
  PyObject* index = PyLong_FromLong(self->index);
  PyObject* stream_key = PyLong_FromUnsignedLongLong(reinterpret_cast<uintptr_t>(stream));
  PyObject *pair = nullptr, *buffer = nullptr;
  const uint64_t x_at = reinterpret_cast<uintptr_t>(x_ptr), out_begin = reinterpret_cast<uintptr_t>(out_ptr), out_end = out_begin + 2 * self->rows * self->out_features;
  Row row;
  bool captured = false;
  long slot = 0;
  bool ok = index && stream_key;
  if (ok && self->follows) {
    captured = c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
    pair = key_of(index, stream_key, nullptr);
    ok = pair != nullptr;
    if (ok && self->follow_flags && under_way == 0) {
      row = Row::of(PyDict_GetItemWithError(self->ahead, pair));
      ok = !PyErr_Occurred();
      slot = row.place(x_at, self->in_features, self->dtype, captured, out_begin, out_end);
    }
  }
  if (ok) {
    buffer = scratch_at(self, index, stream_key, PyTuple_GET_ITEM(self->families, slot));
    ok = !PyErr_Occurred();
    if (ok && !buffer && slot > 0) {  // nothing is allocated in a capture: wait instead
      PyObject* answer = PyObject_CallNoArgs(self->capturing);
      ok = answer != nullptr;
      if (answer == Py_True) {
        slot = 0;
        buffer = scratch_at(self, index, stream_key, PyTuple_GET_ITEM(self->families, 0));
        ok = !PyErr_Occurred();
      }
      Py_XDECREF(answer);
    }
    if (ok && buffer && THPVariable_Unpack(buffer).nbytes() < self->need) buffer = nullptr;
    if (ok) {
      if (buffer)
        Py_INCREF(buffer);
      else
        buffer = PyObject_CallFunction(self->scratch_for, "inO", self->index, (Py_ssize_t)self->need, PyTuple_GET_ITEM(self->families, slot));
      ok = buffer != nullptr;
    } else {
      buffer = nullptr;
    }
  }
  if (ok) {
    const at::Tensor& memory = THPVariable_Unpack(buffer);
    void* const address = memory.data_ptr();
    const size_t bytes = memory.nbytes();
    const unsigned flags = self->flags | (slot ? self->follow_flags : 0u);
    int code = 0;
    const unsigned long long turn = ++turns;
    ++under_way;
    Py_BEGIN_ALLOW_THREADS;
    code = self->run(self->handle, x_ptr, out_ptr, address, bytes, flags, stream);
    Py_END_ALLOW_THREADS;
    const bool alone = --under_way == 0 && turn == turns;
    PyDict_Clear(self->ahead);
    if (code != 0) {
      Py_XDECREF(PyObject_CallFunction(self->failed, "i", code));
      ok = false;
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "native call failed");
    } else if (self->follows && self->follow_flags && alone) {
      PyObject* entry = row.with(slot, x_at, self->in_features, self->dtype, captured, out_begin, out_end).entry();
      ok = entry && PyDict_SetItem(self->ahead, pair, entry) == 0;
      Py_XDECREF(entry);
    }
  }
  Py_XDECREF(buffer), Py_XDECREF(pair), Py_XDECREF(stream_key), Py_XDECREF(index);
  return ok;
}

bool matrix_is(const at::Tensor& t, int64_t rows, int64_t columns, c10::ScalarType dtype, int index) {
  return t.dim() == 2 && t.size(0) == rows && t.size(1) == columns && t.scalar_type() == dtype && t.is_cuda() && t.get_device() == index && t.is_contiguous();
}

bool two_tensors(PyObject* const* args, Py_ssize_t count) {
  if (count == 2 && THPVariable_Check(args[0]) && THPVariable_Check(args[1])) return true;
  PyErr_SetString(PyExc_TypeError, "expected the tensors x and out");
  return false;
}

template <class F>
PyObject* guarded(F body) {
  try {
    return body();
  } catch (const std::exception& error) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, error.what());
    return nullptr;
  }
}

// run(x, out): the caller has checked the operands
PyObject* call_run(PyObject* object, PyObject* const* args, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    if (!two_tensors(args, count) || !run_call(reinterpret_cast<Call*>(object), THPVariable_Unpack(args[0]), THPVariable_Unpack(args[1]))) return nullptr;
    Py_RETURN_NONE;
  });
}

// fits(x, out): False, and nothing done, unless x and out are what the launch was prepared for
PyObject* call_fits(PyObject* object, PyObject* const* args, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    auto* self = reinterpret_cast<Call*>(object);
    if (count != 2 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) Py_RETURN_FALSE;
    const at::Tensor &x = THPVariable_Unpack(args[0]), &out = THPVariable_Unpack(args[1]);
    if (!matrix_is(x, self->rows, self->in_features, self->dtype, self->index) || !matrix_is(out, self->rows, self->out_features, self->dtype, self->index)) Py_RETURN_FALSE;
    if (!run_call(self, x, out)) return nullptr;
    Py_RETURN_TRUE;
  });
}

int call_init(PyObject* object, PyObject* args, PyObject*) {
  auto* self = reinterpret_cast<Call*>(object);
  unsigned long long run = 0, handle = 0;
  Py_ssize_t need = 0;
  int follows = 0;
  long long rows = 0, in_features = 0, out_features = 0;
  if (self->families) return PyErr_SetString(PyExc_RuntimeError, "already made"), -1;
  if (!PyArg_ParseTuple(args, "KKLLLiOIIpnO!O!O!OOO", &run, &handle, &rows, &in_features, &out_features, &self->index, &self->dtype_object, &self->flags,
                        &self->follow_flags, &follows, &need, &PyTuple_Type, &self->families, &PyDict_Type, &self->scratch, &PyDict_Type, &self->ahead,
                        &self->scratch_for, &self->capturing, &self->failed)) {
    self->dtype_object = self->families = self->scratch = self->ahead = self->scratch_for = self->capturing = self->failed = nullptr;
    return -1;
  }
  for (PyObject* held : {self->dtype_object, self->families, self->scratch, self->ahead, self->scratch_for, self->capturing, self->failed}) Py_INCREF(held);
  self->run = reinterpret_cast<RunFn>(static_cast<uintptr_t>(run)), self->handle = reinterpret_cast<const void*>(static_cast<uintptr_t>(handle));
  self->rows = rows, self->in_features = in_features, self->out_features = out_features;
  self->need = static_cast<size_t>(need), self->follows = follows != 0;
  self->dtype = reinterpret_cast<THPDtype*>(self->dtype_object)->scalar_type;
  return self->follows && PyTuple_GET_SIZE(self->families) != kMostInARow ? (PyErr_SetString(PyExc_ValueError, "a launch that follows takes three scratches"), -1) : 0;
}

void call_dealloc(PyObject* object) {
  auto* self = reinterpret_cast<Call*>(object);
  for (PyObject* held : {self->dtype_object, self->families, self->scratch, self->ahead, self->scratch_for, self->capturing, self->failed}) Py_XDECREF(held);
  Py_TYPE(object)->tp_free(object);
}

PyMethodDef call_methods[] = {{"run", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_run)), METH_FASTCALL, nullptr},
                              {"fits", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_fits)), METH_FASTCALL, nullptr},
                              {nullptr, nullptr, 0, nullptr}};
PyTypeObject call_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

struct Bound {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  Call* call;
  PyObject* launch;   // keeps the prepared launch
  PyObject* output;   // [1, O]
  PyObject* shaped;   // its view [1, 1, O]
  PyObject* module;   // weak reference: a dropped module gives its weights back at once
  PyObject* buffers;  // the module's, for the bias
};

PyObject *name_bias, *name_audit, *name_counts, *name_route, *name_last, *name_add;

bool count_route(PyObject* module) {
  PyObject* counts = PyObject_GetAttr(module, name_counts);
  PyObject* before = counts ? PyObject_GetItem(counts, name_route) : nullptr;
  PyObject* one = PyLong_FromLong(1);
  PyObject* after = before && one ? PyNumber_Add(before, one) : nullptr;
  const bool ok = after && PyObject_SetItem(counts, name_route, after) == 0 && PyObject_SetAttr(module, name_last, name_route) == 0;
  Py_XDECREF(after), Py_XDECREF(one), Py_XDECREF(before), Py_XDECREF(counts);
  return ok;
}

PyObject* bound_call(PyObject* object, PyObject* const* args, size_t flags, PyObject* names) {
  return guarded([&]() -> PyObject* {
    auto* self = reinterpret_cast<Bound*>(object);
    if (PyVectorcall_NARGS(flags) != 1 || (names && PyTuple_GET_SIZE(names)) || !THPVariable_Check(args[0])) return PyErr_SetString(PyExc_TypeError, "expected the tensor x"), nullptr;
    if (c10::GradMode::is_enabled()) return PyErr_SetString(PyExc_RuntimeError, "prepared decode is inference only"), nullptr;
    const at::Tensor& x = THPVariable_Unpack(args[0]);
    Call* const call = self->call;
    if (x.dim() != 3 || x.size(0) != 1 || x.size(1) != 1 || x.size(2) != call->in_features || x.scalar_type() != call->dtype || !x.is_cuda() ||
        x.get_device() != call->index || !x.is_contiguous())
      return PyErr_SetString(PyExc_ValueError, "prepared decode input shape/dtype/device/stride mismatch"), nullptr;
    PyObject* module = PyWeakref_GetObject(self->module);  // borrowed
    if (module && module != Py_None) {
      Py_INCREF(module);
      PyObject* audit = PyObject_GetAttr(module, name_audit);
      const int counted = audit ? PyObject_IsTrue(audit) : -1;
      Py_XDECREF(audit);
      const bool ok = counted == 0 || (counted == 1 && count_route(module));
      Py_DECREF(module);
      if (!ok) return nullptr;
    }
    if (!run_call(call, x, THPVariable_Unpack(self->output))) return nullptr;
    PyObject* bias = PyDict_GetItemWithError(self->buffers, name_bias);
    if (bias && bias != Py_None) {
      PyObject* done = PyObject_CallMethodOneArg(self->output, name_add, bias);
      if (!done) return nullptr;
      Py_DECREF(done);
    } else if (!bias && PyErr_Occurred()) {
      return nullptr;
    }
    Py_INCREF(self->shaped);
    return self->shaped;
  });
}

int bound_init(PyObject* object, PyObject* args, PyObject*) {
  auto* self = reinterpret_cast<Bound*>(object);
  PyObject *call, *launch, *output, *shaped, *module, *buffers;
  if (self->call) return PyErr_SetString(PyExc_RuntimeError, "already made"), -1;
  if (!PyArg_ParseTuple(args, "O!OOOOO!", &call_type, &call, &launch, &output, &shaped, &module, &PyDict_Type, &buffers)) return -1;
  if (!THPVariable_Check(output) || !PyWeakref_Check(module)) return PyErr_SetString(PyExc_TypeError, "expected an output tensor and a weak reference"), -1;
  for (PyObject* held : {call, launch, output, shaped, module, buffers}) Py_INCREF(held);
  self->call = reinterpret_cast<Call*>(call), self->launch = launch, self->output = output, self->shaped = shaped, self->module = module, self->buffers = buffers;
  self->vectorcall = bound_call;
  return 0;
}

PyObject* bound_new(PyTypeObject* type, PyObject*, PyObject*) {
  auto* self = reinterpret_cast<Bound*>(type->tp_alloc(type, 0));
  if (self) self->vectorcall = [](PyObject*, PyObject* const*, size_t, PyObject*) -> PyObject* { return PyErr_SetString(PyExc_RuntimeError, "not bound"), nullptr; };
  return reinterpret_cast<PyObject*>(self);
}

void bound_dealloc(PyObject* object) {
  auto* self = reinterpret_cast<Bound*>(object);
  Py_XDECREF(reinterpret_cast<PyObject*>(self->call)), Py_XDECREF(self->launch), Py_XDECREF(self->output), Py_XDECREF(self->shaped);
  Py_XDECREF(self->module), Py_XDECREF(self->buffers);
  Py_TYPE(object)->tp_free(object);
}

PyObject* bound_copy(PyObject* object, PyObject*) { return Py_NewRef(object); }  // as functions are copied

PyMethodDef bound_methods[] = {{"__copy__", bound_copy, METH_NOARGS, nullptr}, {"__deepcopy__", bound_copy, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyTypeObject bound_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// What a check saw of a tensor: compared byte by byte, it costs a call next to nothing.
struct Stamp {
  int64_t address = 0, sizes[4] = {}, dim = 0, dtype = 0, tracked = 0, version = 0;  // version -1: an inference tensor, which has none

  Stamp(const at::Tensor& t, bool with_version) {
    address = static_cast<int64_t>(reinterpret_cast<uintptr_t>(t.const_data_ptr()));
    dim = t.is_contiguous() && t.dim() <= 4 ? t.dim() : -1;
    for (int64_t i = 0; i < dim; ++i) sizes[i] = t.size(i);
    dtype = static_cast<int64_t>(t.scalar_type());
    tracked = with_version;
    if (with_version) version = t.is_inference() ? -1 : static_cast<int64_t>(t._version());
  }
};

// stamp(tensor, whether its version counts) -> bytes
PyObject* stamp(PyObject*, PyObject* const* args, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    if (count != 2 || !THPVariable_Check(args[0])) return PyErr_SetString(PyExc_TypeError, "expected a tensor and a truth value"), nullptr;
    const Stamp seen(THPVariable_Unpack(args[0]), args[1] == Py_True);
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(&seen), sizeof seen);
  });
}

// holds(layout, seen): seen = ((name, weak reference, stamp), ...); whether the layout is exactly these tensors, as they were
PyObject* holds(PyObject*, PyObject* const* args, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    if (count != 2 || !PyTuple_Check(args[1])) return PyErr_SetString(PyExc_TypeError, "expected a layout and a tuple"), nullptr;
    if (!PyDict_Check(args[0]) || PyDict_GET_SIZE(args[0]) != PyTuple_GET_SIZE(args[1])) Py_RETURN_FALSE;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[1]); ++i) {
      PyObject* entry = PyTuple_GET_ITEM(args[1], i);
      PyObject* value = PyDict_GetItemWithError(args[0], PyTuple_GET_ITEM(entry, 0));
      if (!value && PyErr_Occurred()) return nullptr;
      if (!value || PyWeakref_GetObject(PyTuple_GET_ITEM(entry, 1)) != value || !THPVariable_Check(value)) Py_RETURN_FALSE;
      const char* const then = PyBytes_AS_STRING(PyTuple_GET_ITEM(entry, 2));
      const Stamp now(THPVariable_Unpack(value), reinterpret_cast<const Stamp*>(then)->tracked != 0);
      if (memcmp(&now, then, sizeof now)) Py_RETURN_FALSE;
    }
    Py_RETURN_TRUE;
  });
}

// begin() -> (whether no launch is under way, turn); end(turn) -> whether none came in between: the same for a launch by ctypes
PyObject* begin(PyObject*, PyObject*) {
  const bool alone = under_way++ == 0;
  return Py_BuildValue("(NK)", PyBool_FromLong(alone), ++turns);
}
PyObject* end(PyObject*, PyObject* turn) {
  --under_way;
  return PyBool_FromLong(under_way == 0 && PyLong_AsUnsignedLongLong(turn) == turns);
}

// place(entry, x address, K, dtype, captured, output's begin, end) and row(entry, place, the same): for a launch by ctypes
PyObject* place(PyObject*, PyObject* args) {
  PyObject *entry, *dtype;
  unsigned long long x, k, begin, end;
  int captured;
  if (!PyArg_ParseTuple(args, "OKKOpKK", &entry, &x, &k, &dtype, &captured, &begin, &end)) return nullptr;
  return PyLong_FromLong(Row::of(entry).place(x, k, reinterpret_cast<THPDtype*>(dtype)->scalar_type, captured != 0, begin, end));
}
PyObject* row_with(PyObject*, PyObject* args) {
  PyObject *entry, *dtype;
  long at;
  unsigned long long x, k, begin, end;
  int captured;
  if (!PyArg_ParseTuple(args, "OlKKOpKK", &entry, &at, &x, &k, &dtype, &captured, &begin, &end)) return nullptr;
  return Row::of(entry).with(at, x, k, reinterpret_cast<THPDtype*>(dtype)->scalar_type, captured != 0, begin, end).entry();
}

PyMethodDef module_methods[] = {{"place", place, METH_VARARGS, nullptr}, {"row", row_with, METH_VARARGS, nullptr}, {"begin", begin, METH_NOARGS, nullptr}, {"end", end, METH_O, nullptr}, {"stamp", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(stamp)), METH_FASTCALL, nullptr},
                                {"holds", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(holds)), METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_fb_calls", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fb_calls(void) {
  call_type.tp_name = "_fb_calls.Call", call_type.tp_basicsize = sizeof(Call), call_type.tp_flags = Py_TPFLAGS_DEFAULT;
  call_type.tp_new = PyType_GenericNew, call_type.tp_init = call_init, call_type.tp_dealloc = call_dealloc, call_type.tp_methods = call_methods;
  bound_type.tp_name = "_fb_calls.Bound", bound_type.tp_basicsize = sizeof(Bound), bound_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  bound_type.tp_vectorcall_offset = offsetof(Bound, vectorcall), bound_type.tp_call = PyVectorcall_Call;
  bound_type.tp_new = bound_new, bound_type.tp_init = bound_init, bound_type.tp_dealloc = bound_dealloc, bound_type.tp_methods = bound_methods;
  if (PyType_Ready(&call_type) < 0 || PyType_Ready(&bound_type) < 0) return nullptr;
  name_bias = PyUnicode_InternFromString("bias"), name_audit = PyUnicode_InternFromString("_decode_audit");
  name_counts = PyUnicode_InternFromString("route_counts"), name_route = PyUnicode_InternFromString("packed_m1");
  name_last = PyUnicode_InternFromString("last_route"), name_add = PyUnicode_InternFromString("add_");
  PyObject* module = PyModule_Create(&module_def);
  if (!module) return nullptr;
  if (PyModule_AddStringConstant(module, "torch_version", FB_TORCH_VERSION) < 0 || PyModule_AddObjectRef(module, "Call", reinterpret_cast<PyObject*>(&call_type)) < 0 || PyModule_AddObjectRef(module, "Bound", reinterpret_cast<PyObject*>(&bound_type)) < 0) {
    Py_DECREF(module);
    return nullptr;
  }
  return module;
}
