// The calls a Python program makes once per layer, as CPython functions over the C ABI (include/gie_b200.h): arguments
// are taken from the vector-call array and handed on as they are, without building foreign-function objects.  A call
// costs the host ~0.3 us on top of the C function where ctypes costs 1.9 us (16 x 4096 RMSNorm, stream full of such
// calls: 4.8 us a call through ctypes of which the launch itself is 2.9), and small layers are bound by the host.
// Everything else of the ABI (plan creation, queries, status words) stays on ctypes in __init__.py.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>
#include <string.h>

#include "gie_b200.h"

namespace {

// Pointers are ints or None and counts are ints, nothing else: for any other argument the callers in __init__.py go through
// ctypes, whose conversions (objects with `_as_parameter_`, c_void_p, numpy integers for counts, ..) and refusals then apply.
bool to_pointer(PyObject* o, void** out) {
  if (PyLong_Check(o)) {
    *out = reinterpret_cast<void*>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(o)));
    return !PyErr_Occurred();
  }
  if (o == Py_None) {
    *out = nullptr;
    return true;
  }
  PyErr_Format(PyExc_TypeError, "expected a device pointer (int or None), got %.100s", Py_TYPE(o)->tp_name);
  return false;
}

bool to_int(PyObject* o, long long* out) {
  if (!PyLong_Check(o)) {
    PyErr_Format(PyExc_TypeError, "expected an int, got %.100s", Py_TYPE(o)->tp_name);
    return false;
  }
  *out = static_cast<long long>(PyLong_AsUnsignedLongLongMask(o));
  return !PyErr_Occurred();
}

// Reads `n` arguments by a format of one letter each: p pointer, i integer, f float.
struct Arg {
  void* p;
  long long i;
  double f;
};
bool parse(PyObject* const* args, Py_ssize_t given, const char* format, Arg* out) {
  Py_ssize_t n = 0;
  while (format[n]) ++n;
  if (given != n) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", n, given);
    return false;
  }
  for (Py_ssize_t k = 0; k < n; ++k) {
    if (format[k] == 'p') {
      if (!to_pointer(args[k], &out[k].p)) return false;
    } else if (format[k] == 'i') {
      if (!to_int(args[k], &out[k].i)) return false;
    } else {
      out[k].f = PyFloat_AsDouble(args[k]);
      if (out[k].f == -1.0 && PyErr_Occurred()) return false;
    }
  }
  return true;
}

// The global lock is released around the call, as ctypes does: a launch may wait for room in the stream's queue.
template <typename F>
PyObject* status_of(F&& call) {
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = call();
  Py_END_ALLOW_THREADS
  if (status == 0) return Py_NewRef(Py_None);
  return PyLong_FromLong(status);
}

int i32(const Arg& a) { return static_cast<int>(a.i); }

int call_conv(const Arg* a) {
  return gieb_conv_launch(static_cast<const gieb_conv_plan*>(a[0].p), a[1].p, a[2].p, a[3].p, a[4].p, a[5].p, static_cast<size_t>(a[6].i), a[7].p);
}
int call_conv_fused(const Arg* a) {
  return gieb_conv_launch_fused(static_cast<const gieb_conv_plan*>(a[0].p), a[1].p, a[2].p, a[3].p, a[4].p, a[5].p, a[6].p,
                                static_cast<size_t>(a[7].i), a[8].p);
}
int call_rmsnorm(const Arg* a) {
  const gieb_rmsnorm_desc d = {i32(a[0]), i32(a[1]), static_cast<float>(a[2].f), i32(a[3]), static_cast<uint32_t>(a[4].i)};
  return gieb_rmsnorm_launch(&d, a[5].p, a[6].p, a[7].p, a[8].p, a[9].p, a[10].p);
}
int call_bias_act(const Arg* a) { return gieb_bias_act_launch(i32(a[0]), i32(a[1]), i32(a[2]), i32(a[3]), a[4].p, i32(a[5]), a[6].p, a[7].p); }
int call_maxpool(const Arg* a) {
  return gieb_maxpool2d_launch(i32(a[0]), i32(a[1]), i32(a[2]), i32(a[3]), i32(a[4]), i32(a[5]), i32(a[6]), i32(a[7]), a[8].p, a[9].p, a[10].p);
}
int call_maxpool_nhwc(const Arg* a) {
  return gieb_maxpool2d_nhwc_launch(i32(a[0]), i32(a[1]), i32(a[2]), i32(a[3]), i32(a[4]), i32(a[5]), i32(a[6]), i32(a[7]), a[8].p, a[9].p, a[10].p);
}
int call_add_relu(const Arg* a) { return gieb_add_relu_launch(i32(a[0]), i32(a[1]), a[2].p, a[3].p, a[4].p, a[5].i, a[6].p); }

// One table for single calls and recorded sequences; the last argument of every entry is the stream.
struct Entry {
  const char* name;
  const char* format;
  int (*call)(const Arg*);
};
constexpr int kMaxArgs = 12;
const Entry kEntries[] = {
    {"conv_launch", "ppppppip", call_conv},
    {"conv_launch_fused", "pppppppip", call_conv_fused},
    {"rmsnorm_launch", "iifiipppppp", call_rmsnorm},
    {"bias_act_launch", "iiiipipp", call_bias_act},
    {"maxpool2d_launch", "iiiiiiiippp", call_maxpool},
    {"maxpool2d_nhwc_launch", "iiiiiiiippp", call_maxpool_nhwc},
    {"add_relu_launch", "iipppip", call_add_relu},
};
constexpr int kEntryCount = int(sizeof(kEntries) / sizeof(kEntries[0]));

template <int E>
PyObject* single(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Arg a[kMaxArgs];
  if (!parse(args, n, kEntries[E].format, a)) return nullptr;
  return status_of([&] { return kEntries[E].call(a); });
}

// A recorded sequence of calls with fixed arguments (a network whose buffers stay where they are): record(list of
// (entry name, argument, ..)) without the streams, run_sequence(recording, stream) issues them in order and stops at the
// first that fails.
struct Step {
  int entry, stream_at;
  Arg a[kMaxArgs];
};
struct Sequence {
  Py_ssize_t n;
  Step steps[1];
};
constexpr const char* kSequence = "cuda_inference_b200.sequence";

void free_sequence(PyObject* capsule) { PyMem_Free(PyCapsule_GetPointer(capsule, kSequence)); }

PyObject* record(PyObject*, PyObject* list) {
  PyObject* fast = PySequence_Fast(list, "record() takes a list of calls");
  if (fast == nullptr) return nullptr;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
  Sequence* s = static_cast<Sequence*>(PyMem_Calloc(1, sizeof(Sequence) + size_t(n) * sizeof(Step)));
  if (s == nullptr) {
    Py_DECREF(fast);
    return PyErr_NoMemory();
  }
  s->n = n;
  bool ok = true;
  for (Py_ssize_t k = 0; ok && k < n; ++k) {
    PyObject* call = PySequence_Tuple(PySequence_Fast_GET_ITEM(fast, k));
    ok = call != nullptr && PyTuple_GET_SIZE(call) >= 1;
    const char* name = ok ? PyUnicode_AsUTF8(PyTuple_GET_ITEM(call, 0)) : nullptr;
    int e = 0;
    while (name != nullptr && e < kEntryCount && strcmp(name, kEntries[e].name) != 0) ++e;
    if (ok && (name == nullptr || e == kEntryCount)) {
      if (!PyErr_Occurred()) PyErr_Format(PyExc_ValueError, "unknown call %.100s", name);
      ok = false;
    }
    if (ok) {
      char format[kMaxArgs + 1];
      const int len = int(strlen(kEntries[e].format));
      memcpy(format, kEntries[e].format, size_t(len));
      format[len - 1] = 0;  // without the stream
      s->steps[k].entry = e;
      s->steps[k].stream_at = len - 1;
      ok = parse(&PyTuple_GET_ITEM(call, 1), PyTuple_GET_SIZE(call) - 1, format, s->steps[k].a);
    }
    Py_XDECREF(call);
  }
  Py_DECREF(fast);
  if (!ok) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "a call is a tuple (name, argument, ...)");
    PyMem_Free(s);
    return nullptr;
  }
  return PyCapsule_New(s, kSequence, free_sequence);
}

PyObject* run_sequence(PyObject*, PyObject* const* args, Py_ssize_t n) {
  void* stream;
  if (n != 2) {
    PyErr_Format(PyExc_TypeError, "expected 2 arguments, got %zd", n);
    return nullptr;
  }
  const Sequence* s = static_cast<const Sequence*>(PyCapsule_GetPointer(args[0], kSequence));
  if (s == nullptr || !to_pointer(args[1], &stream)) return nullptr;
  return status_of([&] {
    for (Py_ssize_t k = 0; k < s->n; ++k) {
      Step step = s->steps[k];  // (a copy: threads may run one recording on several streams)
      step.a[step.stream_at].p = stream;
      const int status = kEntries[step.entry].call(step.a);
      if (status != 0) return status;
    }
    return 0;
  });
}

template <int E>
PyMethodDef method() {
  return {kEntries[E].name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(single<E>)), METH_FASTCALL, nullptr};
}
PyMethodDef kMethods[] = {
    method<0>(), method<1>(), method<2>(), method<3>(), method<4>(), method<5>(), method<6>(),
    {"record", record, METH_O, nullptr},
    {"run_sequence", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(run_sequence)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
static_assert(kEntryCount == 7, "every entry has its method above");

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) { return PyModule_Create(&kModule); }
