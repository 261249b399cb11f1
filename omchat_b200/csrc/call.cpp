// Calls of the C entries from Python without ctypes: tensors, integers and floats go straight into the registers and stack slots that the x86-64 System V
// convention gives them, and the checks that every wrapper makes of its tensors (on the GPU, on the current device) are one call.
//
// A wrapper of 25 arguments spent some 10 us in ctypes, in one data_ptr() call per tensor and in the device checks, more than the launch itself.
#include <Python.h>
#include <c10/core/impl/VirtualGuardImpl.h>
#include <stdint.h>
#include <string.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>

#if !defined(__x86_64__) || !defined(__linux__)
#error "the register assignment below is that of x86-64 System V"
#endif

namespace {

constexpr int kRegs = 6, kFloats = 8, kStack = 34, kMaxArgs = kRegs + kStack;

// Integers and pointers fill the six registers and then 8-byte stack slots in their order, floats the eight vector registers in theirs, however the two are mixed
// in the prototype; slots behind the last argument are not read.
typedef int (*Fn)(int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, float, float, float, float, float, float, float, float, int64_t, int64_t, int64_t, int64_t, int64_t,
                  int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                  int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t);

struct Entry {
  PyObject_HEAD
  vectorcallfunc call;
  Fn fn;
  PyObject* other;   // the ctypes function: arguments of any other kind go to it
  int n;
  char sig[kMaxArgs + 1];   // P pointer, I int, L long long, F float
};

PyObject* error_type = nullptr;

PyObject* entry_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* names) {
  Entry* e = reinterpret_cast<Entry*>(self);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != e->n || (names != nullptr && PyTuple_GET_SIZE(names) > 0)) return PyObject_Vectorcall(e->other, args, nargsf, names);
  int64_t v[kMaxArgs];
  float f[kFloats] = {};
  int ni = 0, nf = 0;
  try {
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* a = args[i];
      if (e->sig[i] == 'F') {
        const double x = PyFloat_Check(a) ? PyFloat_AS_DOUBLE(a) : (PyLong_Check(a) ? PyLong_AsDouble(a) : 0.0);
        if (!PyFloat_Check(a) && (!PyLong_Check(a) || PyErr_Occurred())) goto other;
        f[nf++] = (float)x;
      } else if (e->sig[i] == 'P' && a == Py_None) {
        v[ni++] = 0;
      } else if (PyLong_Check(a)) {
        v[ni++] = e->sig[i] == 'P' ? (int64_t)PyLong_AsUnsignedLongLong(a) : (int64_t)PyLong_AsLongLong(a);
        if (v[ni - 1] == -1 && PyErr_Occurred()) goto other;
      } else if (e->sig[i] == 'P' && THPVariable_Check(a)) {
        v[ni++] = (int64_t)reinterpret_cast<uintptr_t>(THPVariable_Unpack(a).data_ptr());
      } else {
        goto other;
      }
    }
  } catch (const std::exception& x) {
    PyErr_SetString(PyExc_RuntimeError, x.what());
    return nullptr;
  }
  for (; ni < kMaxArgs; ++ni) v[ni] = 0;
  {
    int rc;
    Py_BEGIN_ALLOW_THREADS;
    rc = e->fn(v[0], v[1], v[2], v[3], v[4], v[5], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], v[6], v[7], v[8], v[9], v[10], v[11], v[12], v[13], v[14], v[15], v[16],
               v[17], v[18], v[19], v[20], v[21], v[22], v[23], v[24], v[25], v[26], v[27], v[28], v[29], v[30], v[31], v[32], v[33], v[34], v[35], v[36], v[37], v[38], v[39]);
    Py_END_ALLOW_THREADS;
    return PyLong_FromLong(rc);
  }
other:
  PyErr_Clear();
  return PyObject_Vectorcall(e->other, args, nargsf, names);
}

void entry_dealloc(PyObject* self) {
  Py_XDECREF(reinterpret_cast<Entry*>(self)->other);
  PyObject_Free(self);
}

PyTypeObject EntryType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// entry(address, signature, ctypes function) -> a callable, or None where the signature does not fit
PyObject* make_entry(PyObject*, PyObject* args) {
  unsigned long long address;
  const char* sig;
  PyObject* other;
  if (!PyArg_ParseTuple(args, "KsO", &address, &sig, &other)) return nullptr;
  const size_t n = strlen(sig);
  int floats = 0;
  for (size_t i = 0; i < n; ++i) floats += sig[i] == 'F';
  if (floats > kFloats || n - floats > (size_t)kMaxArgs || n > (size_t)kMaxArgs || strspn(sig, "PILF") != n) Py_RETURN_NONE;
  Entry* e = PyObject_New(Entry, &EntryType);
  if (e == nullptr) return nullptr;
  e->call = entry_call;
  e->fn = reinterpret_cast<Fn>(static_cast<uintptr_t>(address));
  Py_INCREF(other);
  e->other = other;
  e->n = (int)n;
  memcpy(e->sig, sig, n + 1);
  return reinterpret_cast<PyObject*>(e);
}

// need_cuda(*tensors): an error for one that is not on the GPU, or not on the current one; None counts as no tensor
PyObject* need_cuda(PyObject*, PyObject* const* args, Py_ssize_t n) {
  int cur = -1;
  try {
    for (Py_ssize_t i = 0; i < n; ++i) {
      if (args[i] == Py_None) continue;
      if (!THPVariable_Check(args[i])) {
        PyErr_SetString(PyExc_TypeError, "a tensor or None is wanted");
        return nullptr;
      }
      const c10::Device d = THPVariable_Unpack(args[i]).device();
      if (d.type() != c10::DeviceType::CUDA) {
        PyErr_SetString(error_type != nullptr ? error_type : PyExc_RuntimeError, "omchat_b200 kernels need CUDA tensors (no CPU fallback)");
        return nullptr;
      }
      if (cur < 0) cur = c10::impl::VirtualGuardImpl(c10::DeviceType::CUDA).getDevice().index();
      if (d.index() != cur) {
        PyErr_Format(error_type != nullptr ? error_type : PyExc_RuntimeError,
                     "tensor on cuda:%d but the current device is cuda:%d: run the call under `with torch.cuda.device(%d):` (the model classes do this themselves)",
                     (int)d.index(), cur, (int)d.index());
        return nullptr;
      }
    }
  } catch (const std::exception& x) {
    PyErr_SetString(PyExc_RuntimeError, x.what());
    return nullptr;
  }
  Py_RETURN_NONE;
}

PyObject* set_error_type(PyObject*, PyObject* type) {
  Py_INCREF(type);
  Py_XSETREF(error_type, type);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"entry", make_entry, METH_VARARGS, nullptr},
                         {"need_cuda", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(need_cuda)), METH_FASTCALL, nullptr},
                         {"set_error_type", set_error_type, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "omc_call", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_omc_call() {
  EntryType.tp_name = "omc_call.Entry";
  EntryType.tp_basicsize = sizeof(Entry);
  EntryType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  EntryType.tp_vectorcall_offset = offsetof(Entry, call);
  EntryType.tp_call = PyVectorcall_Call;
  EntryType.tp_dealloc = entry_dealloc;
  if (PyType_Ready(&EntryType) < 0) return nullptr;
  return PyModule_Create(&module);
}
