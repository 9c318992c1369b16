// Native launch path of generated kernels: what the wrapper code Inductor prints calls once per
// fused kernel, `kernel.run(tensor, ..., size, ..., stream=handle)`.
//
// The call turns its arguments into the two arrays of the generated module's C entry
// (`ixb_gen_launch(ptrs, ints, stream)`) and calls it with the interpreter lock released.  In
// Python (an isinstance test, data_ptr() and a list append per argument, two ctypes arrays, the
// ctypes call) this took 5.3 us; here it takes 0.2.  A compiled call of one small kernel (gelu row
// sum, 64 x 1024) went from 30.2 to 23.8 us, the rest being Dynamo's guards and the wrapper.
// Anything out of the ordinary - a host tensor, a tensor subclass, a size that is not an int, no
// stream - goes to the Python method given as `general`.  A launch that returns a non-zero status is
// not tried again (the status may be an earlier call's, and the kernel may have run): the method is
// called with `status` and words the error.  It stands for the launcher closure of the reference
// (inductor_x/npu_triton_heuristics.py:239-253).
#include <Python.h>
#include <structmember.h>

#include <torch/csrc/autograd/python_variable.h>

namespace {

typedef int (*GenLaunch)(void**, const long long*, void*);
constexpr Py_ssize_t kMaxArgs = 256;  // of one kind; a longer list takes the general route

struct Launcher {
  PyObject_HEAD
  vectorcallfunc call;
  PyObject* general;    // bound Python method with the same arguments
  PyObject* flags;      // the package configuration's dict: its switches hold for every call
  GenLaunch entry;      // 0: every call takes the general route
  long long launches;   // kernels this object has launched itself
};

PyObject *name_profile, *name_dry_run;  // interned: "profile_bandwidth", "dry_run"
PyObject* name_status;                  // ("status",): the keyword of a failed launch

// neither of the two switches that the general route serves is set
bool switches_off(PyObject* flags) {
  return PyDict_GetItem(flags, name_profile) == Py_False && PyDict_GetItem(flags, name_dry_run) == Py_False;
}

PyObject* launch(PyObject* self_, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Launcher* self = reinterpret_cast<Launcher*>(self_);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  void* ptrs[kMaxArgs];
  long long ints[kMaxArgs];
  Py_ssize_t np = 0, ni = 0;
  bool plain = self->entry != nullptr && n <= kMaxArgs && kwnames != nullptr && PyTuple_GET_SIZE(kwnames) == 1 &&
               PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, 0), "stream") == 0 &&
               PyLong_CheckExact(args[n]) && switches_off(self->flags);
  for (Py_ssize_t i = 0; plain && i < n; ++i) {
    PyObject* a = args[i];
    if (PyLong_CheckExact(a)) {
      int overflow = 0;
      ints[ni++] = PyLong_AsLongLongAndOverflow(a, &overflow);
      plain = overflow == 0;
    } else if (THPVariable_CheckExact(a)) {
      try {
        const at::Tensor& t = THPVariable_Unpack(a);
        if ((plain = t.is_cuda() && t.has_storage())) ptrs[np++] = t.data_ptr();
      } catch (...) {
        plain = false;  // whatever it is, the general route raises it as Python does
      }
    } else {
      plain = false;
    }
  }
  if (plain) {
    void* stream = PyLong_AsVoidPtr(args[n]);
    if (stream == nullptr && PyErr_Occurred()) return nullptr;
    GenLaunch entry = self->entry;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = entry(ptrs, ints, stream);
    Py_END_ALLOW_THREADS
    if (rc == 0) {
      ++self->launches;
      Py_RETURN_NONE;
    }
    PyObject* status = PyLong_FromLong(rc);
    if (status == nullptr) return nullptr;
    PyObject* raised = PyObject_Vectorcall(self->general, &status, 0, name_status);
    Py_DECREF(status);
    return raised;
  }
  return PyObject_Vectorcall(self->general, args, nargsf & ~PY_VECTORCALL_ARGUMENTS_OFFSET, kwnames);
}

PyObject* make(PyTypeObject* type, PyObject* args, PyObject*) {
  PyObject *general = nullptr, *flags = nullptr;
  if (!PyArg_ParseTuple(args, "OO!", &general, &PyDict_Type, &flags)) return nullptr;
  Launcher* self = reinterpret_cast<Launcher*>(type->tp_alloc(type, 0));
  if (self == nullptr) return nullptr;
  self->call = launch;
  Py_INCREF(general);
  Py_INCREF(flags);
  self->general = general;
  self->flags = flags;
  self->entry = nullptr;
  self->launches = 0;
  return reinterpret_cast<PyObject*>(self);
}

int traverse(PyObject* self, visitproc visit, void* arg) {
  Py_VISIT(reinterpret_cast<Launcher*>(self)->general);
  Py_VISIT(reinterpret_cast<Launcher*>(self)->flags);
  return 0;
}
int clear(PyObject* self) {
  Py_CLEAR(reinterpret_cast<Launcher*>(self)->general);
  Py_CLEAR(reinterpret_cast<Launcher*>(self)->flags);
  return 0;
}
void dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  clear(self);
  Py_TYPE(self)->tp_free(self);
}

// bind(address): calls go straight to the module's entry; bind(0): to the general route
PyObject* bind(PyObject* self, PyObject* address) {
  void* entry = PyLong_AsVoidPtr(address);
  if (entry == nullptr && PyErr_Occurred()) return nullptr;
  reinterpret_cast<Launcher*>(self)->entry = reinterpret_cast<GenLaunch>(entry);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"bind", bind, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyMemberDef members[] = {{"launches", T_LONGLONG, offsetof(Launcher, launches), READONLY, nullptr},
                         {nullptr, 0, 0, 0, nullptr}};

PyTypeObject LauncherType = {PyVarObject_HEAD_INIT(nullptr, 0)};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_ixb_host", nullptr, -1, nullptr, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ixb_host(void) {
  LauncherType.tp_name = "inductor_x_b200._ixb_host.Launcher";
  LauncherType.tp_basicsize = sizeof(Launcher);
  LauncherType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_HAVE_GC;
  LauncherType.tp_vectorcall_offset = offsetof(Launcher, call);
  LauncherType.tp_call = PyVectorcall_Call;
  LauncherType.tp_new = make;
  LauncherType.tp_dealloc = dealloc;
  LauncherType.tp_traverse = traverse;
  LauncherType.tp_clear = clear;
  LauncherType.tp_methods = methods;
  LauncherType.tp_members = members;
  name_profile = PyUnicode_InternFromString("profile_bandwidth");
  name_dry_run = PyUnicode_InternFromString("dry_run");
  name_status = Py_BuildValue("(s)", "status");
  if (name_profile == nullptr || name_dry_run == nullptr || name_status == nullptr || PyType_Ready(&LauncherType) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module_def);
  if (m == nullptr) return nullptr;
  Py_INCREF(&LauncherType);
  if (PyModule_AddObject(m, "Launcher", reinterpret_cast<PyObject*>(&LauncherType)) < 0) return nullptr;
  return m;
}
