// Native launch paths: of generated kernels - what the wrapper code Inductor prints calls once per
// fused kernel, `kernel.run(tensor, ..., size, ..., stream=handle)` - and of three library entry points
// whose calls are short enough for the host to count (rms_norm, fused_attention and its backward, at the
// end of this file).
//
// The call of a generated kernel turns its arguments into the two arrays of the generated module's C entry
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

#include <ATen/Functions.h>
#include <c10/core/Allocator.h>
#include <c10/core/DeviceGuard.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/ixb.h"

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

// ---- library entry points ------------------------------------------------------------------------
// Each takes the arguments of the Python function of the same purpose (ops.py), does what it does for a
// plain call - checks, allocations, strides, the C entry on the current stream - and returns the
// result; a status other than 0 comes back as an int, which the caller words.  Anything else (a tensor
// subclass or a wrapper without storage, a host tensor, a shape, dtype or layout that Python would
// refuse or copy, a dispatch mode that wants to see the allocations, an exception) gives None: the
// Python function then goes its own way, errors included.
// A call of rms_norm (16 x 4096 bf16 with residual) took 9.5 us in Python, launch and two
// allocations included.
decltype(&ixb_rmsnorm) entry_rmsnorm;
decltype(&ixb_fa_fwd) entry_fa_fwd;
decltype(&ixb_fa_bwd_scratch_bytes) entry_fa_bwd_room;
decltype(&ixb_fa_bwd_scratch) entry_fa_bwd;

// bind_library(rmsnorm, fa_fwd, fa_bwd_scratch_bytes, fa_bwd_scratch): addresses of the C entries
PyObject* bind_library(PyObject*, PyObject* const* args, Py_ssize_t n) {
  void* p[4];
  if (n != 4) {
    PyErr_SetString(PyExc_TypeError, "bind_library takes four addresses");
    return nullptr;
  }
  for (int i = 0; i < 4; ++i) {
    p[i] = PyLong_AsVoidPtr(args[i]);
    if (p[i] == nullptr && PyErr_Occurred()) return nullptr;
  }
  entry_rmsnorm = reinterpret_cast<decltype(entry_rmsnorm)>(p[0]);
  entry_fa_fwd = reinterpret_cast<decltype(entry_fa_fwd)>(p[1]);
  entry_fa_bwd_room = reinterpret_cast<decltype(entry_fa_bwd_room)>(p[2]);
  entry_fa_bwd = reinterpret_cast<decltype(entry_fa_bwd)>(p[3]);
  Py_RETURN_NONE;
}

PyObject* left_to_python() {
  PyErr_Clear();   // (an exception that came out of Python code leaves its error set)
  Py_RETURN_NONE;
}
bool observed() { return c10::impl::TorchDispatchModeTLS::any_modes_set(); }

// a CUDA tensor with memory of its own kind behind it
const at::Tensor* plain_tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && t.has_storage() ? &t : nullptr;
}
int dtype_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return IXB_F32;
    case at::kHalf: return IXB_F16;
    case at::kBFloat16: return IXB_BF16;
    default: return -1;
  }
}
bool alike(const at::Tensor& a, const at::Tensor& b) {
  return a.scalar_type() == b.scalar_type() && a.device() == b.device();
}
ixb_stream stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
PyObject* pair(at::Tensor a, at::Tensor b) {
  PyObject *x = THPVariable_Wrap(std::move(a)), *y = x ? THPVariable_Wrap(std::move(b)) : nullptr;
  PyObject* out = y ? PyTuple_Pack(2, x, y) : nullptr;
  Py_XDECREF(x);
  Py_XDECREF(y);
  return out;
}

// rms_norm(x, w, eps, residual or None, return_residual)
PyObject* rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 5 || entry_rmsnorm == nullptr || observed() || !PyFloat_CheckExact(args[2]) || !PyBool_Check(args[4])) Py_RETURN_NONE;
  try {
    const at::Tensor *x = plain_tensor(args[0]), *w = plain_tensor(args[1]);
    if (x == nullptr || w == nullptr || x->dim() < 1 || !x->is_contiguous() || dtype_code(*x) < 0) Py_RETURN_NONE;
    const int64_t cols = x->size(-1), rows = cols ? x->numel() / cols : 0;
    if (!alike(*x, *w) || w->dim() != 1 || w->size(0) != cols || !w->is_contiguous()) Py_RETURN_NONE;
    const at::Tensor* r = nullptr;
    if (args[3] != Py_None) {
      r = plain_tensor(args[3]);
      if (r == nullptr || !alike(*x, *r) || r->sizes() != x->sizes() || !r->is_contiguous()) Py_RETURN_NONE;
    }
    at::Tensor y = at::empty_like(*x), h;
    if (r != nullptr && args[4] == Py_True) h = at::empty_like(*x);
    const ixb_stream stream = stream_of(*x);
    const float eps = (float)PyFloat_AS_DOUBLE(args[2]);
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = entry_rmsnorm(dtype_code(*x), x->data_ptr(), r ? r->data_ptr() : nullptr, w->data_ptr(), y.data_ptr(),
                       h.defined() ? h.data_ptr() : nullptr, rows, cols, eps, nullptr, stream);
    Py_END_ALLOW_THREADS
    if (st != 0) return PyLong_FromLong(st);
    return h.defined() ? pair(std::move(y), std::move(h)) : THPVariable_Wrap(std::move(y));
  } catch (...) {
    return left_to_python();
  }
}

struct Strides {
  int64_t v[3];
  explicit Strides(const at::Tensor& t) : v{t.stride(0), t.stride(1), t.stride(2)} {}
};
// q[B, H, Sq, D], k and v [B, H, Sk, D], 16-bit, D contiguous
bool attention_operands(const at::Tensor* q, const at::Tensor* k, const at::Tensor* v) {
  return q && k && v && q->dim() == 4 && k->dim() == 4 && k->sizes() == v->sizes() && q->size(0) == k->size(0) &&
         q->size(1) == k->size(1) && q->size(3) == k->size(3) && dtype_code(*q) > IXB_F32 && alike(*q, *k) && alike(*q, *v) &&
         q->stride(3) == 1 && k->stride(3) == 1 && v->stride(3) == 1 && q->numel() <= INT32_MAX * (int64_t)128 &&
         k->numel() <= INT32_MAX * (int64_t)128;
}

// fused_attention(q, k, v, scale, causal, return_lse)
PyObject* fused_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 6 || entry_fa_fwd == nullptr || observed() || !PyFloat_CheckExact(args[3]) || !PyBool_Check(args[4]) || !PyBool_Check(args[5]))
    Py_RETURN_NONE;
  try {
    const at::Tensor *q = plain_tensor(args[0]), *k = plain_tensor(args[1]), *v = plain_tensor(args[2]);
    if (!attention_operands(q, k, v)) Py_RETURN_NONE;
    const int64_t B = q->size(0), H = q->size(1), Sq = q->size(2), D = q->size(3), Sk = k->size(2);
    at::Tensor out = at::empty({B, H, Sq, D}, q->options()), lse;
    if (args[5] == Py_True) lse = at::empty({B, H, Sq}, q->options().dtype(at::kFloat));
    const Strides qs(*q), ks(*k), vs(*v), os(out);
    const ixb_stream stream = stream_of(*q);
    const float scale = (float)PyFloat_AS_DOUBLE(args[3]);
    const int causal = args[4] == Py_True;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = entry_fa_fwd(dtype_code(*q), q->data_ptr(), k->data_ptr(), v->data_ptr(), out.data_ptr(),
                      lse.defined() ? static_cast<float*>(lse.data_ptr()) : nullptr, (int32_t)B, (int32_t)H, (int32_t)Sq,
                      (int32_t)Sk, (int32_t)D, qs.v, ks.v, vs.v, os.v, scale, causal, nullptr, stream);
    Py_END_ALLOW_THREADS
    if (st != 0) return PyLong_FromLong(st);
    return lse.defined() ? pair(std::move(out), std::move(lse)) : THPVariable_Wrap(std::move(out));
  } catch (...) {
    return left_to_python();
  }
}

// fused_attention_backward(q, k, v, out, lse, dout, scale, causal, bytes of dS at most); False where all
// but the memory for dS was to be had, so that the caller does not ask for the same again
PyObject* fused_attention_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 9 || entry_fa_bwd == nullptr || observed() || !PyFloat_CheckExact(args[6]) || !PyBool_Check(args[7]) || !PyLong_CheckExact(args[8]))
    Py_RETURN_NONE;
  try {
    const at::Tensor *q = plain_tensor(args[0]), *k = plain_tensor(args[1]), *v = plain_tensor(args[2]),
                     *o = plain_tensor(args[3]), *lse = plain_tensor(args[4]), *go = plain_tensor(args[5]);
    const long long limit = PyLong_AsLongLong(args[8]);
    if (limit < 0) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    if (!attention_operands(q, k, v) || !o || !lse || !go || o->sizes() != q->sizes() || go->sizes() != q->sizes() ||
        !alike(*q, *o) || !alike(*q, *go) || o->stride(3) != 1 || go->stride(3) != 1)
      Py_RETURN_NONE;
    const int64_t B = q->size(0), H = q->size(1), Sq = q->size(2), D = q->size(3), Sk = k->size(2);
    for (int i = 0; i < 3; ++i)
      if (go->stride(i) % 8 != 0) Py_RETURN_NONE;
    if (lse->dim() != 3 || lse->size(0) != B || lse->size(1) != H || lse->size(2) != Sq ||
        lse->scalar_type() != at::kFloat || lse->device() != q->device() || !lse->is_contiguous())
      Py_RETURN_NONE;
    at::Tensor dq = at::empty({B, H, Sq, D}, q->options()), dk = at::empty({B, H, Sk, D}, q->options()),
               dv = at::empty({B, H, Sk, D}, q->options());
    const int causal = args[7] == Py_True;
    const size_t room = entry_fa_bwd_room((int32_t)B, (int32_t)H, (int32_t)Sq, (int32_t)Sk, causal, (size_t)limit);
    // memory as it is: at::empty would fill it where torch's deterministic algorithms are asked for
    // (4 x 32 heads of 4096 causal keys: 2359 us a call, 1662 without them)
    const c10::OptionalDeviceGuard device(q->device());
    c10::DataPtr scratch;
    try {
      scratch = c10::GetAllocator(c10::kCUDA)->allocate(room + 4 * (size_t)(B * H * Sq));
    } catch (const c10::OutOfMemoryError&) {
      if (room > 0) Py_RETURN_FALSE;
      throw;
    }
    unsigned char* base = static_cast<unsigned char*>(scratch.get());
    const Strides qs(*q), ks(*k), vs(*v), os(*o), gs(*go), dqs(dq), dks(dk), dvs(dv);
    const ixb_stream stream = stream_of(*q);
    const float scale = (float)PyFloat_AS_DOUBLE(args[6]);
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = entry_fa_bwd(dtype_code(*q), q->data_ptr(), k->data_ptr(), v->data_ptr(), o->data_ptr(), go->data_ptr(),
                      static_cast<const float*>(lse->data_ptr()), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                      reinterpret_cast<float*>(base + room), room ? base : nullptr, room, (int32_t)B, (int32_t)H,
                      (int32_t)Sq, (int32_t)Sk, (int32_t)D, qs.v, ks.v, vs.v, os.v, gs.v, dqs.v, dks.v, dvs.v, scale, causal,
                      nullptr, stream);
    Py_END_ALLOW_THREADS
    if (st != 0) return PyLong_FromLong(st);
    PyObject* rest = pair(std::move(dk), std::move(dv));
    PyObject* first = rest ? THPVariable_Wrap(std::move(dq)) : nullptr;
    PyObject* all = first ? PyTuple_Pack(3, first, PyTuple_GET_ITEM(rest, 0), PyTuple_GET_ITEM(rest, 1)) : nullptr;
    Py_XDECREF(first);
    Py_XDECREF(rest);
    return all;
  } catch (...) {
    return left_to_python();
  }
}

#define IXB_FASTCALL(fn) {#fn, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fn)), METH_FASTCALL, nullptr}
PyMethodDef functions[] = {IXB_FASTCALL(bind_library), IXB_FASTCALL(rms_norm), IXB_FASTCALL(fused_attention),
                           IXB_FASTCALL(fused_attention_backward), {nullptr, nullptr, 0, nullptr}};

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
  module_def.m_methods = functions;
  PyObject* m = PyModule_Create(&module_def);
  if (m == nullptr) return nullptr;
  Py_INCREF(&LauncherType);
  if (PyModule_AddObject(m, "Launcher", reinterpret_cast<PyObject*>(&LauncherType)) < 0) return nullptr;
  return m;
}
