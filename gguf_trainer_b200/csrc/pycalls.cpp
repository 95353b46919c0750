// The queued entry points as CPython functions. A call through ctypes costs 1.1 to 1.5 us, nearly all of it the conversion of
// the arguments; here the conversion is compiled per signature from include/gguftrain.h and a call costs 0.2 to 0.4 us (four
// tokens decoded by 30 layers: 9.9 -> 8.4 ms). An argument that is not a plain number, the context or an array goes back to
// the ctypes function, which converts or refuses it as before.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <dlfcn.h>
#include <stddef.h>
#include <stdint.h>

#include <tuple>
#include <utility>

#include "../../include/gguftrain.h"

namespace {

// One argument: true and the value, or false with no Python error set.
inline bool take(PyObject* o, int32_t& v) {
  if (!PyLong_Check(o)) return false;
  int over = 0;
  const long l = PyLong_AsLongAndOverflow(o, &over);
  v = (int32_t)l;
  return !over && l == v;
}
inline bool take(PyObject* o, uint64_t& v) {
  if (!PyLong_Check(o)) return false;
  v = PyLong_AsUnsignedLongLong(o);
  if (v == (uint64_t)-1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}
inline bool take(PyObject* o, double& v) {
  if (PyFloat_Check(o)) v = PyFloat_AS_DOUBLE(o);
  else if (PyLong_Check(o)) {
    v = PyLong_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  } else return false;
  return true;
}
inline bool take(PyObject* o, float& v) {
  double d;
  if (!take(o, d)) return false;
  v = (float)d;
  return true;
}
inline bool buffer(PyObject* o, size_t item, void** p, Py_ssize_t* bytes) {
  Py_buffer b;
  if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) { PyErr_Clear(); return false; }
  *p = b.buf;
  *bytes = b.len;
  PyBuffer_Release(&b);       // (the caller's reference keeps the memory)
  return *bytes > 0 && *bytes % item == 0;
}
inline bool take(PyObject* o, gt_ctx*& v) {       // a c_void_p
  void* p;
  Py_ssize_t n;
  if (!buffer(o, 8, &p, &n) || n != 8) return false;
  v = *static_cast<gt_ctx**>(p);
  return v != nullptr;
}
template <typename T>
inline bool take(PyObject* o, const T*& v) {      // a ctypes array of numbers
  void* p;
  Py_ssize_t n;
  if (!buffer(o, sizeof(T), &p, &n)) return false;
  v = static_cast<const T*>(p);
  return true;
}

template <typename... A, size_t... I>
PyObject* invoke(gt_status (*fn)(A...), PyObject* slow, PyObject* const* args, Py_ssize_t n, std::index_sequence<I...>) {
  std::tuple<A...> v;
  if (fn && n == (Py_ssize_t)sizeof...(A) && (take(args[I], std::get<I>(v)) && ...))
    return PyLong_FromLong(fn(std::get<I>(v)...));
  return PyObject_Vectorcall(slow, args, n, nullptr);
}
template <typename... A>
PyObject* invoke(gt_status (*fn)(A...), PyObject* slow, PyObject* const* args, Py_ssize_t n) {
  return invoke(fn, slow, args, n, std::index_sequence_for<A...>());
}

#define GT_CALLS(X)                                                                                                          \
  X(gt_gemm) X(gt_gemm_scaled) X(gt_gemm2) X(gt_gemm_multi) X(gt_gemm_grouped) X(gt_gemm_grouped_scaled)                     \
  X(gt_linear_rope_grouped) X(gt_ew_fwd) X(gt_ew_bwd) X(gt_glu_fwd) X(gt_glu_linear_fwd) X(gt_glu_bwd) X(gt_rmsnorm_fwd)      \
  X(gt_add_rmsnorm_fwd) X(gt_rmsnorm_heads_rope_fwd) X(gt_rmsnorm_bwd) X(gt_rmsnorm_bwd_add) X(gt_embedding_fwd)              \
  X(gt_embedding_bwd) X(gt_rope_fwd) X(gt_rope_bwd) X(gt_attention_fwd) X(gt_attention_bwd) X(gt_attention_bwd_rope)          \
  X(gt_ce_fwd) X(gt_ce_bwd) X(gt_readout_ce_fwd) X(gt_readout_ce_stats) X(gt_readout_ce_grad) X(gt_ce_loss_from_stats) X(gt_zero) X(gt_copy)

#define X(name)                                                                       \
  decltype(&name) fn_##name = nullptr;                                                \
  PyObject* slow_##name = nullptr;                                                    \
  PyObject* py_##name(PyObject*, PyObject* const* args, Py_ssize_t n) {               \
    return invoke(fn_##name, slow_##name, args, n);                                   \
  }
GT_CALLS(X)
#undef X

// bind(handle, functions): the library's handle and its ctypes functions by name
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long handle;
  PyObject* by_name;
  if (!PyArg_ParseTuple(args, "KO!", &handle, &PyDict_Type, &by_name)) return nullptr;
#define X(name)                                                                       \
  {                                                                                   \
    PyObject* f = PyDict_GetItemString(by_name, #name);                               \
    if (!f) return PyErr_Format(PyExc_KeyError, #name);                               \
    Py_INCREF(f);                                                                     \
    Py_XSETREF(slow_##name, f);                                                       \
    fn_##name = (decltype(fn_##name))dlsym((void*)(uintptr_t)handle, #name);          \
  }
  GT_CALLS(X)
#undef X
  Py_RETURN_NONE;
}

// maker(cls, {slot: value}, (slot, ...)): a callable that makes an instance of a class with __slots__, the named slots taken from
// its arguments, the others set to the given values. Written in Python the two records that every op makes, a tensor and
// its device entry, cost 0.9 us of slot stores.
struct Maker {
  PyObject_HEAD
  vectorcallfunc call;
  PyTypeObject* cls;
  Py_ssize_t nargs, nfixed;
  Py_ssize_t arg_at[16], fixed_at[32];
  PyObject* fixed[32];
};
PyObject* make(PyObject* self, PyObject* const* args, size_t nf, PyObject* kw) {
  Maker* m = reinterpret_cast<Maker*>(self);
  if (PyVectorcall_NARGS(nf) != m->nargs || (kw && PyTuple_GET_SIZE(kw)))
    return PyErr_Format(PyExc_TypeError, "%s takes %zd arguments", m->cls->tp_name, m->nargs);
  PyObject* o = m->cls->tp_alloc(m->cls, 0);       // (slots start out null)
  if (!o) return nullptr;
  char* base = reinterpret_cast<char*>(o);
  for (Py_ssize_t i = 0; i < m->nargs; i++) *reinterpret_cast<PyObject**>(base + m->arg_at[i]) = Py_NewRef(args[i]);
  for (Py_ssize_t i = 0; i < m->nfixed; i++) *reinterpret_cast<PyObject**>(base + m->fixed_at[i]) = Py_NewRef(m->fixed[i]);
  return o;
}
void maker_dealloc(PyObject* self) {
  Maker* m = reinterpret_cast<Maker*>(self);
  for (Py_ssize_t i = 0; i < m->nfixed; i++) Py_DECREF(m->fixed[i]);
  Py_XDECREF(m->cls);
  Py_TYPE(self)->tp_free(self);
}
PyTypeObject MakerType = {PyVarObject_HEAD_INIT(nullptr, 0) "_calls.maker", sizeof(Maker)};
Py_ssize_t slot_offset(PyObject* cls, PyObject* name) {
  PyObject* d = PyObject_GetAttr(cls, name);
  if (!d) return -1;
  Py_ssize_t at = -1;
  if (Py_IS_TYPE(d, &PyMemberDescr_Type) && reinterpret_cast<PyMemberDescrObject*>(d)->d_common.d_type == reinterpret_cast<PyTypeObject*>(cls))
    at = reinterpret_cast<PyMemberDescrObject*>(d)->d_member->offset;
  Py_DECREF(d);
  if (at < 0) PyErr_Format(PyExc_TypeError, "%R is no slot of %R", name, cls);
  return at;
}
PyObject* maker(PyObject*, PyObject* args) {
  PyObject *cls, *fixed, *names;
  if (!PyArg_ParseTuple(args, "O!O!O!", &PyType_Type, &cls, &PyDict_Type, &fixed, &PyTuple_Type, &names)) return nullptr;
  if (PyDict_GET_SIZE(fixed) > 32 || PyTuple_GET_SIZE(names) > 16) return PyErr_Format(PyExc_ValueError, "too many slots");
  Maker* m = PyObject_New(Maker, &MakerType);
  if (!m) return nullptr;
  m->call = make;
  m->cls = reinterpret_cast<PyTypeObject*>(Py_NewRef(cls));
  m->nargs = m->nfixed = 0;
  PyObject *k, *v;
  Py_ssize_t pos = 0, at;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(names); i++) {
    if ((at = slot_offset(cls, PyTuple_GET_ITEM(names, i))) < 0) { Py_DECREF(m); return nullptr; }
    m->arg_at[m->nargs++] = at;
  }
  while (PyDict_Next(fixed, &pos, &k, &v)) {
    if ((at = slot_offset(cls, k)) < 0) { Py_DECREF(m); return nullptr; }
    m->fixed_at[m->nfixed] = at;
    m->fixed[m->nfixed++] = Py_NewRef(v);
  }
  return reinterpret_cast<PyObject*>(m);
}

PyMethodDef methods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"maker", maker, METH_VARARGS, nullptr},
#define X(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr},
    GT_CALLS(X)
#undef X
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) {
  MakerType.tp_dealloc = maker_dealloc;
  MakerType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  MakerType.tp_vectorcall_offset = offsetof(Maker, call);
  MakerType.tp_call = PyVectorcall_Call;
  if (PyType_Ready(&MakerType) < 0) return nullptr;
  return PyModule_Create(&module);
}
