// py_marshal.cpp -- the Python binding's argument conversion in native code
// (module _marshal, loaded by rbk.py and adjoint.py when it is built).
//
// apply(): bra instruction tuples straight to the C ABI's gate calls.  Through
// ctypes each gate took about 1.0 us of interpreter time (20-qubit brick of 423
// instructions: 426 us, a third of the call); here it is some 0.1 us.
// fill_gates(): a parametrised circuit as the array of rbk_circuit_gate that
// the adjoint calls take (960 gates: 558 us in Python).
// Both take the plain forms only and hand any other to the Python code that
// converts through ctypes, so that what is accepted, what is refused and with
// which error do not depend on this module.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <cstring>

#include "rbk.h"

namespace {

// The C ABI's entry points, bound once from the loaded library (bind).
struct abi {
  int (*hadamard)(rbk_state*, uint32_t, const uint32_t*, int);
  int (*pauli_x)(rbk_state*, uint32_t, const uint32_t*, int);
  int (*pauli_y)(rbk_state*, uint32_t, const uint32_t*, int);
  int (*pauli_z)(rbk_state*, const uint32_t*, int);
  int (*phase_shift)(rbk_state*, double, const uint32_t*, int);
  int (*phase_shift_k)(rbk_state*, int, const uint32_t*, int);
  int (*phase_shift2)(rbk_state*, double, double, uint32_t, const uint32_t*, int);
  int (*phase_shift3)(rbk_state*, double, double, double, uint32_t, const uint32_t*, int);
  int (*exp_x)(rbk_state*, double, uint32_t, const uint32_t*, int);
  int (*exp_y)(rbk_state*, double, uint32_t, const uint32_t*, int);
  int (*exp_z)(rbk_state*, double, uint32_t, const uint32_t*, int);
  int (*swap)(rbk_state*, uint32_t, uint32_t, const uint32_t*, int);
  int (*begin_fusion)(rbk_state*);
  int (*end_fusion)(rbk_state*);
} A;
constexpr int kEntries = 14;
static_assert(sizeof(abi) == kEntries * sizeof(void*), "one pointer per entry");
bool bound = false;

PyObject* py_bind(PyObject*, PyObject* args)
{
  PyObject* list;
  if (!PyArg_ParseTuple(args, "O!", &PyList_Type, &list)) return nullptr;
  if (PyList_GET_SIZE(list) != kEntries) {
    PyErr_SetString(PyExc_ValueError, "wrong number of entry points");
    return nullptr;
  }
  void* p[kEntries];
  for (int i = 0; i < kEntries; ++i) {
    p[i] = PyLong_AsVoidPtr(PyList_GET_ITEM(list, i));
    if (PyErr_Occurred()) return nullptr;
  }
  std::memcpy(&A, p, sizeof(p));
  bound = true;
  Py_RETURN_NONE;
}

// A Python object's reference, given back at the end of the scope.
struct held {
  PyObject* o = nullptr;
  explicit held(PyObject* x) : o(x) {}
  held(const held&) = delete;
  ~held() { Py_XDECREF(o); }
};

// A plain tuple or list; its items, nullptr past the end.
inline bool plain(PyObject* x) { return PyTuple_CheckExact(x) || PyList_CheckExact(x); }
inline Py_ssize_t plain_size(PyObject* x) { return PyTuple_CheckExact(x) ? PyTuple_GET_SIZE(x) : PyList_GET_SIZE(x); }
inline PyObject* plain_item(PyObject* x, Py_ssize_t i)
{
  if (i >= plain_size(x)) return nullptr;
  return PyTuple_CheckExact(x) ? PyTuple_GET_ITEM(x, i) : PyList_GET_ITEM(x, i);
}

// x[i] as Python subscripts it, a new reference; nullptr, with an error set or
// not, where there is none.  An object of its own class may run any code.
inline PyObject* subscript(PyObject* x, Py_ssize_t i, bool* foreign)
{
  if (plain(x)) {
    PyObject* o = plain_item(x, i);
    Py_XINCREF(o);
    return o;
  }
  *foreign = true;
  const held index(PyLong_FromSsize_t(i));
  return index.o ? PyObject_GetItem(x, index.o) : nullptr;
}

// The conversions below return false, with an error set or not, where the value
// is one for the ctypes calls to judge.
inline bool as_qubit(PyObject* o, uint32_t* out, bool* foreign)
{
  if (PyLong_CheckExact(o)) {
    *out = static_cast<uint32_t>(PyLong_AsUnsignedLongMask(o));  // a negative index wraps, and is refused as out of range
    return true;
  }
  *foreign = true;
  if (!PyIndex_Check(o)) return false;
  const held v(PyNumber_Index(o));
  if (!v.o) return false;
  *out = static_cast<uint32_t>(PyLong_AsUnsignedLongMask(v.o));
  return !PyErr_Occurred();
}

inline bool as_real(PyObject* o, double* out, bool* foreign)
{
  if (PyFloat_CheckExact(o)) {
    *out = PyFloat_AS_DOUBLE(o);
    return true;
  }
  if (!PyLong_CheckExact(o)) *foreign = true;
  *out = PyFloat_AsDouble(o);
  return !PyErr_Occurred();
}

// int(o), where it fits.
inline bool as_int(PyObject* o, int* out, bool* foreign)
{
  if (PyLong_CheckExact(o)) {
    int overflow = 0;
    *out = static_cast<int>(PyLong_AsLongAndOverflow(o, &overflow));
    return overflow == 0;
  }
  *foreign = true;
  const held v(PyNumber_Long(o));
  if (!v.o) return false;
  const long x = PyLong_AsLong(v.o);
  if (PyErr_Occurred()) return false;
  *out = static_cast<int>(x);
  return true;
}

// float(o): strings of digits too.
inline bool as_float(PyObject* o, double* out, bool* foreign)
{
  if (PyFloat_CheckExact(o)) {
    *out = PyFloat_AS_DOUBLE(o);
    return true;
  }
  if (!PyLong_CheckExact(o)) *foreign = true;
  const held v(PyNumber_Float(o));
  if (!v.o) return false;
  *out = PyFloat_AS_DOUBLE(v.o);
  return true;
}

template <auto as, typename T>
inline bool at(PyObject* x, Py_ssize_t i, T* out, bool* foreign)
{
  const held o(subscript(x, i, foreign));
  return o.o && as(o.o, out, foreign);
}

// Whether an error other than a conversion's (an interrupt, say) is set; a
// conversion's is cleared.
bool hard_error()
{
  if (!PyErr_Occurred()) return false;
  if (!PyErr_ExceptionMatches(PyExc_Exception)) return true;
  PyErr_Clear();
  return false;
}

// The C handle of a State (its attribute h, a c_void_p or None) in *s; 0 with an error set.
int handle_of(PyObject* state, rbk_state** s)
{
  *s = nullptr;
  const held h(PyObject_GetAttrString(state, "h"));
  if (!h.o) return 0;
  if (h.o == Py_None) return 1;
  const held v(PyObject_GetAttrString(h.o, "value"));
  if (!v.o) return 0;
  if (v.o != Py_None) *s = static_cast<rbk_state*>(PyLong_AsVoidPtr(v.o));
  return !PyErr_Occurred();
}

// One instruction.  1: called, with its status in *rc; 0: not of the plain form
// (or one that the ctypes calls refuse, whose error they raise).
int apply_plain(PyObject* state, rbk_state* s, PyObject* op, int* rc, bool* foreign)
{
  if (!plain(op) || plain_size(op) != 3 || !PyUnicode_CheckExact(plain_item(op, 0))) return 0;
  const held name_o(Py_NewRef(plain_item(op, 0))), q_o(Py_NewRef(plain_item(op, 1))), p_o(Py_NewRef(plain_item(op, 2)));
  PyObject *q = q_o.o, *p = p_o.o;
  Py_ssize_t length = 0;
  const char* name = PyUnicode_AsUTF8AndSize(name_o.o, &length);
  if (!name || std::strlen(name) != static_cast<size_t>(length)) return 0;
  uint32_t a = 0, b = 0;
  double x = 0, y = 0, z = 0;
  int n = 0;
  const uint32_t* none = nullptr;
  // Foreign code may have closed the state.
  auto usable = [&] { return !*foreign || (handle_of(state, &s) && s); };
  auto qubit = [&](Py_ssize_t i, uint32_t* out) { return at<as_qubit>(q, i, out, foreign); };
  auto real = [&](Py_ssize_t i, double* out) { return at<as_real>(p, i, out, foreign); };
#define RBK_CALL(expr) { if (!usable()) return 0; Py_BEGIN_ALLOW_THREADS *rc = (expr); Py_END_ALLOW_THREADS return 1; }
  if (!std::strcmp(name, "U3")) {
    if (real(0, &x) && real(1, &y) && real(2, &z) && qubit(0, &a)) RBK_CALL(A.phase_shift3(s, x, y, z, a, none, 0))
  } else if (!std::strcmp(name, "CNOT")) {
    if (qubit(1, &b) && qubit(0, &a)) RBK_CALL(A.pauli_x(s, b, &a, 1))
  } else if (!std::strcmp(name, "H")) {
    if (qubit(0, &a)) RBK_CALL(A.hadamard(s, a, none, 0))
  } else if (!std::strcmp(name, "X")) {
    if (qubit(0, &a)) RBK_CALL(A.pauli_x(s, a, none, 0))
  } else if (!std::strcmp(name, "Y")) {
    if (qubit(0, &a)) RBK_CALL(A.pauli_y(s, a, none, 0))
  } else if (!std::strcmp(name, "Z")) {
    if (qubit(0, &a)) RBK_CALL(A.pauli_z(s, &a, 1))
  } else if (!std::strcmp(name, "U1")) {
    if (real(0, &x) && qubit(0, &a)) RBK_CALL(A.phase_shift(s, x, &a, 1))
  } else if (!std::strcmp(name, "U2")) {
    if (real(0, &x) && real(1, &y) && qubit(0, &a)) RBK_CALL(A.phase_shift2(s, x, y, a, none, 0))
  } else if (!std::strcmp(name, "CZ")) {
    uint32_t qs[2];
    if (qubit(0, &qs[0]) && qubit(1, &qs[1])) RBK_CALL(A.pauli_z(s, qs, 2))
  } else if (!std::strcmp(name, "U")) {
    uint32_t qs[2];
    if (at<as_int>(p, 0, &n, foreign) && qubit(0, &qs[0]) && qubit(1, &qs[1])) RBK_CALL(A.phase_shift_k(s, n, qs, 2))
  } else if (!std::strcmp(name, "EY")) {
    if (real(0, &x) && qubit(0, &a)) RBK_CALL(A.exp_y(s, x, a, none, 0))
  } else if (!std::strcmp(name, "EZ")) {
    if (real(0, &x) && qubit(0, &a)) RBK_CALL(A.exp_z(s, x, a, none, 0))
  } else if (!std::strcmp(name, "EX")) {
    if (real(0, &x) && qubit(0, &a)) RBK_CALL(A.exp_x(s, x, a, none, 0))
  } else if (!std::strcmp(name, "SWAP")) {
    if (qubit(0, &a) && qubit(1, &b)) RBK_CALL(A.swap(s, a, b, none, 0))
  } else if (!std::strcmp(name, "BEGIN FUSION")) {
    RBK_CALL(A.begin_fusion(s))
  } else if (!std::strcmp(name, "END FUSION")) {
    RBK_CALL(A.end_fusion(s))
  }
#undef RBK_CALL
  return 0;
}

// apply(state, ops, one): every instruction in order; the first failing call's
// status code, or 0.  Instructions of the plain form -- a tuple or list of a known
// mnemonic, qubits and parameters that convert -- go straight to the C ABI; one(op)
// takes any other.  The handle is read again wherever Python code may have run.
PyObject* py_apply(PyObject*, PyObject* args)
{
  PyObject *state, *ops, *one;
  if (!PyArg_ParseTuple(args, "OOO", &state, &ops, &one)) return nullptr;
  if (!bound) {
    PyErr_SetString(PyExc_RuntimeError, "entry points not bound");
    return nullptr;
  }
  const bool list = plain(ops);
  const held it(list ? nullptr : PyObject_GetIter(ops));
  if (!list && !it.o) return nullptr;
  rbk_state* s = nullptr;
  bool foreign = true;
  int rc = 0;
  for (Py_ssize_t k = 0; rc == 0; ++k) {
    PyObject* item = list ? plain_item(ops, k) : PyIter_Next(it.o);
    if (!item) {
      if (PyErr_Occurred()) return nullptr;
      break;
    }
    if (list) Py_INCREF(item);
    const held op(item);  // held: a call below runs without the interpreter's lock
    if (!list) foreign = true;
    if (foreign && !handle_of(state, &s)) return nullptr;
    foreign = false;
    if (s && apply_plain(state, s, op.o, &rc, &foreign)) continue;
    if (hard_error()) return nullptr;
    const held r(PyObject_CallOneArg(one, op.o));
    if (!r.o) return nullptr;
    foreign = true;
  }
  return PyLong_FromLong(rc);
}

// x[:n] as Python slices it: a tuple or list of which the first n items count.  A new reference.
inline PyObject* first_of(PyObject* x, Py_ssize_t n)
{
  if (plain(x)) return Py_NewRef(x);
  const held part(PySequence_GetSlice(x, 0, n));
  return part.o ? PySequence_Tuple(part.o) : nullptr;
}

// One gate of the plain form in *r; false otherwise.
bool gate_plain(PyObject* g, PyObject* kinds, rbk_circuit_gate* r)
{
  if (!plain(g) || plain_size(g) != 5) return false;
  const held name(Py_NewRef(plain_item(g, 0))), q_o(Py_NewRef(plain_item(g, 1))), param(Py_NewRef(plain_item(g, 2))),
    scale(Py_NewRef(plain_item(g, 3))), angles_o(Py_NewRef(plain_item(g, 4)));
  PyObject* kind = PyDict_GetItemWithError(kinds, name.o);
  if (!kind) return false;
  std::memset(r, 0, sizeof(*r));
  bool foreign = false;
  int v = 0;
  if (!as_int(kind, &v, &foreign)) return false;
  r->kind = v;
  const held q(first_of(q_o.o, 2));
  if (!q.o) return false;
  for (Py_ssize_t j = 0; j < 2 && j < plain_size(q.o); ++j) {
    if (!at<as_int>(q.o, j, &v, &foreign)) return false;
    r->qubits[j] = v;
  }
  r->param = -1;
  if (param.o != Py_None) {
    if (!as_int(param.o, &v, &foreign)) return false;
    r->param = v;
  }
  if (!as_float(scale.o, &r->scale, &foreign)) return false;
  const held angles(first_of(angles_o.o, 3));
  if (!angles.o) return false;
  for (Py_ssize_t j = 0; j < 3 && j < plain_size(angles.o); ++j)
    if (!at<as_float>(angles.o, j, &r->angles[j], &foreign)) return false;
  return true;
}

// fill_gates(address, count, spec, kinds, one): spec's (mnemonic, qubits, param, scale,
// angles) as rbk_circuit_gate records at `address`, where `count` have room; kinds:
// {mnemonic: code}.  one(i, gate) takes gates that are not of the plain form, and
// any past the room.
PyObject* py_fill_gates(PyObject*, PyObject* args)
{
  PyObject *address, *spec, *kinds, *one;
  Py_ssize_t count;
  if (!PyArg_ParseTuple(args, "OnOO!O", &address, &count, &spec, &PyDict_Type, &kinds, &one)) return nullptr;
  rbk_circuit_gate* out = static_cast<rbk_circuit_gate*>(PyLong_AsVoidPtr(address));
  if (PyErr_Occurred()) return nullptr;
  const bool list = plain(spec);
  const held it(list ? nullptr : PyObject_GetIter(spec));
  if (!list && !it.o) return nullptr;
  for (Py_ssize_t k = 0;; ++k) {
    PyObject* item = list ? plain_item(spec, k) : PyIter_Next(it.o);
    if (!item) {
      if (PyErr_Occurred()) return nullptr;
      break;
    }
    if (list) Py_INCREF(item);
    const held g(item);
    rbk_circuit_gate r;
    if (k < count && gate_plain(g.o, kinds, &r)) {
      out[k] = r;
      continue;
    }
    if (hard_error()) return nullptr;
    const held index(PyLong_FromSsize_t(k));
    if (!index.o) return nullptr;
    const held done(PyObject_CallFunctionObjArgs(one, index.o, g.o, nullptr));
    if (!done.o) return nullptr;
  }
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
  {"bind", py_bind, METH_VARARGS, "bind(addresses): the C ABI's entry points"},
  {"apply", py_apply, METH_VARARGS, "apply(state, ops, one): status code of the first failing call, or 0"},
  {"fill_gates", py_fill_gates, METH_VARARGS, "fill_gates(address, count, spec, kinds, one)"},
  {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_marshal", "Argument conversion of the binding", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__marshal(void) { return PyModule_Create(&module); }
