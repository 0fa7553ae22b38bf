// py_marshal.cpp -- the Python binding's argument conversion in native code
// (module _marshal, loaded by rbk.py and adjoint.py when it is built).
//
// apply(): bra instruction tuples straight to the C ABI's gate calls.  Through
// ctypes each gate took about 1.0 us of interpreter time (20-qubit brick of 423
// instructions: 426 us, a third of the call); here it is some 0.1 us.
// fill_gates(): a parametrised circuit as the array of rbk_circuit_gate that
// the adjoint calls take (960 gates: 558 us in Python).
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

// A tuple or list as it is, any other sequence (a numpy row, say) as a new tuple.
struct as_sequence {
  PyObject* o = nullptr;
  explicit as_sequence(PyObject* x)
  {
    if (!x) return;
    if (PyTuple_Check(x) || PyList_Check(x)) {
      Py_INCREF(x);
      o = x;
    } else {
      o = PySequence_Tuple(x);
    }
  }
  as_sequence(const as_sequence&) = delete;
  ~as_sequence() { Py_XDECREF(o); }
};

// Element i of a tuple or list, borrowed; nullptr with IndexError set when there is none.
PyObject* item(PyObject* seq, Py_ssize_t i)
{
  if (!seq) return nullptr;  // an error is set
  if (PyTuple_Check(seq)) {
    if (i < PyTuple_GET_SIZE(seq)) return PyTuple_GET_ITEM(seq, i);
  } else if (PyList_Check(seq)) {
    if (i < PyList_GET_SIZE(seq)) return PyList_GET_ITEM(seq, i);
  } else {
    PyErr_SetString(PyExc_TypeError, "expected a tuple or list");
    return nullptr;
  }
  PyErr_SetString(PyExc_IndexError, "tuple index out of range");
  return nullptr;
}

bool get_qubit(PyObject* seq, Py_ssize_t i, uint32_t* out)
{
  PyObject* o = item(seq, i);
  if (!o) return false;
  PyObject* idx = PyNumber_Index(o);
  if (!idx) return false;
  *out = static_cast<uint32_t>(PyLong_AsUnsignedLongMask(idx));  // a negative index wraps, and is refused as out of range
  Py_DECREF(idx);
  return !PyErr_Occurred();
}

bool get_real(PyObject* seq, Py_ssize_t i, double* out)
{
  PyObject* o = item(seq, i);
  if (!o) return false;
  *out = PyFloat_AsDouble(o);
  return !PyErr_Occurred();
}

// As float(x) takes it: strings of digits too.
bool get_float(PyObject* seq, Py_ssize_t i, double* out)
{
  PyObject* o = item(seq, i);
  PyObject* v = o ? PyNumber_Float(o) : nullptr;
  if (!v) return false;
  *out = PyFloat_AS_DOUBLE(v);
  Py_DECREF(v);
  return true;
}

// int(value) of element i.
bool get_int(PyObject* seq, Py_ssize_t i, int* out)
{
  PyObject* o = item(seq, i);
  if (!o) return false;
  PyObject* v = PyNumber_Long(o);
  if (!v) return false;
  const long x = PyLong_AsLong(v);
  Py_DECREF(v);
  if (PyErr_Occurred()) return false;
  *out = static_cast<int>(x);
  return true;
}

// apply(state, ops): every instruction in order; the first failing call's status code, or 0.
PyObject* py_apply(PyObject*, PyObject* args)
{
  PyObject *handle, *ops;
  if (!PyArg_ParseTuple(args, "OO", &handle, &ops)) return nullptr;
  if (!bound) {
    PyErr_SetString(PyExc_RuntimeError, "entry points not bound");
    return nullptr;
  }
  rbk_state* s = static_cast<rbk_state*>(PyLong_AsVoidPtr(handle));
  if (PyErr_Occurred()) return nullptr;
  PyObject* seq = PySequence_Fast(ops, "instructions must be a sequence");
  if (!seq) return nullptr;
  int rc = 0;
  bool ok = true;
  for (Py_ssize_t k = 0; ok && rc == 0 && k < PySequence_Fast_GET_SIZE(seq); ++k) {
    // References are held: a call below runs without the interpreter's lock.
    const as_sequence held(PySequence_Fast_GET_ITEM(seq, k));
    PyObject* op = held.o;
    if (!op || PySequence_Fast_GET_SIZE(op) != 3) {
      if (op) PyErr_SetString(PyExc_ValueError, "an instruction is (mnemonic, qubits, params)");
      ok = false;
      break;
    }
    const as_sequence qubits(item(op, 1)), params(item(op, 2));
    PyObject *q = qubits.o, *p = params.o;
    if (!q || !p) {
      ok = false;
      break;
    }
    const char* name = PyUnicode_Check(item(op, 0)) ? PyUnicode_AsUTF8(item(op, 0)) : nullptr;
    uint32_t a = 0, b = 0;
    double x = 0, y = 0, z = 0;
    int n = 0;
#define RBK_CALL(expr) { Py_BEGIN_ALLOW_THREADS rc = (expr); Py_END_ALLOW_THREADS }
    const uint32_t* none = nullptr;
    if (!name) {
      PyErr_Clear();
      PyErr_Format(PyExc_ValueError, "unsupported instruction %S", item(op, 0));
      ok = false;
    } else if (!std::strcmp(name, "U3")) {
      if ((ok = get_real(p, 0, &x) && get_real(p, 1, &y) && get_real(p, 2, &z) && get_qubit(q, 0, &a))) RBK_CALL(A.phase_shift3(s, x, y, z, a, none, 0))
    } else if (!std::strcmp(name, "CNOT")) {
      if ((ok = get_qubit(q, 1, &b) && get_qubit(q, 0, &a))) RBK_CALL(A.pauli_x(s, b, &a, 1))
    } else if (!std::strcmp(name, "H")) {
      if ((ok = get_qubit(q, 0, &a))) RBK_CALL(A.hadamard(s, a, none, 0))
    } else if (!std::strcmp(name, "X")) {
      if ((ok = get_qubit(q, 0, &a))) RBK_CALL(A.pauli_x(s, a, none, 0))
    } else if (!std::strcmp(name, "Y")) {
      if ((ok = get_qubit(q, 0, &a))) RBK_CALL(A.pauli_y(s, a, none, 0))
    } else if (!std::strcmp(name, "Z")) {
      if ((ok = get_qubit(q, 0, &a))) RBK_CALL(A.pauli_z(s, &a, 1))
    } else if (!std::strcmp(name, "U1")) {
      if ((ok = get_real(p, 0, &x) && get_qubit(q, 0, &a))) RBK_CALL(A.phase_shift(s, x, &a, 1))
    } else if (!std::strcmp(name, "U2")) {
      if ((ok = get_real(p, 0, &x) && get_real(p, 1, &y) && get_qubit(q, 0, &a))) RBK_CALL(A.phase_shift2(s, x, y, a, none, 0))
    } else if (!std::strcmp(name, "CZ")) {
      uint32_t qs[2];
      if ((ok = get_qubit(q, 0, &qs[0]) && get_qubit(q, 1, &qs[1]))) RBK_CALL(A.pauli_z(s, qs, 2))
    } else if (!std::strcmp(name, "U")) {
      uint32_t qs[2];
      if ((ok = get_int(p, 0, &n) && get_qubit(q, 0, &qs[0]) && get_qubit(q, 1, &qs[1]))) RBK_CALL(A.phase_shift_k(s, n, qs, 2))
    } else if (!std::strcmp(name, "EY")) {
      if ((ok = get_real(p, 0, &x) && get_qubit(q, 0, &a))) RBK_CALL(A.exp_y(s, x, a, none, 0))
    } else if (!std::strcmp(name, "EZ")) {
      if ((ok = get_real(p, 0, &x) && get_qubit(q, 0, &a))) RBK_CALL(A.exp_z(s, x, a, none, 0))
    } else if (!std::strcmp(name, "EX")) {
      if ((ok = get_real(p, 0, &x) && get_qubit(q, 0, &a))) RBK_CALL(A.exp_x(s, x, a, none, 0))
    } else if (!std::strcmp(name, "SWAP")) {
      if ((ok = get_qubit(q, 0, &a) && get_qubit(q, 1, &b))) RBK_CALL(A.swap(s, a, b, none, 0))
    } else if (!std::strcmp(name, "BEGIN FUSION")) {
      RBK_CALL(A.begin_fusion(s))
    } else if (!std::strcmp(name, "END FUSION")) {
      RBK_CALL(A.end_fusion(s))
    } else {
      PyErr_Format(PyExc_ValueError, "unsupported instruction %s", name);
      ok = false;
    }
#undef RBK_CALL
  }
  Py_DECREF(seq);
  return ok ? PyLong_FromLong(rc) : nullptr;
}

// fill_gates(address, spec, kinds): spec's (mnemonic, qubits, param, scale, angles)
// as rbk_circuit_gate records at `address` (room for len(spec)); kinds: {mnemonic: code}.
PyObject* py_fill_gates(PyObject*, PyObject* args)
{
  PyObject *address, *spec, *kinds;
  if (!PyArg_ParseTuple(args, "OOO!", &address, &spec, &PyDict_Type, &kinds)) return nullptr;
  rbk_circuit_gate* out = static_cast<rbk_circuit_gate*>(PyLong_AsVoidPtr(address));
  if (PyErr_Occurred()) return nullptr;
  PyObject* seq = PySequence_Fast(spec, "a circuit must be a sequence");
  if (!seq) return nullptr;
  for (Py_ssize_t k = 0; k < PySequence_Fast_GET_SIZE(seq); ++k) {
    const as_sequence held(PySequence_Fast_GET_ITEM(seq, k));
    PyObject* g = held.o;
    if (!g || PySequence_Fast_GET_SIZE(g) != 5) {
      if (g) PyErr_SetString(PyExc_ValueError, "a gate is (mnemonic, qubits, param, scale, angles)");
      break;
    }
    rbk_circuit_gate r;
    std::memset(&r, 0, sizeof(r));
    PyObject* kind = PyDict_GetItemWithError(kinds, item(g, 0));
    if (!kind) {
      if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, item(g, 0));
      break;
    }
    r.kind = static_cast<int32_t>(PyLong_AsLong(kind));
    const as_sequence qubits(item(g, 1)), turns(item(g, 4));
    PyObject *q = qubits.o, *angles = turns.o;
    if (!q || !angles) break;
    int v = 0;
    bool ok = true;
    for (Py_ssize_t j = 0; ok && j < 2 && j < PySequence_Fast_GET_SIZE(q); ++j)
      if ((ok = get_int(q, j, &v))) r.qubits[j] = v;
    r.param = -1;
    if (ok && item(g, 2) != Py_None && (ok = get_int(g, 2, &v))) r.param = v;
    ok = ok && get_float(g, 3, &r.scale);
    for (Py_ssize_t j = 0; ok && j < 3 && j < PySequence_Fast_GET_SIZE(angles); ++j) ok = get_float(angles, j, &r.angles[j]);
    if (!ok) break;
    out[k] = r;
  }
  Py_DECREF(seq);
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
  {"bind", py_bind, METH_VARARGS, "bind(addresses): the C ABI's entry points"},
  {"apply", py_apply, METH_VARARGS, "apply(state, ops): status code of the first failing call, or 0"},
  {"fill_gates", py_fill_gates, METH_VARARGS, "fill_gates(address, spec, kinds)"},
  {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_marshal", "Argument conversion of the binding", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__marshal(void) { return PyModule_Create(&module); }
