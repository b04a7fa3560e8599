// Device addresses of a list of expert slots, read from the tensors themselves.  A prefill call names over a thousand matrices and
// the GPU waits for it: data_ptr() through the interpreter takes 85 us for 384 experts, this 10.
#include <torch/csrc/autograd/python_variable.h>
#include <cstdint>

// The PyTorch and Python whose headers this was compiled with: their objects' layout is not promised to be another's.
extern "C" const char* msb_host_built_for() { return MSB_BUILT_FOR; }

namespace {
bool address(PyObject* t, uint64_t* out) {
  if (t == Py_None) { *out = 0; return true; }
  if (!THPVariable_Check(t) || !THPVariable_Unpack(t).is_cuda()) return false;
  *out = reinterpret_cast<uint64_t>(THPVariable_Unpack(t).data_ptr());
  return true;
}
}  // namespace

// slots: sequence of at most n objects with attributes gate, up and down, each a device tensor or None; out: [n][3], 0 for None.
// One that is exactly a `cls` (ExpertSlot) keeps them in a tuple _m, a single attribute to fetch; the others' are asked for one by
// one.  Returns 0, or -1 with a Python exception set (called with the interpreter lock held).
extern "C" int msb_slot_addresses(PyObject* slots, PyObject* cls, int64_t n, uint64_t* out) {
  static PyObject* const packed = PyUnicode_InternFromString("_m");
  static PyObject* const names[3] = {PyUnicode_InternFromString("gate"), PyUnicode_InternFromString("up"), PyUnicode_InternFromString("down")};
  PyObject* seq = PySequence_Fast(slots, "expert slots: a sequence expected");
  if (!seq) return -1;
  bool ok = PySequence_Fast_GET_SIZE(seq) <= n;
  if (!ok) PyErr_SetString(PyExc_IndexError, "more expert slots than counted");
  for (Py_ssize_t i = 0; ok && i < PySequence_Fast_GET_SIZE(seq); i++) {
    PyObject* s = PySequence_Fast_GET_ITEM(seq, i);
    if (reinterpret_cast<PyObject*>(Py_TYPE(s)) == cls) {
      PyObject* m = PyObject_GetAttr(s, packed);
      ok = m && PyTuple_Check(m) && PyTuple_GET_SIZE(m) == 3;
      for (int k = 0; ok && k < 3; k++) ok = address(PyTuple_GET_ITEM(m, k), out + 3 * i + k);
      Py_XDECREF(m);
    } else {
      for (int k = 0; ok && k < 3; k++) {
        PyObject* t = PyObject_GetAttr(s, names[k]);
        ok = t && address(t, out + 3 * i + k);
        Py_XDECREF(t);
      }
    }
  }
  if (!ok && !PyErr_Occurred()) PyErr_SetString(PyExc_AssertionError, "device tensor expected");
  Py_DECREF(seq);
  return ok ? 0 : -1;
}
