// Device addresses of a list of expert slots, read from the tensors themselves.  A prefill call names over a thousand matrices and
// the GPU waits for it: data_ptr() through the interpreter takes 85 us for 384 experts, this 10.
#include <torch/csrc/autograd/python_variable.h>
#include <cstdint>

// slots: sequence of ExpertSlot, each with a tuple _m of three tensors or None; out: [n][3], 0 for None.  Returns 0, or -1 with a
// Python exception set (called with the interpreter lock held).
extern "C" int msb_slot_addresses(PyObject* slots, uint64_t* out) {
  static PyObject* name = PyUnicode_InternFromString("_m");
  PyObject* seq = PySequence_Fast(slots, "expert slots: a sequence expected");
  if (!seq) return -1;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
  for (Py_ssize_t i = 0; i < n; i++) {
    PyObject* m = PyObject_GetAttr(PySequence_Fast_GET_ITEM(seq, i), name);
    bool ok = m && PyTuple_Check(m) && PyTuple_GET_SIZE(m) == 3;
    for (int k = 0; ok && k < 3; k++) {
      PyObject* t = PyTuple_GET_ITEM(m, k);
      if (t == Py_None) { out[3 * i + k] = 0; continue; }
      ok = THPVariable_Check(t) && THPVariable_Unpack(t).is_cuda();
      if (ok) out[3 * i + k] = reinterpret_cast<uint64_t>(THPVariable_Unpack(t).data_ptr());
    }
    Py_XDECREF(m);
    if (!ok) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_AssertionError, "device tensor expected");
      Py_DECREF(seq);
      return -1;
    }
  }
  Py_DECREF(seq);
  return 0;
}
