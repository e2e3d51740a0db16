// Calls of the exported launchers from Python without ctypes, whose conversion of 15 to 45 arguments takes 2 to 5 us a call, as
// much as the launch itself (27 arguments: 3.2 us, here 0.23).  Host code only.
//
// q3_make_caller(function, kinds) returns a Python function that takes one argument per letter of kinds -- i: a whole number
// or what stands for one (__index__), p: an address or None, f: a number that is passed as float -- and returns the launcher's int.
//
// All launchers are called through one type.  The calling convention of x86-64 Linux hands whole numbers and addresses over in six
// registers and then in 8-byte places on the stack, in their order, and up to eight floats in registers of their own, so a
// function finds its arguments whatever stands behind the last of them, and wherever the floats stand between the others.
// Elsewhere, and without Python's headers, there is no q3_make_caller and ctypes does it.
#if defined(__x86_64__) && defined(__linux__) && __has_include(<Python.h>)
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <string.h>

namespace {

constexpr int MOST_WHOLE = 48, MOST_FLOATS = 8;
typedef int (*Launcher)(long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long,
                        long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long,
                        long, long, long, long, long, long, long, long, long, long, long, long, float, float, float, float, float,
                        float, float, float);

struct Callee {
  Launcher function;
  int arguments;
  char kinds[MOST_WHOLE + MOST_FLOATS];
};

PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  const Callee* c = reinterpret_cast<const Callee*>(PyBytes_AS_STRING(self));
  if (n != c->arguments) {
    PyErr_Format(PyExc_TypeError, "%d arguments expected, %zd given", c->arguments, n);
    return nullptr;
  }
  long v[MOST_WHOLE] = {};
  float f[MOST_FLOATS] = {};
  int whole = 0, floats = 0;
  for (int i = 0; i < c->arguments; ++i) {
    PyObject* a = args[i];
    if (c->kinds[i] == 'f') {
      const double x = PyFloat_AsDouble(a);
      if (x == -1.0 && PyErr_Occurred()) return nullptr;
      f[floats++] = (float)x;
    } else {
      long x = 0;
      if (PyLong_Check(a)) {
        x = PyLong_AsLong(a);
        if (x == -1 && PyErr_Occurred()) return nullptr;
      } else if (c->kinds[i] == 'i' && PyIndex_Check(a)) {  // numpy's and torch's whole numbers, as ctypes takes them
        PyObject* whole_number = PyNumber_Index(a);
        if (!whole_number) return nullptr;
        x = PyLong_AsLong(whole_number);
        Py_DECREF(whole_number);
        if (x == -1 && PyErr_Occurred()) return nullptr;
      } else if (c->kinds[i] == 'i' || a != Py_None) {
        PyErr_Format(PyExc_TypeError, "argument %d: %s expected, not %s", i + 1,
                     c->kinds[i] == 'p' ? "an address or None" : "an int", Py_TYPE(a)->tp_name);
        return nullptr;
      }
      v[whole++] = x;
    }
  }
  int code;
  Py_BEGIN_ALLOW_THREADS
  code = c->function(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[12], v[13], v[14], v[15], v[16],
                     v[17], v[18], v[19], v[20], v[21], v[22], v[23], v[24], v[25], v[26], v[27], v[28], v[29], v[30], v[31], v[32],
                     v[33], v[34], v[35], v[36], v[37], v[38], v[39], v[40], v[41], v[42], v[43], v[44], v[45], v[46], v[47], f[0],
                     f[1], f[2], f[3], f[4], f[5], f[6], f[7]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(code);
}

PyMethodDef method = {"launcher", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call)), METH_FASTCALL,
                      "one argument per letter; the launcher's status"};

}  // namespace

// (called with the interpreter's lock held)
extern "C" __attribute__((visibility("default"))) PyObject* q3_make_caller(void* function, const char* kinds) {
  Callee c = {};
  c.function = reinterpret_cast<Launcher>(function);
  int floats = 0;
  for (const char* k = kinds; *k; ++k) {
    if ((*k != 'i' && *k != 'p' && *k != 'f') || c.arguments == MOST_WHOLE + MOST_FLOATS) Py_RETURN_NONE;
    floats += *k == 'f';
    c.kinds[c.arguments++] = *k;
  }
  if (floats > MOST_FLOATS || c.arguments - floats > MOST_WHOLE) Py_RETURN_NONE;
  PyObject* self = PyBytes_FromStringAndSize(reinterpret_cast<const char*>(&c), sizeof c);
  if (!self) return nullptr;
  PyObject* made = PyCFunction_NewEx(&method, self, nullptr);
  Py_DECREF(self);
  return made;
}
#else
extern "C" __attribute__((visibility("default"))) int q3_no_caller = 1;
#endif
