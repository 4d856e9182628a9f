/* Python call path of the step launchers: a small extension module that parses
 * the arguments of the hot entry points and calls the C ABI directly.
 *
 * A step of a small box takes the GPU about 2 us, less than ctypes needs to
 * convert ten arguments, so the host loop sets the pace there: 50 steps of D2Q9 FP64 128^2 took 234 us through ctypes and take
 * 131 us through this module.
 * Each function takes the arguments of the lbcube.py function of its name,
 * in order, and returns the launcher's status; it returns None, having
 * launched nothing, when an argument is not of the plain type it handles
 * (names as str, extents as int, rates as float, buffers as None, int
 * or an object with data_ptr(), stream as None, int or an object with
 * cuda_stream), and lbcube.py then takes its ctypes path, which accepts and
 * refuses what it always did. The launchers' addresses are handed over once by
 * setup(); the module itself links against nothing.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stddef.h>
#include <stdint.h>
#include <string.h>

typedef int (*step_fn)(int, int, int, const void*, void*, size_t, size_t, size_t, double, void*);
typedef int (*step16_fn)(int, int, int, const void*, void*, size_t, size_t, size_t, float, float, void*);
typedef int (*scalar_fn)(int, int, const void*, void*, const void*, size_t, size_t, size_t, double, double, void*);
typedef int (*reaction_fn)(int, int, const void*, void*, const void*, void*, const void*, size_t, size_t, size_t,
                           double, double, void*);
typedef int (*coupled_fn)(int, int, int, const void*, void*, const void*, void*, const void*, void*, size_t, size_t,
                          size_t, double, double, double, double*, size_t, void*);

static step_fn g_step;
static step16_fn g_step16;
static scalar_fn g_scalar;
static reaction_fn g_reaction;
static coupled_fn g_coupled;
static PyObject *s_data_ptr, *s_cuda_stream;

/* The outcome of one argument: parsed, not a plain type, or a Python error. */
enum { OK = 0, OTHER = 1, FAILED = -1 };

struct name {
  const char* text;
  int code;
};
static const struct name kLattices[] = {{"D2Q9", 0}, {"D3Q19", 1}, {"D3Q27", 2}, {NULL, 0}};
static const struct name kReals[] = {{"float", 0}, {"double", 1}, {NULL, 0}};
static const struct name kOps[] = {{"BGK", 0}, {"TRT", 1}, {"MRT", 2}, {"RLBM", 3}, {NULL, 0}};
static const struct name kFormats[] = {{"f16s", 2}, {"bf16s", 3}, {"e3m12s", 4}, {"q15s", 5}, {NULL, 0}};

static int parse_name(PyObject* o, const struct name* names, int* out) {
  if (!PyUnicode_CheckExact(o)) return OTHER;
  for (; names->text != NULL; ++names)
    if (PyUnicode_CompareWithASCIIString(o, names->text) == 0) {
      *out = names->code;
      return OK;
    }
  return OTHER;
}

/* real_name() of lbcube.py: "float" and "double", or anything whose text holds
 * float32 or float64 (a torch or numpy dtype). */
static int parse_real(PyObject* o, int* out) {
  if (PyUnicode_CheckExact(o)) return parse_name(o, kReals, out);
  PyObject* text = PyObject_Str(o);
  if (text == NULL) return FAILED;
  const char* s = PyUnicode_AsUTF8(text);
  const int real = s == NULL ? -1 : strstr(s, "float32") != NULL ? 0 : strstr(s, "float64") != NULL ? 1 : -1;
  Py_DECREF(text);
  if (s == NULL) return FAILED;
  *out = real;
  return real < 0 ? OTHER : OK;
}

static int parse_size(PyObject* o, size_t* out) {
  if (!PyLong_CheckExact(o)) return OTHER;
  const unsigned long long v = PyLong_AsUnsignedLongLong(o);
  if (v == (unsigned long long)-1 && PyErr_Occurred()) {
    PyErr_Clear();
    return OTHER;
  }
  *out = (size_t)v;
  return OK;
}

static int parse_rate(PyObject* o, double* out) {
  if (PyFloat_CheckExact(o)) {
    *out = PyFloat_AS_DOUBLE(o);
    return OK;
  }
  return OTHER;
}

static int parse_address(PyObject* o, PyObject* attribute, int call, void** out) {
  if (o == Py_None) {
    *out = NULL;
    return OK;
  }
  PyObject* v = NULL;
  if (!PyLong_CheckExact(o)) {
    if (PyLong_Check(o)) return OTHER; /* an int of a class of its own: lbcube.py takes its value */
    v = call ? PyObject_CallMethodNoArgs(o, attribute) : PyObject_GetAttr(o, attribute);
    if (v == NULL) return FAILED;
    o = v;
  }
  size_t a = 0;
  const int r = parse_size(o, &a);
  Py_XDECREF(v);
  *out = (void*)(uintptr_t)a;
  return r;
}

static int parse_buffer(PyObject* o, void** out) { return parse_address(o, s_data_ptr, 1, out); }
static int parse_stream(PyObject* o, void** out) { return parse_address(o, s_cuda_stream, 0, out); }

/* Evaluates a parser; leaves the function unless the argument was parsed. */
#define TRY(expr)                    \
  do {                               \
    const int r_ = (expr);           \
    if (r_ == FAILED) return NULL;   \
    if (r_ == OTHER) Py_RETURN_NONE; \
  } while (0)

#define NEED(n)                                                              \
  if (count != (n)) {                                                        \
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", n, count); \
    return NULL;                                                             \
  }

#define CALL(expr)              \
  do {                          \
    int rc_;                    \
    Py_BEGIN_ALLOW_THREADS;     \
    rc_ = (expr);               \
    Py_END_ALLOW_THREADS;       \
    return PyLong_FromLong(rc_); \
  } while (0)

/* step_async(lattice, real, collision, cur, nxt, nx, ny, nz, omega, stream) */
static PyObject* py_step(PyObject* self, PyObject* const* a, Py_ssize_t count) {
  int lat, real, op;
  void *cur, *nxt, *s;
  size_t n[3];
  double omega;
  NEED(10);
  TRY(parse_name(a[0], kLattices, &lat));
  TRY(parse_real(a[1], &real));
  TRY(parse_name(a[2], kOps, &op));
  for (int i = 0; i < 3; ++i) TRY(parse_size(a[5 + i], &n[i]));
  TRY(parse_rate(a[8], &omega));
  TRY(parse_buffer(a[3], &cur));
  TRY(parse_buffer(a[4], &nxt));
  TRY(parse_stream(a[9], &s));
  CALL(g_step(lat, real, op, cur, nxt, n[0], n[1], n[2], omega, s));
}

/* step_shifted_async(lattice, fmt, collision, cur, nxt, nx, ny, nz, omega, rho0, stream) */
static PyObject* py_step16(PyObject* self, PyObject* const* a, Py_ssize_t count) {
  int lat, fmt, op;
  void *cur, *nxt, *s;
  size_t n[3];
  double omega, rho0;
  NEED(11);
  TRY(parse_name(a[0], kLattices, &lat));
  TRY(parse_name(a[1], kFormats, &fmt));
  TRY(parse_name(a[2], kOps, &op));
  for (int i = 0; i < 3; ++i) TRY(parse_size(a[5 + i], &n[i]));
  TRY(parse_rate(a[8], &omega));
  TRY(parse_rate(a[9], &rho0));
  TRY(parse_buffer(a[3], &cur));
  TRY(parse_buffer(a[4], &nxt));
  TRY(parse_stream(a[10], &s));
  CALL(g_step16(lat, fmt, op, cur, nxt, n[0], n[1], n[2], (float)omega, (float)rho0, s));
}

/* scalar_step_async(lattice, real, cur_s, nxt_s, cur_f, nx, ny, nz, omega_c, source, stream) */
static PyObject* py_scalar(PyObject* self, PyObject* const* a, Py_ssize_t count) {
  int lat, real;
  void *cur, *nxt, *f, *s;
  size_t n[3];
  double omega_c, source;
  NEED(11);
  TRY(parse_name(a[0], kLattices, &lat));
  TRY(parse_real(a[1], &real));
  for (int i = 0; i < 3; ++i) TRY(parse_size(a[5 + i], &n[i]));
  TRY(parse_rate(a[8], &omega_c));
  TRY(parse_rate(a[9], &source));
  TRY(parse_buffer(a[2], &cur));
  TRY(parse_buffer(a[3], &nxt));
  TRY(parse_buffer(a[4], &f));
  TRY(parse_stream(a[10], &s));
  CALL(g_scalar(lat, real, cur, nxt, f, n[0], n[1], n[2], omega_c, source, s));
}

/* reaction_ab_async(lattice, real, cur_a, nxt_a, cur_b, nxt_b, cur_f, nx, ny, nz, omega_c, k, stream) */
static PyObject* py_reaction(PyObject* self, PyObject* const* a, Py_ssize_t count) {
  int lat, real;
  void *p[5], *s;
  size_t n[3];
  double omega_c, k;
  NEED(13);
  TRY(parse_name(a[0], kLattices, &lat));
  TRY(parse_real(a[1], &real));
  for (int i = 0; i < 3; ++i) TRY(parse_size(a[7 + i], &n[i]));
  TRY(parse_rate(a[10], &omega_c));
  TRY(parse_rate(a[11], &k));
  for (int i = 0; i < 5; ++i) TRY(parse_buffer(a[2 + i], &p[i]));
  TRY(parse_stream(a[12], &s));
  CALL(g_reaction(lat, real, p[0], p[1], p[2], p[3], p[4], n[0], n[1], n[2], omega_c, k, s));
}

/* fluid_reaction_ab_async(lattice, real, collision, cur_f, nxt_f, cur_a, nxt_a, cur_b, nxt_b, nx, ny, nz,
 *                         omega, omega_c, k, partials, partials_bytes, stream) */
static PyObject* py_coupled(PyObject* self, PyObject* const* a, Py_ssize_t count) {
  int lat, real, op;
  void *p[6], *partials, *s;
  size_t n[3], bytes;
  double omega, omega_c, k;
  NEED(18);
  TRY(parse_name(a[0], kLattices, &lat));
  TRY(parse_real(a[1], &real));
  TRY(parse_name(a[2], kOps, &op));
  for (int i = 0; i < 3; ++i) TRY(parse_size(a[9 + i], &n[i]));
  TRY(parse_rate(a[12], &omega));
  TRY(parse_rate(a[13], &omega_c));
  TRY(parse_rate(a[14], &k));
  TRY(parse_size(a[16], &bytes));
  for (int i = 0; i < 6; ++i) TRY(parse_buffer(a[3 + i], &p[i]));
  TRY(parse_buffer(a[15], &partials));
  TRY(parse_stream(a[17], &s));
  CALL(g_coupled(lat, real, op, p[0], p[1], p[2], p[3], p[4], p[5], n[0], n[1], n[2], omega, omega_c, k,
                 (double*)partials, bytes, s));
}

/* setup(step, step_shifted, scalar_step, reaction_ab, fluid_reaction_ab): the launchers' addresses */
static PyObject* py_setup(PyObject* self, PyObject* const* a, Py_ssize_t count) {
  size_t p[5];
  NEED(5);
  for (int i = 0; i < 5; ++i)
    if (parse_size(a[i], &p[i]) != OK || p[i] == 0) {
      PyErr_SetString(PyExc_ValueError, "setup() takes five function addresses");
      return NULL;
    }
  g_step = (step_fn)(uintptr_t)p[0];
  g_step16 = (step16_fn)(uintptr_t)p[1];
  g_scalar = (scalar_fn)(uintptr_t)p[2];
  g_reaction = (reaction_fn)(uintptr_t)p[3];
  g_coupled = (coupled_fn)(uintptr_t)p[4];
  Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"setup", (PyCFunction)(void (*)(void))py_setup, METH_FASTCALL, NULL},
    {"step", (PyCFunction)(void (*)(void))py_step, METH_FASTCALL, NULL},
    {"step_shifted", (PyCFunction)(void (*)(void))py_step16, METH_FASTCALL, NULL},
    {"scalar_step", (PyCFunction)(void (*)(void))py_scalar, METH_FASTCALL, NULL},
    {"reaction_ab", (PyCFunction)(void (*)(void))py_reaction, METH_FASTCALL, NULL},
    {"fluid_reaction_ab", (PyCFunction)(void (*)(void))py_coupled, METH_FASTCALL, NULL},
    {NULL, NULL, 0, NULL}};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_lbcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__lbcall(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_cuda_stream = PyUnicode_InternFromString("cuda_stream");
  if (s_data_ptr == NULL || s_cuda_stream == NULL) return NULL;
  return PyModule_Create(&module);
}
