// Host side of a call on CUDA tensors, natively: the tensor checks, the current
// torch stream and the C ABI call, which in Python (attribute lookups, tuples of
// sizes, ctypes conversions) took 3 of the 6.3 us that a small call cost.
//
//   exec(kind, handle, in, out, n_in, n_out) -> status, or None
//   vmmul(v, m, out) -> status, or None
//
// None means that the tensors are not plain matrices (or do not match the
// plan): the caller then takes the general path, which converts what it can and
// reports what it cannot.  Nothing is kept between calls.
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

using ExecFn = int (*)(void *, const void *, long long, void *, long long, long long, int);
using StreamFn = int (*)(void *, void *);
using VmmulFn = int (*)(const void *, const void *, long long, void *, long long, long long, long long, void *);

// complex rows, real rows to half spectra and back, complex columns
enum Kind { kRows = 0, kR2C = 1, kC2R = 2, kCols = 3, kKinds = 4 };
constexpr int kDevice = 1;  // FCB_DEVICE

ExecFn g_exec[kKinds] = {};
StreamFn g_set_stream = nullptr;
VmmulFn g_vmmul = nullptr;

struct Matrix
{
  void *p = nullptr;
  long long rows = 0, cols = 0, rs = 0;
};

// A CUDA tensor of its own storage whose memory holds its values (no lazy conjugate or
// negation).
bool held(PyObject *o, bool real)
{
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor &t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && t.has_storage() &&
         t.scalar_type() == (real ? at::kFloat : at::kComplexFloat) && !t.is_conj() && !t.is_neg();
}

// A matrix with unit-stride rows that do not overlap, or a vector: one row.
bool plain(PyObject *o, bool real, Matrix &m)
{
  if (!held(o, real)) return false;
  const at::Tensor &t = THPVariable_Unpack(o);
  const int64_t d = t.dim();
  if (d < 1 || d > 2) return false;
  m.rows = d == 2 ? t.size(0) : 1;
  m.cols = t.size(d - 1);
  if (m.rows < 1 || m.cols < 1 || t.stride(d - 1) != 1) return false;
  m.rs = m.rows > 1 ? t.stride(0) : m.cols;
  if (m.rs < m.cols) return false;
  m.p = t.data_ptr();
  return true;
}

// What a column transform's transposing form refuses: a vector, an output that torch
// must not write behind autograd's back.
bool column_form(PyObject *in, PyObject *out)
{
  const at::Tensor &t = THPVariable_Unpack(out);
  return THPVariable_Unpack(in).dim() == 2 && t.dim() == 2 && !t.requires_grad();
}

bool same_or_apart(const Matrix &a, const Matrix &b)
{
  if (a.p == b.p) return a.rs == b.rs;
  const char *x = static_cast<const char *>(a.p), *y = static_cast<const char *>(b.p);
  return x + 8 * ((a.rows - 1) * a.rs + a.cols) <= y || y + 8 * ((b.rows - 1) * b.rs + b.cols) <= x;
}

PyObject *exec(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
  if (nargs != 6) return PyErr_Format(PyExc_TypeError, "exec takes six arguments");
  const long kind = PyLong_AsLong(args[0]);
  void *plan = PyLong_AsVoidPtr(args[1]);
  const long long n_in = PyLong_AsLongLong(args[4]), n_out = PyLong_AsLongLong(args[5]);
  if (PyErr_Occurred()) return nullptr;
  if (kind < 0 || kind >= kKinds || !g_exec[kind] || !plan) Py_RETURN_NONE;
  Matrix in, out;
  void *stream = nullptr;
  try
  {
    if (!plain(args[2], kind == kR2C, in) || !plain(args[3], kind == kC2R, out)) Py_RETURN_NONE;
    if (in.rows != out.rows) Py_RETURN_NONE;
    if (kind == kCols)
    {
      if (!column_form(args[2], args[3])) Py_RETURN_NONE;
      // a column plan: n_in the length, n_out the most columns
      if (in.rows != n_in || in.cols > n_out || in.cols != out.cols || !same_or_apart(in, out)) Py_RETURN_NONE;
    }
    else if (in.cols != n_in || out.cols != n_out)
      Py_RETURN_NONE;
    stream = c10::cuda::getCurrentCUDAStream().stream();
  }
  catch (...)
  {
    Py_RETURN_NONE;  // the general path meets the same error and reports it
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_set_stream(plan, stream);
  if (!rc) rc = g_exec[kind](plan, in.p, in.rs, out.p, out.rs, kind == kCols ? in.cols : in.rows, kDevice);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// out[r][c] = v[c] m[r][c]
PyObject *vmmul(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
  if (nargs != 3) return PyErr_Format(PyExc_TypeError, "vmmul takes three arguments");
  Matrix m, out;
  const void *v = nullptr;
  void *stream = nullptr;
  try
  {
    if (!g_vmmul || !held(args[0], false) || !plain(args[1], false, m) || !plain(args[2], false, out)) Py_RETURN_NONE;
    const at::Tensor &t = THPVariable_Unpack(args[0]);
    if (!t.is_contiguous() || t.numel() != m.cols || out.rows != m.rows || out.cols != m.cols) Py_RETURN_NONE;
    v = t.data_ptr();
    stream = c10::cuda::getCurrentCUDAStream().stream();
  }
  catch (...)
  {
    Py_RETURN_NONE;
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_vmmul(v, m.p, m.rs, out.p, out.rs, m.rows, m.cols, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// bind(fcb_set_stream, fcb_exec, fcb_exec_r2c, fcb_exec_c2r, fcb_exec_cols, fcb_vmmul_rows): addresses
PyObject *bind(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
  if (nargs != 2 + kKinds) return PyErr_Format(PyExc_TypeError, "bind takes six addresses");
  g_set_stream = reinterpret_cast<StreamFn>(PyLong_AsVoidPtr(args[0]));
  for (int i = 0; i < kKinds; ++i) g_exec[i] = reinterpret_cast<ExecFn>(PyLong_AsVoidPtr(args[1 + i]));
  g_vmmul = reinterpret_cast<VmmulFn>(PyLong_AsVoidPtr(args[1 + kKinds]));
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {
    {"exec", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(exec)), METH_FASTCALL, nullptr},
    {"vmmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(vmmul)), METH_FASTCALL, nullptr},
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_fcb_torch", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// built_for: the Python and torch this was compiled against, whose object layouts it relies on
PyMODINIT_FUNC PyInit__fcb_torch(void)
{
  PyObject *m = PyModule_Create(&g_module);
  if (m && PyModule_AddStringConstant(m, "built_for", FCB_BUILT_FOR) < 0) Py_CLEAR(m);
  return m;
}
