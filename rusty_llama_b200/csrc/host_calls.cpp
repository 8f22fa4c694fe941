// The host's side of a launch, as a Python extension module: calling a launcher of the kernel libraries with tensors and numbers as they
// are, the checks that every launch makes of its tensors, and the two tensor operations that it needs (an empty tensor, a range of columns).
//
// Through ctypes a launch of 15 arguments makes 15 objects and reads every tensor through Python attributes: `add_rmsnorm` with the tensor of
// its result took 10.9 us, now 6.2, and a latent attention's sublayer over 568 tokens (nine kernels, 58 us of work) 165 us a pass, now 92.
// What is here is kernels/host.py's Python classes once more, with the same results and messages; where it cannot be built, those are used.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>

#if !(defined(__x86_64__) || defined(__aarch64__)) || defined(__APPLE__) || defined(_WIN32)
#error "calls are made by the System V (x86-64) or AAPCS64 rules"
#endif

static PyObject* kernel_error = nullptr;  // errors.KernelError

static PyObject* refuse(PyObject* what, const char* rest) { return PyErr_Format(kernel_error, "%S: %s", what, rest); }

// A C++ exception (a tensor without storage, no memory, a range that is not there) as the Python one that PyTorch makes of it
#define HC_TRY try {
#define HC_CATCH                                                      \
  }                                                                   \
  catch (...) {                                                       \
    torch::translate_exception_to_python(std::current_exception());   \
    return nullptr;                                                   \
  }

struct Unlocked {  // without the interpreter's lock, which an exception takes again on its way out
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

// ---------------------------------------------------------------- launchers
// An exported launcher takes pointers, int, long long, unsigned, float and the stream, and returns int (or long long).  Both calling
// conventions hand integers (and pointers) over in one row of registers and then 8-byte stack places, floats in another row of eight
// registers, each in the order of its own kind; so all integers first and all floats behind them reach the callee as it declared them,
// however the two are mixed in its list, as long as there are no more than eight floats.  Places that the callee does not declare are not read.
#define HC_INTS 56
#define HC_FLOATS 8
typedef long long L;
typedef L (*Fn)(L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L,
                L, L, L, L, L, L, L, float, float, float, float, float, float, float, float);

struct Launcher {
  PyObject_HEAD
  vectorcallfunc call;
  Fn fn;
  int wide;  // returns long long
  int n;     // arguments, or -1: nobody said, and each goes by its own type
  char kinds[HC_INTS + HC_FLOATS];  // of each: 'p' a pointer, 'i' a whole number, 'f' a float
};

static PyObject* too_many() { return PyErr_Format(PyExc_TypeError, "a launcher takes %d floats and %d integers and tensors at most", HC_FLOATS, HC_INTS); }

static PyObject* launcher_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  const Launcher* l = reinterpret_cast<Launcher*>(self);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (kwnames && PyTuple_GET_SIZE(kwnames)) return PyErr_Format(PyExc_TypeError, "a launcher takes no keywords");
  if (l->n >= 0 && n != l->n) return PyErr_Format(PyExc_TypeError, "this launcher takes %d arguments, not %zd", l->n, n);
  L i[HC_INTS] = {};
  float f[HC_FLOATS] = {};
  int ni = 0, nf = 0;
  HC_TRY
  for (Py_ssize_t k = 0; k < n; ++k) {
    PyObject* a = args[k];
    const char kind = l->n >= 0 ? l->kinds[k] : PyFloat_Check(a) ? 'f' : a == Py_None || THPVariable_Check(a) ? 'p' : 'i';
    if (kind == 'f') {
      if (nf == HC_FLOATS) return too_many();
      const double x = PyFloat_CheckExact(a) ? PyFloat_AS_DOUBLE(a) : PyFloat_AsDouble(a);
      if (x == -1.0 && PyErr_Occurred()) return nullptr;
      f[nf++] = (float)x;
      continue;
    }
    if (ni == HC_INTS) return too_many();
    if (PyLong_Check(a)) {  // (a pointer's, too: an address)
      i[ni] = (L)PyLong_AsUnsignedLongLongMask(a);
      if (i[ni] == -1 && PyErr_Occurred()) return nullptr;
      ++ni;
    } else if (kind == 'p') {
      if (THPVariable_Check(a)) i[ni++] = (L)(uintptr_t)THPVariable_Unpack(a).data_ptr();
      else if (a == Py_None) i[ni++] = 0;
      else return PyErr_Format(PyExc_TypeError, "argument %zd of a launcher is a tensor, an address or None, not %s", k + 1, Py_TYPE(a)->tp_name);
    } else {
      PyObject* whole = PyNumber_Index(a);  // (refuses floats and None)
      if (!whole) return nullptr;
      i[ni++] = (L)PyLong_AsUnsignedLongLongMask(whole);
      Py_DECREF(whole);
    }
  }
  L r;
  {
    Unlocked here;
    r = l->fn(i[0], i[1], i[2], i[3], i[4], i[5], i[6], i[7], i[8], i[9], i[10], i[11], i[12], i[13], i[14], i[15], i[16], i[17], i[18], i[19], i[20], i[21],
              i[22], i[23], i[24], i[25], i[26], i[27], i[28], i[29], i[30], i[31], i[32], i[33], i[34], i[35], i[36], i[37], i[38], i[39], i[40], i[41], i[42],
              i[43], i[44], i[45], i[46], i[47], i[48], i[49], i[50], i[51], i[52], i[53], i[54], i[55], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]);
  }
  return PyLong_FromLongLong(l->wide ? r : (L)(int)r);
  HC_CATCH
}

static PyTypeObject launcher_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// launcher(address, returns long long, kinds=None) -> callable.  Kinds are what every call's arguments are checked against, in number and in
// kind: without the check an argument of another kind moves all behind it to other places of their rows.
static PyObject* make_launcher(PyObject*, PyObject* args) {
  unsigned long long address;
  int wide;
  const char* kinds = nullptr;
  if (!PyArg_ParseTuple(args, "Kp|z", &address, &wide, &kinds)) return nullptr;
  int floats = 0, n = 0;
  for (; kinds && kinds[n]; ++n) {
    if (kinds[n] == 'f') ++floats;
    else if (kinds[n] != 'p' && kinds[n] != 'i') return PyErr_Format(PyExc_ValueError, "unknown kind of argument in '%s'", kinds);
  }
  if (floats > HC_FLOATS || n - floats > HC_INTS) return too_many();
  Launcher* l = PyObject_New(Launcher, &launcher_type);
  if (!l) return nullptr;
  l->call = launcher_call;
  l->fn = reinterpret_cast<Fn>((uintptr_t)address);
  l->wide = wide;
  l->n = kinds ? n : -1;
  for (int k = 0; k < n; ++k) l->kinds[k] = kinds[k];
  return reinterpret_cast<PyObject*>(l);
}

// ---------------------------------------------------------------- checks
// cuda(t, what, dtype=None, contiguous=True) -> t
static PyObject* check_cuda(PyObject*, PyObject* const* args, Py_ssize_t n, PyObject* kwnames) {
  PyObject *t = n > 0 ? args[0] : nullptr, *what = n > 1 ? args[1] : nullptr, *dtype = n > 2 ? args[2] : Py_None;
  int contiguous = n > 3 ? PyObject_IsTrue(args[3]) : 1;
  for (Py_ssize_t k = 0; kwnames && k < PyTuple_GET_SIZE(kwnames); ++k) {
    PyObject* name = PyTuple_GET_ITEM(kwnames, k);
    if (PyUnicode_CompareWithASCIIString(name, "contiguous") == 0) contiguous = PyObject_IsTrue(args[n + k]);
    else if (PyUnicode_CompareWithASCIIString(name, "dtype") == 0) dtype = args[n + k];
    else return PyErr_Format(PyExc_TypeError, "cuda: unexpected keyword '%S'", name);
  }
  if (!what || contiguous < 0) return PyErr_Format(PyExc_TypeError, "cuda(t, what, dtype=None, contiguous=True)");
  HC_TRY
  if (!THPVariable_Check(t)) return refuse(what, "not a tensor");
  const at::Tensor& x = THPVariable_Unpack(t);
  if (!x.is_cuda()) {
    PyObject* device = PyObject_GetAttrString(t, "device");
    if (!device) return nullptr;
    PyErr_Format(kernel_error, "%S: tensor is on %S, the kernels run on CUDA only", what, device);
    Py_DECREF(device);
    return nullptr;
  }
  if (dtype != Py_None) {
    if (!THPDtype_Check(dtype)) return PyErr_Format(PyExc_TypeError, "cuda: dtype is not a torch.dtype");
    if (x.scalar_type() != reinterpret_cast<THPDtype*>(dtype)->scalar_type) {
      PyObject* mine = PyObject_GetAttrString(t, "dtype");
      if (!mine) return nullptr;
      PyErr_Format(kernel_error, "%S: dtype %S, expected %S", what, mine, dtype);
      Py_DECREF(mine);
      return nullptr;
    }
  }
  if (contiguous && !x.is_contiguous()) return refuse(what, "tensor is not contiguous");
  Py_INCREF(t);
  return t;
  HC_CATCH
}

// rows(t, what) -> row stride of a 2-D tensor whose rows are dense
static PyObject* check_rows(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2 || !THPVariable_Check(args[0])) return PyErr_Format(PyExc_TypeError, "rows(tensor, what)");
  HC_TRY
  const at::Tensor& x = THPVariable_Unpack(args[0]);
  if (x.dim() != 2 || x.stride(1) != 1) return refuse(args[1], "expected a 2-D tensor with dense rows");
  return PyLong_FromLongLong(x.stride(0));
  HC_CATCH
}

// matrices(t, other, like, what) -> (matrices, rows, columns, row stride, matrix stride) of a 3-D tensor of like's type and device whose rows are
// dense; other: None or a tensor that has to lie in the same way
static PyObject* check_matrices(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4 || !THPVariable_Check(args[0]) || !(args[1] == Py_None || THPVariable_Check(args[1])) || !THPVariable_Check(args[2]))
    return PyErr_Format(PyExc_TypeError, "matrices(tensor, tensor or None, tensor, what)");
  HC_TRY
  const at::Tensor &x = THPVariable_Unpack(args[0]), &like = THPVariable_Unpack(args[2]);
  if (x.dim() != 3 || x.stride(2) != 1 || x.scalar_type() != like.scalar_type() || x.device() != like.device())
    return refuse(args[3], "expected a 3-D tensor with dense rows beside the others");
  if (args[1] != Py_None) {
    const at::Tensor& y = THPVariable_Unpack(args[1]);
    if (y.sizes() != x.sizes() || y.strides() != x.strides() || y.scalar_type() != x.scalar_type() || y.device() != x.device()) return refuse(args[3], "two tensors that do not lie in the same way");
  }
  return Py_BuildValue("(LLLLL)", (L)x.size(0), (L)x.size(1), (L)x.size(2), (L)x.stride(1), (L)x.stride(0));
  HC_CATCH
}

// odd(x, w) -> whether rows of the two cannot be moved in 16-byte pieces: eight 16-bit numbers
static PyObject* check_odd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) return PyErr_Format(PyExc_TypeError, "odd(x, w)");
  HC_TRY
  const at::Tensor &x = THPVariable_Unpack(args[0]), &w = THPVariable_Unpack(args[1]);
  if (x.dim() != 2 || w.dim() < 1) return PyErr_Format(PyExc_IndexError, "odd: rows expected");
  return PyBool_FromLong(x.size(1) % 8 || x.stride(0) % 8 || w.stride(0) % 8 || (((uintptr_t)x.data_ptr() | (uintptr_t)w.data_ptr()) & 15));
  HC_CATCH
}

// stream() -> the current stream of the current device
static PyObject* current_stream(PyObject*, PyObject*) {
  HC_TRY
  return PyLong_FromUnsignedLongLong((uintptr_t)c10::cuda::getCurrentCUDAStream().stream());
  HC_CATCH
}

// empty(like, dtype, sizes...) -> an empty tensor on like's device
static PyObject* make_empty(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n < 3 || n > 6 || !THPVariable_Check(args[0]) || !THPDtype_Check(args[1])) return PyErr_Format(PyExc_TypeError, "empty(like, dtype, one to four sizes)");
  HC_TRY
  int64_t sizes[4];
  for (Py_ssize_t k = 2; k < n; ++k) {
    sizes[k - 2] = PyLong_AsLongLong(args[k]);
    if (sizes[k - 2] == -1 && PyErr_Occurred()) return nullptr;
  }
  const at::Device device = THPVariable_Unpack(args[0]).device();
  const at::ScalarType type = reinterpret_cast<THPDtype*>(args[1])->scalar_type;
  at::Tensor out;
  {
    Unlocked here;
    out = at::empty(at::IntArrayRef(sizes, n - 2), at::TensorOptions().dtype(type).device(device));
  }
  return THPVariable_Wrap(out);
  HC_CATCH
}

// columns(t, first, end) -> t[:, first:end]
static PyObject* take_columns(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3 || !THPVariable_Check(args[0])) return PyErr_Format(PyExc_TypeError, "columns(tensor, first, end)");
  HC_TRY
  const L first = PyLong_AsLongLong(args[1]), end = PyLong_AsLongLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  return THPVariable_Wrap(THPVariable_Unpack(args[0]).narrow(1, first, end - first));
  HC_CATCH
}

static PyObject* set_error(PyObject*, PyObject* kind) {
  Py_XDECREF(kernel_error);
  Py_INCREF(kind);
  kernel_error = kind;
  Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"launcher", make_launcher, METH_VARARGS, nullptr},
    {"cuda", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(check_cuda)), METH_FASTCALL | METH_KEYWORDS, nullptr},
    {"rows", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(check_rows)), METH_FASTCALL, nullptr},
    {"matrices", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(check_matrices)), METH_FASTCALL, nullptr},
    {"odd", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(check_odd)), METH_FASTCALL, nullptr},
    {"stream", current_stream, METH_NOARGS, nullptr},
    {"empty", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(make_empty)), METH_FASTCALL, nullptr},
    {"columns", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(take_columns)), METH_FASTCALL, nullptr},
    {"set_error", set_error, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

static PyModuleDef module = {PyModuleDef_HEAD_INIT, "_rl_host_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

PyMODINIT_FUNC PyInit__rl_host_calls() {
  launcher_type.tp_name = "_rl_host_calls.Launcher";
  launcher_type.tp_basicsize = sizeof(Launcher);
  launcher_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  launcher_type.tp_vectorcall_offset = offsetof(Launcher, call);
  launcher_type.tp_call = PyVectorcall_Call;
  if (PyType_Ready(&launcher_type) < 0) return nullptr;
  kernel_error = PyExc_RuntimeError;
  Py_INCREF(kernel_error);
  return PyModule_Create(&module);
}
