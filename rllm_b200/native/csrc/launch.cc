// The way from Python to a kernel's entry point: an ``Entry`` is called with tensors and numbers, turns them into the
// C arguments that its signature names, adds the current stream and calls.  Built as an extension module (it takes a
// tensor's pointer from the tensor itself), so that a launch costs the host little more than the launch: through ctypes
// objects made one by one a decoded token's product cost 13 us, 3 of them cudaLaunchKernelEx.
//
// Signature letters: p a CUDA tensor or None (its address or null), i int, l long long, f float.  Every entry point
// takes its stream last and returns an int: 0, a CUDA error (> 0) or a refusal (< 0).  As with ctypes, numbers are
// narrowed without a check and the interpreter's lock is released during the call.
//
// ``product(x, w, out_f32, silu, limit, slope, shift)``: x . w^T for the plain cases of the bfloat16 kernels (see
// rllm_b200/kernels/ops.py, small_m_takes and tcgen05_takes, which hold the same rule), or None: the caller's own path.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <cstring>
#include <tuple>
#include <utility>

namespace {

PyObject* g_error = nullptr;        // the exception class of the kernels' refusals
PyObject* g_launches = nullptr;     // a list of one int: entry points called so far

template <char C> struct Arg;
template <> struct Arg<'p'> {
  typedef void* type;
  static type get(PyObject* o, bool& bad) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) {
      bad = true;
      PyErr_Format(PyExc_TypeError, "a tensor or None is wanted, not %s", Py_TYPE(o)->tp_name);
      return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda()) {
      bad = true;
      PyErr_SetString(g_error, "the engine's kernels run on CUDA tensors only; there is no CPU path");
      return nullptr;
    }
    return t.data_ptr();
  }
};
inline long long whole(PyObject* o, bool& bad) {
  const long long v = PyLong_AsLongLong(o);        // True, 3, and what has __index__
  if (v == -1 && PyErr_Occurred()) bad = true;
  return v;
}
template <> struct Arg<'i'> {
  typedef int type;
  static type get(PyObject* o, bool& bad) { return (int)whole(o, bad); }
};
template <> struct Arg<'l'> {
  typedef long long type;
  static type get(PyObject* o, bool& bad) { return whole(o, bad); }
};
template <> struct Arg<'f'> {
  typedef float type;
  static type get(PyObject* o, bool& bad) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) bad = true;
    return (float)v;
  }
};

// the current device's current stream
cudaStream_t stream_now() { return c10::cuda::getCurrentCUDAStream().stream(); }

typedef int (*Invoke)(void* fn, PyObject* const* args, bool& bad);

template <typename Ch, Ch... C> struct Signature {
  static constexpr char text[] = {C..., 0};
  template <std::size_t... I>
  static int run(void* fn, PyObject* const* a, bool& bad, std::index_sequence<I...>) {
    const std::tuple<typename Arg<C>::type...> v{(bad ? typename Arg<C>::type() : Arg<C>::get(a[I], bad))...};
    if (bad) return 0;
    const cudaStream_t stream = stream_now();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = reinterpret_cast<int (*)(typename Arg<C>::type..., cudaStream_t)>(fn)(std::get<I>(v)..., stream);
    Py_END_ALLOW_THREADS
    return rc;
  }
  static int invoke(void* fn, PyObject* const* a, bool& bad) {
    return run(fn, a, bad, std::make_index_sequence<sizeof...(C)>());
  }
};
template <typename Ch, Ch... C> constexpr Signature<Ch, C...> operator""_sig() { return {}; }

struct Row { const char* text; Invoke invoke; };
#define ROW(s) {s, decltype(s##_sig)::invoke}
const Row kSignatures[] = {
    ROW("piiiiippfpppipppfiiiiiip"), ROW("piiippipp"), ROW("piiippp"), ROW("piiippppp"), ROW("piiippppppp"),
    ROW("piiipppppppi"), ROW("piippifpppfippppiiiiiippip"), ROW("piippippppiiipiiip"),
    ROW("piippppifpippiiiiiiipiiippififiip"), ROW("piippppippiiiiiiiiifiifppiipp"), ROW("piippppippiiiiiiiiifpi"),
    ROW("piipppppipipppippiiiiiiiiipp"), ROW("piippppppppiiiiff"), ROW("piiipppppppppiiipiiiip"), ROW("pipifpipiiiiifff"),
    ROW("pipipiiii"), ROW("pipipiiiiifff"), ROW("pipipiiiiifffp"), ROW("pipipippipippiii"), ROW("pippifpppfipppppiiiiiiipp"),
    ROW("pippiiipppiiiiiiiifpp"), ROW("pippippppipppppppiiiiiiiiiiiiifffip"), ROW("pipppipippiiiiiiifp"),
    ROW("pipppipippiiiiiiiifiifppiipiip"), ROW("pipppipippiiiiiiip"), ROW("pipppippiiiiiiiiifpp"),
    ROW("pippppffpppiiiippiiiip"), ROW("pippppipiiiiiiiifiifppiipiipfpppp"), ROW("pippppipiiiiiiiifpiippp"),
    ROW("pippppippiiiiiiiiifiifppiipp"), ROW("pippppippiiiiiiiiifp"), ROW("pippppippiiiiiiiiiiiifp"), ROW("pipppppipiiiip"),
    ROW("pipppppipiiipiip"), ROW("plf"), ROW("plipppppfiiii"), ROW("pllplliplliiiii"), ROW("pllpllpiliiiip"), ROW("ppffpil"),
    ROW("ppfppiii"), ROW("ppiii"), ROW("ppiiifff"), ROW("ppiiii"), ROW("ppiip"), ROW("ppil"), ROW("ppili"), ROW("ppipiii"),
    ROW("ppipiiifip"), ROW("ppipipiiif"), ROW("ppipipiiiif"), ROW("ppippiiiif"), ROW("ppipppppppippili"), ROW("ppl"),
    ROW("pppffpffpiiii"), ROW("pppiiiiii"), ROW("pppiiippi"), ROW("pppiipppffppppiiiiiiippp"), ROW("pppiiippppppiiipiiip"),
    ROW("pppipippiiiiiiifpp"), ROW("pppippippfppfplippiiii"), ROW("ppppfiiiiiii"), ROW("ppppiii"), ROW("ppppiiiii"),
    ROW("ppppiiipppiiipppppiiipiip"), ROW("ppppipiiif"), ROW("ppppipiiifi"), ROW("ppppippiiiiiiiifpiipp"),
    ROW("ppppippiippfiiiiiiiiiiip"), ROW("pppppiipppiipiiiip"), ROW("pppppippiiiiiiiiiiifiipp"), ROW("ppppppipiiii"),
    ROW("ppppppipiilii"), ROW("ppppppppiiifi"), ROW("ppppppppppiiiiifffi"), ROW("ppppppppppiiiiiifffp"),
};

struct Entry {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  Invoke invoke;
  Py_ssize_t count;
  void* fn;
  PyObject* find;                   // () -> the entry point's address; called once, by the first call
  PyObject* what;
};

bool ready(Entry* e) {
  if (e->fn) return true;
  PyObject* at = PyObject_CallNoArgs(e->find);
  if (!at) return false;
  e->fn = PyLong_AsVoidPtr(at);
  Py_DECREF(at);
  return e->fn != nullptr || (PyErr_Occurred() ? false : (PyErr_SetString(g_error, "an entry point without an address"), false));
}

bool finish(int rc, PyObject* what) {
  PyObject* n = PyList_GET_ITEM(g_launches, 0);
  PyObject* more = PyLong_FromLongLong(PyLong_AsLongLong(n) + 1);
  if (!more || PyList_SetItem(g_launches, 0, more)) return false;
  if (rc == 0) return true;
  if (rc == -1) PyErr_Format(g_error, "%U: refused its arguments (bad size or pointer)", what);
  else if (rc == -2) PyErr_Format(g_error, "%U: this size is legal but no kernel of this build takes it", what);
  else PyErr_Format(g_error, "%U: CUDA error %d", what, rc);
  return false;
}

// What ATen throws (no strides, no memory) becomes the exception that PyTorch makes of it: nothing of C++ may leave a function
// that the interpreter calls.
template <typename F> PyObject* guarded(F&& body) {
  try {
    return body();
  } catch (const std::exception&) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

PyObject* entry_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* names) {
  Entry* e = (Entry*)self;
  if ((names && PyTuple_GET_SIZE(names)) || PyVectorcall_NARGS(nargsf) != e->count)
    return PyErr_Format(PyExc_TypeError, "%U takes %zd arguments, by position", e->what, e->count);
  if (!ready(e)) return nullptr;
  return guarded([&]() -> PyObject* {
    bool bad = false;
    const int rc = e->invoke(e->fn, args, bad);
    if (bad || !finish(rc, e->what)) return nullptr;
    Py_RETURN_NONE;
  });
}

void entry_free(PyObject* self) {
  Py_XDECREF(((Entry*)self)->find);
  Py_XDECREF(((Entry*)self)->what);
  Py_TYPE(self)->tp_free(self);
}

PyTypeObject EntryType = {PyVarObject_HEAD_INIT(nullptr, 0) "rllm_launch.Entry"};

// entry(signature, find, what)
PyObject* make_entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3 || !PyUnicode_Check(args[0]) || !PyUnicode_Check(args[2])) return PyErr_Format(PyExc_TypeError, "entry(signature, find, what)");
  const char* text = PyUnicode_AsUTF8(args[0]);
  if (!text) return nullptr;
  for (const Row& row : kSignatures) {
    if (std::strcmp(row.text, text)) continue;
    Entry* e = PyObject_New(Entry, &EntryType);
    if (!e) return nullptr;
    e->vectorcall = entry_call;
    e->invoke = row.invoke;
    e->count = (Py_ssize_t)std::strlen(text);
    e->fn = nullptr;
    e->find = Py_NewRef(args[1]);
    e->what = Py_NewRef(args[2]);
    return (PyObject*)e;
  }
  return PyErr_Format(PyExc_ValueError, "no signature %s among those that were compiled", text);
}

// ---------------------------------------------------------------------------------------------------------------
// products
// ---------------------------------------------------------------------------------------------------------------
Entry *g_small = nullptr, *g_tcgen05 = nullptr;
long long g_small_rows = 0, g_min_tiles = 0;
void* g_error_word[64] = {};        // by device; null: ask Python

// products(small_m entry, tcgen05 entry, most rows of the first, fewest tiles of the second)
PyObject* set_products(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4 || Py_TYPE(args[0]) != &EntryType || Py_TYPE(args[1]) != &EntryType) return PyErr_Format(PyExc_TypeError, "products(entry, entry, rows, tiles)");
  g_small = (Entry*)Py_NewRef(args[0]);
  g_tcgen05 = (Entry*)Py_NewRef(args[1]);
  g_small_rows = PyLong_AsLongLong(args[2]);
  g_min_tiles = PyLong_AsLongLong(args[3]);
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

// error_word(device index, tensor): the word that the tcgen05 product reports to on that device (the caller keeps it)
PyObject* set_error_word(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    const long long d = n == 2 ? PyLong_AsLongLong(args[0]) : -1;
    if (d < 0 || d >= 64 || !THPVariable_Check(args[1])) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_TypeError, "error_word(device index, tensor)");
    g_error_word[d] = THPVariable_Unpack(args[1]).data_ptr();
    Py_RETURN_NONE;
  });
}

bool is(const char* value, const char* text) { return value && !std::strcmp(value, text); }

PyObject* checked_product(PyObject* const* args) {
  const at::Tensor &x = THPVariable_Unpack(args[0]), &w = THPVariable_Unpack(args[1]);
  const bool f32 = args[2] == Py_True, silu = args[3] == Py_True;
  if (!x.is_cuda() || !w.is_cuda() || x.dim() != 2 || w.dim() != 2 || x.scalar_type() != at::kBFloat16 || w.scalar_type() != at::kBFloat16)
    Py_RETURN_NONE;
  const long long M = x.size(0), K = x.size(1), N = silu ? w.size(0) / 2 : w.size(0), lda = x.stride(0), ldw = w.stride(0);
  if (M <= 0 || N <= 0 || w.size(1) != K || x.stride(1) != 1 || w.stride(1) != 1 || K % 8 || lda % 8 || ldw % 8 || (silu && w.size(0) != 2 * N))
    Py_RETURN_NONE;
  const char* mode = std::getenv("RLLM_GEMM");
  if (is(mode, "library")) Py_RETURN_NONE;
  const bool small = M <= g_small_rows;
  if (small) {
    if (!silu && w.size(0) > 65536 && (M > 8 || is(std::getenv("RLLM_HEAD"), "library"))) Py_RETURN_NONE;
  } else {
    if (is(mode, "no_tcgen05") || (((uintptr_t)x.data_ptr() | (uintptr_t)w.data_ptr()) & 15)) Py_RETURN_NONE;
    const long long cols = silu ? 128 : 256, tiles = (M + 127) / 128 * ((N + cols - 1) / cols);
    if (!is(mode, "tcgen05") && tiles < g_min_tiles) Py_RETURN_NONE;
  }
  const int device = x.get_device();
  Entry* e = small ? g_small : g_tcgen05;
  if (!small && (device < 0 || device >= 64 || !g_error_word[device])) Py_RETURN_NONE;
  if (!ready(e)) return nullptr;
  at::Tensor out = at::empty({M, N}, x.options().dtype(f32 ? at::kFloat : at::kBFloat16));
  bool bad = false;
  const float limit = Arg<'f'>::get(args[4], bad), slope = Arg<'f'>::get(args[5], bad), shift = Arg<'f'>::get(args[6], bad);
  if (bad) return nullptr;
  void *px = x.data_ptr(), *pw = w.data_ptr(), *po = out.data_ptr();
  const int code = silu ? 2 : (f32 ? 1 : 0);
  const cudaStream_t stream = stream_now();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  if (small)
    rc = reinterpret_cast<int (*)(void*, int, void*, int, void*, int, int, int, int, int, float, float, float, cudaStream_t)>(e->fn)(
        px, (int)lda, pw, (int)ldw, po, (int)N, (int)M, (int)N, (int)K, code, limit, slope, shift, stream);
  else
    rc = reinterpret_cast<int (*)(void*, int, void*, int, void*, int, int, int, int, int, float, float, float, void*, cudaStream_t)>(e->fn)(
        px, (int)lda, pw, (int)ldw, po, (int)N, (int)M, (int)N, (int)K, code, limit, slope, shift, g_error_word[device], stream);
  Py_END_ALLOW_THREADS
  if (!finish(rc, e->what)) return nullptr;
  return THPVariable_Wrap(std::move(out));
}

PyObject* product(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 7) return PyErr_Format(PyExc_TypeError, "product(x, w, out_f32, silu, limit, slope, shift)");
  if (!g_small || !THPVariable_CheckExact(args[0]) || !THPVariable_CheckExact(args[1])) Py_RETURN_NONE;      // tensors and parameters
  return guarded([&] { return checked_product(args); });
}

// setup(exception class, list of one int)
PyObject* setup(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2 || !PyList_Check(args[1]) || PyList_GET_SIZE(args[1]) != 1) return PyErr_Format(PyExc_TypeError, "setup(exception, [count])");
  g_error = Py_NewRef(args[0]);
  g_launches = Py_NewRef(args[1]);
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {{"setup", (PyCFunction)(void*)setup, METH_FASTCALL, nullptr},
                          {"entry", (PyCFunction)(void*)make_entry, METH_FASTCALL, nullptr},
                          {"products", (PyCFunction)(void*)set_products, METH_FASTCALL, nullptr},
                          {"error_word", (PyCFunction)(void*)set_error_word, METH_FASTCALL, nullptr},
                          {"product", (PyCFunction)(void*)product, METH_FASTCALL, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "launch", nullptr, -1, kMethods};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_launch() {
  EntryType.tp_basicsize = sizeof(Entry);
  EntryType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  EntryType.tp_vectorcall_offset = offsetof(Entry, vectorcall);
  EntryType.tp_call = PyVectorcall_Call;
  EntryType.tp_dealloc = entry_free;
  if (PyType_Ready(&EntryType) < 0) return nullptr;
  return PyModule_Create(&kModule);
}
