// Native half of the Python host path: argument checks, expression keys and the calls into the
// C ABI, for the calls that a program makes thousands of times.
//
// A short kernel takes 2-5 us of device time; walking its arguments in Python and through ctypes
// took 4 us for a product and 22 us for a batch-norm expression, so that small layers ran at the
// pace of the interpreter. Every function here is the fast path of a Python method of the same
// meaning (nervanagpu.py, float_ew.py): it returns None, having done nothing, whenever anything
// about the call is not the plain case (a failed check, timing output, an unusual argument), and
// the method then goes on to its full form, which raises the errors and prints the timings.
//
// Measured with the device idle (host time per call, median of 2000, before -> now): ng.dot 8.1 -> 4.6 us, the
// batch-norm expression 27.8 -> 8.5 us, O[:] = X + Y 11.6 -> 4.3 us, fprop_conv 5.9 -> 4.3 us.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include "../../include/nervana_b200.h"

namespace {

constexpr int kMaxDims = 6;
enum Dtype : int { kF16 = 0, kF32 = 1 };   // positions in the tuple that setup() is given

PyObject *g_tensor_type, *g_node_type, *g_prepare, *g_check, *g_dtypes, *g_ops;
PyObject* g_cache;   // expression key -> Launch
constexpr Py_ssize_t kCacheLimit = 4096;
constexpr int kMaxArgs = 1024;   // 4 KB of kernel parameters of 4 bytes and more

PyObject *s_gpudata, *s_shape, *s_strides, *s_dtype, *s_is_trans, *s_rounding, *s_take_array, *s_backend, *s_stream,
    *s_value, *s_ptr, *s_bench, *s_rand_state, *s_seed, *s_offset, *s_op, *s_axis, *s_as_parameter, *s_desc, *s_path, *s_sizeI, *s_sizeF,
    *s_sizeO;

// "not the plain case": forget the error, let the Python form of the call take over
PyObject* decline() {
  PyErr_Clear();
  Py_RETURN_NONE;
}

PyObject* failed(int rc) {   // raises NervanaError with the library's message
  PyObject* r = PyObject_CallFunction(g_check, "i", rc);
  if (r) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, "library call failed");
  }
  return nullptr;
}

// A C call as ctypes makes it: other threads run meanwhile. A launch waits while the stream's queue
// is full, and what the queued kernels wait for may be another thread's launch.
template <typename F>
int without_gil(F call) {
  PyThreadState* state = PyEval_SaveThread();
  const int rc = call();
  PyEval_RestoreThread(state);
  return rc;
}

// owned reference that goes away with its scope
struct Ref {
  PyObject* o;
  explicit Ref(PyObject* p) : o(p) {}
  ~Ref() { Py_XDECREF(o); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  explicit operator bool() const { return o != nullptr; }
};

bool to_ll(PyObject* o, long long& v) {
  if (!o || !PyLong_Check(o)) return false;
  v = PyLong_AsLongLong(o);
  return !(v == -1 && PyErr_Occurred());
}
bool attr_ll(PyObject* o, PyObject* name, long long& v) {
  Ref r(PyObject_GetAttr(o, name));
  return r && to_ll(r.o, v);
}

// Address behind a tensor's gpudata: an int, an allocation object with a `ptr`, or anything with __index__.
bool address(PyObject* data, unsigned long long& out) {
  if (data == Py_None) {
    out = 0;
    return true;
  }
  if (PyLong_Check(data)) {
    out = PyLong_AsUnsignedLongLong(data);
    return !PyErr_Occurred();
  }
  Ref idx(PyObject_GetAttr(data, s_ptr));
  if (!idx || !PyLong_Check(idx.o)) {
    PyErr_Clear();
    Ref i2(PyNumber_Index(data));
    if (!i2) return false;
    out = PyLong_AsUnsignedLongLong(i2.o);
    return !PyErr_Occurred();
  }
  out = PyLong_AsUnsignedLongLong(idx.o);
  return !PyErr_Occurred();
}

struct Tensor {
  unsigned long long ptr;
  long long shape[kMaxDims], strides[kMaxDims];
  int nd, dtype, is_trans, rounding;
  long long size() const {
    long long n = 1;
    for (int i = 0; i < nd; ++i) n *= shape[i];
    return n;
  }
};

bool read_dims(PyObject* seq, long long* out, int& n) {
  const bool tuple = PyTuple_Check(seq);
  if (!tuple && !PyList_Check(seq)) return false;
  n = static_cast<int>(tuple ? PyTuple_GET_SIZE(seq) : PyList_GET_SIZE(seq));
  if (n > kMaxDims) return false;
  for (int i = 0; i < n; ++i)
    if (!to_ll(tuple ? PyTuple_GET_ITEM(seq, i) : PyList_GET_ITEM(seq, i), out[i])) return false;
  return true;
}

// False for anything but a plain tensor (views through index arrays included).
bool read_tensor(PyObject* o, Tensor& t) {
  if (reinterpret_cast<PyObject*>(Py_TYPE(o)) != g_tensor_type) return false;
  {
    Ref take(PyObject_GetAttr(o, s_take_array));
    if (!take || take.o != Py_None) return false;
  }
  {
    Ref d(PyObject_GetAttr(o, s_gpudata));
    if (!d || !address(d.o, t.ptr)) return false;
  }
  int ns = 0;
  {
    Ref sh(PyObject_GetAttr(o, s_shape));
    if (!sh || !read_dims(sh.o, t.shape, t.nd)) return false;
    Ref st(PyObject_GetAttr(o, s_strides));
    if (!st || !read_dims(st.o, t.strides, ns) || ns != t.nd) return false;
  }
  {
    Ref dt(PyObject_GetAttr(o, s_dtype));
    if (!dt) return false;
    t.dtype = -1;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(g_dtypes); ++i)
      if (PyTuple_GET_ITEM(g_dtypes, i) == dt.o) t.dtype = static_cast<int>(i);
    if (t.dtype < 0) return false;
  }
  Ref tr(PyObject_GetAttr(o, s_is_trans));
  if (!tr) return false;
  t.is_trans = PyObject_IsTrue(tr.o);
  Ref ro(PyObject_GetAttr(o, s_rounding));
  if (!ro) return false;
  if (ro.o == Py_True) t.rounding = 10;
  else if (ro.o == Py_None) t.rounding = 0;
  else {
    long long v;
    if (!to_ll(ro.o, v)) return false;
    if (v < 0 || v > 255) return false;   // (one byte of an expression's key)
    t.rounding = static_cast<int>(v);
  }
  return t.is_trans >= 0;
}

// The forms of a stream that ctypes takes for a void pointer: None, an int, a c_void_p, or an object
// that says in _as_parameter_ which of these it stands for (a torch.cuda.Stream does).
bool read_stream(PyObject* backend, void*& stream) {
  stream = nullptr;
  if (backend == Py_None) return true;
  PyObject* s = PyObject_GetAttr(backend, s_stream);
  for (int depth = 0; s && depth < 8; ++depth) {
    if (s == Py_None || PyLong_Check(s)) {
      Ref v(s);
      if (s != Py_None) stream = reinterpret_cast<void*>(PyLong_AsUnsignedLongLong(s));
      return !PyErr_Occurred();
    }
    PyObject* next = PyObject_GetAttr(s, s_as_parameter);
    if (!next) {
      PyErr_Clear();
      next = PyObject_GetAttr(s, s_value);
    }
    Py_SETREF(s, next);
  }
  Py_XDECREF(s);
  return false;
}

// The position of a RandState (or None) in its random stream, moved on by one.
bool next_random(PyObject* rs, unsigned long long& seed, unsigned& offset) {
  seed = 0;
  offset = 0;
  if (rs == Py_None) return true;
  Ref sd(PyObject_GetAttr(rs, s_seed));
  if (!sd || !PyLong_Check(sd.o)) return false;
  seed = PyLong_AsUnsignedLongLongMask(sd.o);
  long long off;
  if (!attr_ll(rs, s_offset, off)) return false;
  offset = static_cast<unsigned>(off);
  Ref next(PyLong_FromUnsignedLong(static_cast<unsigned>(offset + 1u)));
  return next && PyObject_SetAttr(rs, s_offset, next.o) == 0;
}

bool as_float(PyObject* o, float& v) {
  const double d = PyFloat_AsDouble(o);
  if (d == -1.0 && PyErr_Occurred()) return false;
  v = static_cast<float>(d);
  return true;
}

// ------------------------------------------------------------------------------------------
// Expressions
// ------------------------------------------------------------------------------------------
// A prepared launch. The argument block belongs to ctypes objects that `keep` holds.
struct Launch {
  PyObject_HEAD
  void* kernel;
  unsigned grid[3], block[3];
  void** argv;
  int n_args;      // the last four: seed low, seed high, random offset, rounding
  PyObject* keep;
};

void launch_dealloc(PyObject* self) {
  Py_XDECREF(reinterpret_cast<Launch*>(self)->keep);
  Py_TYPE(self)->tp_free(self);
}

// Launch(kernel, grid, block, address and number of the argument pointers, owner)
PyObject* launch_new(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long kernel, argv;
  unsigned g[3], b[3];
  int n_args;
  PyObject* keep;
  if (!PyArg_ParseTuple(args, "K(III)(III)KiO", &kernel, &g[0], &g[1], &g[2], &b[0], &b[1], &b[2], &argv, &n_args, &keep))
    return nullptr;
  if (n_args < 4 || n_args > kMaxArgs) {
    PyErr_SetString(PyExc_ValueError, "too many kernel arguments");
    return nullptr;
  }
  Launch* l = reinterpret_cast<Launch*>(type->tp_alloc(type, 0));
  if (!l) return nullptr;
  l->kernel = reinterpret_cast<void*>(kernel);
  memcpy(l->grid, g, sizeof(g));
  memcpy(l->block, b, sizeof(b));
  l->argv = reinterpret_cast<void**>(argv);
  l->n_args = n_args;
  l->keep = Py_NewRef(keep);
  return reinterpret_cast<PyObject*>(l);
}

PyTypeObject g_launch_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// Runs a prepared launch on the backend's stream with the next random offset of `rs`. The caller
// holds a reference to it: another thread may run it at the same time, or drop it from the cache.
int launch_run(const Launch* l, PyObject* backend, PyObject* rs, bool& plain) {
  unsigned long long seed;
  unsigned off;
  void* stream;
  plain = read_stream(backend, stream) && next_random(rs, seed, off);
  if (!plain) return NG_ERR_INVALID_ARG;
  uint32_t lo = static_cast<uint32_t>(seed), hi = static_cast<uint32_t>(seed >> 32);
  void* argv[kMaxArgs];
  memcpy(argv, l->argv, sizeof(void*) * l->n_args);
  argv[l->n_args - 4] = &lo;
  argv[l->n_args - 3] = &hi;
  argv[l->n_args - 2] = &off;
  return without_gil([&] {
    return ng_ew_launch(l->kernel, l->grid[0], l->grid[1], l->grid[2], l->block[0], l->block[1], l->block[2], 0, argv,
                        stream);
  });
}

// Key of an expression: everything its prepared launch depends on, in postfix order. A tensor
// object that occurs again is named by the number of its first occurrence.
struct Key {
  unsigned char buf[2048];
  size_t n = 0;
  PyObject* seen[32];
  int n_seen = 0;
  bool put(const void* p, size_t bytes) {
    if (n + bytes > sizeof(buf)) return false;
    memcpy(buf + n, p, bytes);
    n += bytes;
    return true;
  }
  bool tag(char c) { return put(&c, 1); }

  bool leaf(PyObject* o) {
    if (PyFloat_CheckExact(o) || PyLong_CheckExact(o)) {
      const double d = PyFloat_AsDouble(o);
      if (d == -1.0 && PyErr_Occurred()) return false;
      return tag('c') && put(&d, sizeof(d));
    }
    for (int i = 0; i < n_seen; ++i)
      if (seen[i] == o) return tag('s') && tag(static_cast<char>(i));
    Tensor t;
    if (n_seen == 32 || !read_tensor(o, t)) return false;
    seen[n_seen++] = o;
    const unsigned char head[4] = {static_cast<unsigned char>(t.nd), static_cast<unsigned char>(t.dtype),
                                   static_cast<unsigned char>(t.is_trans), static_cast<unsigned char>(t.rounding)};
    return tag('t') && put(head, 4) && put(&t.ptr, 8) && put(t.shape, 8 * t.nd) && put(t.strides, 8 * t.nd);
  }
  bool op(PyObject* d) {   // {"op": name} or {"op": name, "axis": 0 or 1}
    if (!PyDict_CheckExact(d)) return false;
    PyObject* name = PyDict_GetItemWithError(d, s_op);
    PyObject* id = name ? PyDict_GetItemWithError(g_ops, name) : nullptr;
    long long v, axis = -1;
    if (!to_ll(id, v)) return false;
    const Py_ssize_t items = PyDict_GET_SIZE(d);
    if (items == 2) {
      PyObject* a = PyDict_GetItemWithError(d, s_axis);
      if (!to_ll(a, axis) || axis < 0 || axis > 1) return false;
    } else if (items != 1) {
      return false;
    }
    const char c[3] = {'o', static_cast<char>(v), static_cast<char>(axis)};
    return put(c, 3);
  }
  bool node(PyObject* t, int depth) {
    if (depth > 64 || PyTuple_GET_SIZE(t) != 3) return false;
    for (int i = 1; i <= 2; ++i) {
      PyObject* c = PyTuple_GET_ITEM(t, i);
      if (reinterpret_cast<PyObject*>(Py_TYPE(c)) == g_node_type) {
        if (!node(c, depth + 1)) return false;
      } else if (c != Py_None && !leaf(c)) {
        return false;
      }
    }
    return op(PyTuple_GET_ITEM(t, 0));
  }
};

// assign(out, value): out[...] = value, a node, tensor or number. Returns out.
PyObject* py_assign(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) return decline();
  PyObject *out = args[0], *value = args[1];
  Key key;
  if (!key.leaf(out)) return decline();
  const bool is_node = reinterpret_cast<PyObject*>(Py_TYPE(value)) == g_node_type;
  if (!(is_node ? key.node(value, 0) : key.leaf(value))) return decline();
  Ref backend(PyObject_GetAttr(out, s_backend));
  if (!backend) return decline();
  {
    Ref bench(PyObject_GetAttr(backend.o, s_bench));
    if (!bench || (bench.o != Py_False && bench.o != Py_None && bench.o != Py_True)) return decline();
  }
  Ref k(PyBytes_FromStringAndSize(reinterpret_cast<const char*>(key.buf), static_cast<Py_ssize_t>(key.n)));
  if (!k) return nullptr;
  PyObject* hit = PyDict_GetItemWithError(g_cache, k.o);
  Ref fresh(nullptr);
  if (!hit) {
    if (PyErr_Occurred()) return nullptr;
    fresh.o = PyObject_CallFunctionObjArgs(g_prepare, out, value, nullptr);   // analyses, generates and compiles
    if (!fresh) return nullptr;
    if (!PyObject_TypeCheck(fresh.o, &g_launch_type)) return decline();       // an empty tensor
    if (PyDict_GET_SIZE(g_cache) >= kCacheLimit) PyDict_Clear(g_cache);
    if (PyDict_SetItem(g_cache, k.o, fresh.o) != 0) return nullptr;
    hit = fresh.o;
  }
  Ref held(Py_NewRef(hit)), rs(PyObject_GetAttr(backend.o, s_rand_state));
  if (!rs) return decline();
  bool plain;
  const int rc = launch_run(reinterpret_cast<Launch*>(hit), backend.o, rs.o, plain);
  if (!plain) return decline();
  if (rc != NG_OK) return failed(rc);
  return Py_NewRef(out);
}

// run(launch, backend, random state or None): a launch the caller looked up itself
PyObject* py_run(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3 || !PyObject_TypeCheck(args[0], &g_launch_type)) {
    PyErr_SetString(PyExc_TypeError, "run(launch, backend, rand_state)");
    return nullptr;
  }
  bool plain;
  const int rc = launch_run(reinterpret_cast<Launch*>(args[0]), args[1], args[2], plain);
  if (!plain) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "the backend has no usable stream or random state");
    return nullptr;
  }
  if (rc != NG_OK) return failed(rc);
  Py_RETURN_TRUE;
}

// node(op dict, a, b): an OpTreeNode; NotImplemented for operands that are no tensor, node or number
PyObject* py_node(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) {
    PyErr_SetString(PyExc_TypeError, "node(op, a, b)");
    return nullptr;
  }
  for (int i = 1; i <= 2; ++i) {
    PyObject* a = args[i];
    PyObject* ty = reinterpret_cast<PyObject*>(Py_TYPE(a));
    if (ty == g_tensor_type || ty == g_node_type || a == Py_None || PyFloat_Check(a) || PyLong_Check(a)) continue;
    const int sub = PyObject_IsInstance(a, g_tensor_type);
    if (sub < 0) return nullptr;
    if (!sub && !PyObject_TypeCheck(a, reinterpret_cast<PyTypeObject*>(g_node_type))) Py_RETURN_NOTIMPLEMENTED;
  }
  PyTypeObject* type = reinterpret_cast<PyTypeObject*>(g_node_type);
  PyObject* t = type->tp_alloc(type, 3);
  if (!t) return nullptr;
  for (int i = 0; i < 3; ++i) PyTuple_SET_ITEM(t, i, Py_NewRef(args[i]));
  return t;
}

// ------------------------------------------------------------------------------------------
// Products, convolutions, pooling, copies
// ------------------------------------------------------------------------------------------
bool unit_rows(const Tensor& t, int first, long long& ld, int dims) {   // one stride is 1, ld is the other
  long long lo = t.strides[first], hi = lo;
  for (int i = first; i < first + dims; ++i) {
    lo = t.strides[i] < lo ? t.strides[i] : lo;
    hi = t.strides[i] > hi ? t.strides[i] : hi;
  }
  ld = hi;
  return lo == 1 && hi <= 0x7fffffff;
}

bool rounding_bits(PyObject* arg, const Tensor& c, int& sr) {
  if (arg == Py_None) sr = c.rounding;
  else if (arg == Py_True) sr = 10;
  else if (arg == Py_False) sr = 0;
  else {
    long long v;
    if (!to_ll(arg, v)) return false;
    sr = static_cast<int>(v);
  }
  return true;
}

struct Product {
  Tensor a, b, c;
  long long lda, ldb, ldc;
  int m, n, k, relu, sr;
  float alpha, beta;
  unsigned long long seed;
  unsigned off;
  void* stream;
};

// (backend, A, B, C, alpha, beta, relu, stochastic_round); fa / fb / fc: first matrix dimension of each
bool read_product(PyObject* const* args, Product& p, int fa, int fb, int fc) {
  if (p.a.dtype != kF16 || p.b.dtype != kF16 || p.c.dtype != kF16) return false;
  if (!unit_rows(p.a, fa, p.lda, 2) || !unit_rows(p.b, fb, p.ldb, 2) || !unit_rows(p.c, fc, p.ldc, 2)) return false;
  if (p.a.is_trans && p.b.is_trans) return false;
  const long long m = p.a.shape[fa], n = p.b.shape[fb + 1], k = p.a.shape[fa + 1];
  if (m != p.c.shape[fc] || n != p.c.shape[fc + 1] || k != p.b.shape[fb] || m > 0x7fffffff || n > 0x7fffffff || k > 0x7fffffff)
    return false;
  p.m = static_cast<int>(m); p.n = static_cast<int>(n); p.k = static_cast<int>(k);
  if (!as_float(args[4], p.alpha) || !as_float(args[5], p.beta)) return false;
  p.relu = PyObject_IsTrue(args[6]);
  if (p.relu < 0 || !rounding_bits(args[7], p.c, p.sr) || !read_stream(args[0], p.stream)) return false;
  p.seed = 0;
  p.off = 0;
  if (p.sr == 0) return true;     // no random bits wanted
  Ref rs(PyObject_GetAttr(args[0], s_rand_state));
  return rs && next_random(rs.o, p.seed, p.off);   // (last: it moves the random stream on)
}

PyObject* py_dot(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Product p;
  if (n != 8 || !read_tensor(args[1], p.a) || !read_tensor(args[2], p.b) || !read_tensor(args[3], p.c) || p.a.nd != 2 ||
      p.b.nd != 2 || p.c.nd != 2 || !read_product(args, p, 0, 0, 0))
    return decline();
  const int rc = without_gil([&] {
    return ng_hgemm(reinterpret_cast<void*>(p.a.ptr), reinterpret_cast<void*>(p.b.ptr), reinterpret_cast<void*>(p.c.ptr),
                    p.a.is_trans, p.b.is_trans, p.m, p.n, p.k, static_cast<int>(p.lda), static_cast<int>(p.ldb),
                    static_cast<int>(p.ldc), p.alpha, p.beta, p.relu, p.sr, p.seed, p.off, p.stream);
  });
  if (rc != NG_OK) return failed(rc);
  return Py_NewRef(args[3]);
}

PyObject* py_batched_dot(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Product p;
  if (n != 8 || !read_tensor(args[1], p.a) || !read_tensor(args[2], p.b) || !read_tensor(args[3], p.c)) return decline();
  const int fa = p.a.nd == 3, fb = p.b.nd == 3, fc = p.c.nd == 3;
  if (p.a.nd != 2 + fa || p.b.nd != 2 + fb || p.c.nd != 2 + fc || !(fa || fb)) return decline();
  const long long batch = fa ? p.a.shape[0] : p.b.shape[0];
  if ((fa && fb && p.b.shape[0] != batch) || (fc && p.c.shape[0] != batch) || batch < 1 || batch > 0x7fffffff)
    return decline();
  if (!read_product(args, p, fa, fb, fc)) return decline();
  const int rc = without_gil([&] {
    return ng_hgemm_batched(reinterpret_cast<void*>(p.a.ptr), reinterpret_cast<void*>(p.b.ptr),
                            reinterpret_cast<void*>(p.c.ptr), p.a.is_trans, p.b.is_trans, p.m, p.n, p.k,
                            static_cast<int>(p.lda), static_cast<int>(p.ldb), static_cast<int>(p.ldc), p.alpha, p.beta,
                            p.relu, p.sr, p.seed, p.off, fc ? static_cast<int>(batch) : 1,
                            fc ? 1 : static_cast<int>(batch), fa ? p.a.strides[0] : 0, fb ? p.b.strides[0] : 0,
                            fc ? p.c.strides[0] : 0, p.stream);
  });
  if (rc != NG_OK) return failed(rc);
  return Py_NewRef(args[3]);
}

// The C descriptor that a layer object carries (a ctypes structure).
template <typename D>
bool read_desc(PyObject* layer, D& out) {
  Ref d(PyObject_GetAttr(layer, s_desc));
  Py_buffer view;
  if (!d || PyObject_GetBuffer(d.o, &view, PyBUF_SIMPLE) != 0) return false;
  const bool ok = view.len == static_cast<Py_ssize_t>(sizeof(D));
  if (ok) memcpy(&out, view.buf, sizeof(D));
  PyBuffer_Release(&view);
  return ok;
}

// conv(pass, backend, layer, I or F, ..., alpha, relu): pass 0 (I, F, O), 1 (F, E, dI), 2 (I, E, dF)
PyObject* py_conv(PyObject*, PyObject* const* args, Py_ssize_t n) {
  long long pass, path, si, sf, so;
  Tensor a, b, c;
  ng_conv_desc d;
  float alpha;
  void* stream;
  if (n != 8 || !to_ll(args[0], pass) || !read_tensor(args[3], a) || !read_tensor(args[4], b) || !read_tensor(args[5], c) ||
      !attr_ll(args[2], s_sizeI, si) || !attr_ll(args[2], s_sizeF, sf) || !attr_ll(args[2], s_sizeO, so) ||
      !attr_ll(args[2], s_path, path) || !as_float(args[6], alpha) || !read_desc(args[2], d) || !read_stream(args[1], stream))
    return decline();
  const int relu = PyObject_IsTrue(args[7]);
  const long long want[3][3] = {{si, sf, so}, {sf, so, si}, {si, so, sf}};
  if (relu < 0 || pass < 0 || pass > 2 || a.size() != want[pass][0] || b.size() != want[pass][1] || c.size() != want[pass][2])
    return decline();
  if (a.dtype != kF16 || b.dtype != kF16 || !(c.dtype == kF16 || (pass == 2 && c.dtype == kF32))) return decline();
  void *pa = reinterpret_cast<void*>(a.ptr), *pb = reinterpret_cast<void*>(b.ptr), *pc = reinterpret_cast<void*>(c.ptr);
  const int rc = without_gil([&] {
    if (pass == 0) return ng_conv_fprop(&d, pa, pb, pc, alpha, relu, static_cast<int>(path), stream);
    if (pass == 1) return ng_conv_bprop(&d, pa, pb, pc, alpha, static_cast<int>(path), stream);
    return ng_conv_update(&d, pa, pb, pc, c.dtype == kF32, alpha, static_cast<int>(path), stream);
  });
  if (rc != NG_OK) return failed(rc);
  Py_RETURN_TRUE;
}

// pool(backend, layer, I, O or E, gradI or None, mode, argmax or None): max pooling; mode 0 forward,
// 1 backward, 2 backward with the ReLU mask
PyObject* py_pool(PyObject*, PyObject* const* args, Py_ssize_t n) {
  long long si, so, mode;
  Tensor in, eo, out = {}, arg = {};
  ng_pool_desc d;
  void* stream;
  if (n != 7 || !read_tensor(args[2], in) || !read_tensor(args[3], eo) || !attr_ll(args[1], s_sizeI, si) ||
      !attr_ll(args[1], s_sizeO, so) || !to_ll(args[5], mode) || !read_desc(args[1], d) || !read_stream(args[0], stream))
    return decline();
  {
    Ref op(PyObject_GetAttr(args[1], s_op));
    if (!op || !PyUnicode_Check(op.o) || PyUnicode_CompareWithASCIIString(op.o, "max") != 0) return decline();
  }
  const bool record = args[6] != Py_None;
  if (in.dtype != eo.dtype || (in.dtype != kF16 && in.dtype != kF32) || in.size() != si || eo.size() != so || mode < 0 || mode > 2)
    return decline();
  if (mode != 0 && (!read_tensor(args[4], out) || out.dtype != in.dtype || out.size() != si)) return decline();
  if (record && (!read_tensor(args[6], arg) || arg.dtype <= kF32 || arg.size() < so)) return decline();
  const int esz = in.dtype == kF16 ? 2 : 4;
  void *pi = reinterpret_cast<void*>(in.ptr), *pe = reinterpret_cast<void*>(eo.ptr), *po = reinterpret_cast<void*>(out.ptr),
       *pr = reinterpret_cast<void*>(arg.ptr);
  const int rc = without_gil([&] {
    if (mode == 0) return record ? ng_pool_fprop_argmax(&d, esz, pi, pe, pr, stream) : ng_pool_fprop(&d, esz, pi, pe, stream);
    if (record) return ng_pool_bprop_argmax(&d, esz, pr, pe, po, mode == 2, stream);
    return mode == 1 ? ng_pool_bprop(&d, esz, pi, pe, po, stream) : ng_pool_bprop_relu(&d, esz, pi, pe, po, stream);
  });
  if (rc != NG_OK) return failed(rc);
  Py_RETURN_TRUE;
}

// setup(tensor type, node type, prepare, check, dtypes (fp16 and fp32 first), {operation: number})
PyObject* py_setup(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 6 || !PyTuple_Check(args[4]) || !PyDict_Check(args[5])) {
    PyErr_SetString(PyExc_TypeError, "setup(tensor, node, prepare, check, dtypes, ops)");
    return nullptr;
  }
  PyObject** slots[6] = {&g_tensor_type, &g_node_type, &g_prepare, &g_check, &g_dtypes, &g_ops};
  for (int i = 0; i < 6; ++i) Py_XSETREF(*slots[i], Py_NewRef(args[i]));
  Py_RETURN_NONE;
}

#define NG_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {NG_METHOD("setup", py_setup), NG_METHOD("node", py_node), NG_METHOD("assign", py_assign),
                           NG_METHOD("run", py_run), NG_METHOD("dot", py_dot), NG_METHOD("batched_dot", py_batched_dot),
                           NG_METHOD("conv", py_conv), NG_METHOD("pool", py_pool), {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  struct {
    PyObject** slot;
    const char* text;
  } names[] = {{&s_gpudata, "gpudata"}, {&s_shape, "shape"}, {&s_strides, "strides"}, {&s_dtype, "dtype"},
               {&s_is_trans, "is_trans"}, {&s_rounding, "rounding"}, {&s_take_array, "take_array"},
               {&s_backend, "backend"}, {&s_stream, "stream"}, {&s_value, "value"}, {&s_ptr, "ptr"}, {&s_bench, "bench"},
               {&s_rand_state, "rand_state"}, {&s_seed, "seed"}, {&s_offset, "offset"}, {&s_op, "op"}, {&s_axis, "axis"},
               {&s_as_parameter, "_as_parameter_"},
               {&s_desc, "desc"}, {&s_path, "path"}, {&s_sizeI, "sizeI"}, {&s_sizeF, "sizeF"}, {&s_sizeO, "sizeO"}};
  for (auto& x : names)
    if (!(*x.slot = PyUnicode_InternFromString(x.text))) return nullptr;
  if (!(g_cache = PyDict_New())) return nullptr;
  g_launch_type.tp_name = "nervanagpu_b200._native.Launch";
  g_launch_type.tp_basicsize = sizeof(Launch);
  g_launch_type.tp_flags = Py_TPFLAGS_DEFAULT;
  g_launch_type.tp_new = launch_new;
  g_launch_type.tp_dealloc = launch_dealloc;
  if (PyType_Ready(&g_launch_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&g_module);
  if (!m) return nullptr;
  if (PyModule_AddObjectRef(m, "Launch", reinterpret_cast<PyObject*>(&g_launch_type)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
