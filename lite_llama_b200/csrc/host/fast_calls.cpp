// The plain form of the hot kernel shims in native code: tensors that need no conversion, no copy and no reshape go from the
// Python call to the C ABI (include/b200_lite_kernels.h) without ctypes and without Tensor attribute lookups in Python.  A
// decode step calls a few dozen shims, and a kernel takes 4 - 20 us: w8a16_matmul took 13.5 us of host time in Python (5 of
// them in ctypes and the launch), here 5.5; skip_rmsnorm 9.6 and 5.2.
//
// Every function returns None for anything else (other dimensions, strides, types or devices, a bias, tensor subclasses,
// wrapped or fake tensors, active torch modes): the Python shim then does what it always did, error messages included.  The
// results are those of the Python path: same kernels, same arguments, outputs without a gradient; exceptions too (torch's own
// translation: an allocation that fails is a torch.OutOfMemoryError, which the graph captures of ModelRunner wait for).
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <unordered_map>

namespace {

using i64 = int64_t;
struct {
  int64_t (*quant_workspace)(int, i64, i64, i64, i64);
  int64_t (*linear_workspace)(i64, i64, i64, int);
  int (*w8a16)(void*, const void*, const void*, int, const void*, const void*, int, i64, i64, i64, i64, i64, i64, i64, i64, i64,
               i64, void*, i64, void*, i64, void*);
  int (*w4a16)(void*, const void*, const void*, const void*, const void*, const void*, int, i64, i64, i64, int, int, i64, i64, i64,
               void*, i64, void*, i64, int, void*);
  int (*linear)(void*, const void*, const void*, const void*, i64, i64, i64, i64, i64, i64, void*, i64, void*, i64, int, void*);
  int (*w8a8)(void*, const void*, const void*, const void*, const void*, const void*, i64, i64, i64, i64, i64, i64, void*, i64,
              void*, i64, int, void*);
  int (*quantize)(void*, void*, const void*, i64, i64, i64, i64, int, void*);
  int (*norm)(void*, const void*, void*, const void*, i64, i64, i64, i64, i64, float, int, void*);
  int (*norm_quant)(void*, void*, const void*, void*, const void*, i64, i64, i64, i64, i64, float, int, void*);
  int (*swiglu)(void*, const void*, const void*, i64, i64, i64, i64, i64, int, void*);
  const char* (*last_error)();
} abi;
PyObject* py_zeroed = nullptr;      // kernels._common.zeroed_workspace(bytes, device)
PyObject* py_counters = nullptr;    // kernels._common.counters(device)

// ---- which calls are plain ----
constexpr c10::DispatchKeySet kPlainKeys({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::AutocastCUDA,
                                          c10::DispatchKey::ADInplaceOrView});

// a dense CUDA tensor that is exactly a torch.Tensor (or Parameter); nullptr otherwise
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.defined() && (t.key_set().raw_repr() & ~kPlainKeys.raw_repr()) == 0 && t.is_cuda() ? &t : nullptr;
}
// the current device if every tensor is plain and there, and no mode wants to see the call; -1 otherwise.  A missing function
// (a library built from a subset of the sources) counts as not plain: the Python shim names it.
template <class F>
int device_for(F* fn, std::initializer_list<const at::Tensor*> ts) {
  if (!fn || c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled()) return -1;
  for (const at::Tensor* t : ts)
    if (!t) return -1;
  const int device = c10::cuda::current_device();
  for (const at::Tensor* t : ts)
    if (t->get_device() != device) return -1;
  return device;
}
// ctypes lets other threads run while a launch waits for room in its queue; so does this
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};
int half_code(const at::Tensor& t) { return t.scalar_type() == at::kHalf ? 0 : t.scalar_type() == at::kBFloat16 ? 1 : -1; }
// matrix with unit column stride and at least one element
bool matrix(const at::Tensor& t) { return t.dim() == 2 && t.stride(1) == 1 && t.size(0) > 0 && t.size(1) > 0; }
// activation rows as TMA reads them
bool tma_rows(const at::Tensor& t) { return matrix(t) && t.stride(0) % 8 == 0 && (uintptr_t)t.data_ptr() % 16 == 0; }

PyObject* none() { Py_RETURN_NONE; }
PyObject* failed(int rc) {
  PyErr_Format(PyExc_ValueError, "b200lite error %d: %s", rc, abi.last_error());
  return nullptr;
}
void* stream(int device) { return (void*)c10::cuda::getCurrentCUDAStream(device).stream(); }

// The persistent buffers of kernels/_common.py, one per device; asked for again when a call needs more than before.
struct Kept { at::Tensor zeroed, counters; };
std::unordered_map<int, Kept>& kept() {
  static auto* m = new std::unordered_map<int, Kept>;      // outlives the interpreter's module teardown
  return *m;
}
bool fetch(PyObject* fn, PyObject* args, at::Tensor& out) {
  if (!args) return false;
  PyObject* r = PyObject_CallObject(fn, args);
  Py_DECREF(args);
  if (!r) return false;
  const bool ok = THPVariable_Check(r);
  if (ok) out = THPVariable_Unpack(r);
  Py_DECREF(r);
  if (!ok) PyErr_SetString(PyExc_RuntimeError, "buffer is not a tensor");
  return ok;
}
PyObject* device_of(PyObject* tensor) { return PyObject_GetAttrString(tensor, "device"); }
bool need_counters(int device, PyObject* like, Kept& k) {
  if (k.counters.defined()) return true;
  return fetch(py_counters, Py_BuildValue("(N)", device_of(like)), k.counters);
}
bool need_zeroed(i64 bytes, PyObject* like, Kept& k) {
  if (bytes <= 0 || (k.zeroed.defined() && k.zeroed.numel() >= bytes)) return true;
  return fetch(py_zeroed, Py_BuildValue("(LN)", (long long)bytes, device_of(like)), k.zeroed);
}

// workspace of a quantised GEMM, remembered by its sizes (the plan walks over the tiles); bounded
struct Sizes {
  i64 kind, m, n, k, group, device;
  bool operator==(const Sizes& o) const { return kind == o.kind && m == o.m && n == o.n && k == o.k && group == o.group && device == o.device; }
};
struct Hash {
  size_t operator()(const Sizes& s) const {
    size_t h = 1469598103934665603ull;
    for (i64 v : {s.kind, s.m, s.n, s.k, s.group, s.device}) h = (h ^ (size_t)v) * 1099511628211ull;
    return h;
  }
};
i64 quant_workspace(int kind, i64 m, i64 n, i64 k, i64 group, int device) {
  static auto* seen = new std::unordered_map<Sizes, i64, Hash>;
  const Sizes s{kind, m, n, k, group, device};
  auto it = seen->find(s);
  if (it != seen->end()) return it->second;
  if (seen->size() >= 4096) seen->clear();
  return (*seen)[s] = abi.quant_workspace(kind, m, n, k, group);
}

// Torch's translation of exceptions, without the buffer for warnings of HANDLE_TH_ERRORS: nothing here warns.
#define FAST_BEGIN try {
#define FAST_END                                                      \
  }                                                                   \
  catch (...) {                                                       \
    torch::translate_exception_to_python(std::current_exception());   \
    return nullptr;                                                   \
  }
#define ARGS(n) \
  if (count != (n)) { PyErr_SetString(PyExc_TypeError, "wrong number of arguments"); return nullptr; }

// (x, qweight, scales, group_n, group_k) -> y
PyObject* w8a16(PyObject*, PyObject* const* a, Py_ssize_t count) {
  ARGS(5)
  FAST_BEGIN
  const at::Tensor *x = plain(a[0]), *q = plain(a[1]), *s = plain(a[2]);
  const int device = device_for(abi.w8a16, {x, q, s});
  if (device < 0 || !PyLong_CheckExact(a[3]) || !PyLong_CheckExact(a[4])) return none();
  const bool fp8 = q->scalar_type() == at::kByte;
  if ((!fp8 && q->scalar_type() != at::kChar) || x->scalar_type() != at::kHalf || s->scalar_type() != at::kFloat) return none();
  if (!tma_rows(*x) || !matrix(*q) || s->dim() != 2 || x->size(1) != q->size(1)) return none();
  const i64 gn = PyLong_AsLongLong(a[3]), gk = PyLong_AsLongLong(a[4]), m = x->size(0), n = q->size(0), k = q->size(1);
  if (PyErr_Occurred()) return nullptr;
  if (gn < 1 || gk < 1 || (gk % 128 != 0 && gk < k)) return none();
  Kept& kp = kept()[device];
  const int kind = fp8 ? 1 : 2;
  const i64 bytes = quant_workspace(kind, m, n, k, gk, device);
  if (!need_zeroed(bytes, a[0], kp) || !need_counters(device, a[0], kp)) return nullptr;
  void* zeroed = bytes > 0 ? kp.zeroed.data_ptr() : nullptr;
  void* tickets = kp.counters.data_ptr();
  const i64 num_tickets = kp.counters.numel();
  at::Tensor y;
  int rc;
  {
    const Unlocked unlocked;
    y = at::empty({m, n}, x->options());
    rc = abi.w8a16(y.data_ptr(), x->data_ptr(), q->data_ptr(), fp8 ? 1 : 0, s->data_ptr(), nullptr, 0, m, n, k, gn, gk,
                   x->stride(0), q->stride(0), s->stride(0), s->stride(1), n, zeroed,
                   bytes, tickets, num_tickets, stream(device));
  }
  return rc ? failed(rc) : THPVariable_Wrap(std::move(y));
  FAST_END
}

// (x, qweight, scales, zeros, n, k, group_size, zeros_foldable, swiglu) -> y
PyObject* w4a16_packed(PyObject*, PyObject* const* a, Py_ssize_t count) {
  ARGS(9)
  FAST_BEGIN
  const at::Tensor *x = plain(a[0]), *q = plain(a[1]), *s = plain(a[2]), *z = plain(a[3]);
  const int device = device_for(abi.w4a16, {x, q, s, z});
  if (device < 0) return none();
  for (int i = 4; i < 7; ++i)
    if (!PyLong_CheckExact(a[i])) return none();
  const i64 n = PyLong_AsLongLong(a[4]), k = PyLong_AsLongLong(a[5]), group = PyLong_AsLongLong(a[6]);
  const int fold = PyObject_IsTrue(a[7]), swiglu = PyObject_IsTrue(a[8]);
  if (PyErr_Occurred()) return nullptr;
  if (x->scalar_type() != at::kHalf || !tma_rows(*x) || x->size(1) != k || q->dim() != 2) return none();
  const i64 m = x->size(0), out = swiglu ? n / 2 : n;
  Kept& kp = kept()[device];
  const i64 bytes = quant_workspace(0, m, n, k, group, device);
  if (!need_zeroed(bytes, a[0], kp) || !need_counters(device, a[0], kp)) return nullptr;
  void* zeroed = bytes > 0 ? kp.zeroed.data_ptr() : nullptr;
  void* tickets = kp.counters.data_ptr();
  const i64 num_tickets = kp.counters.numel();
  at::Tensor y;
  int rc;
  {
    const Unlocked unlocked;
    y = at::empty({m, out}, x->options());
    rc = abi.w4a16(y.data_ptr(), x->data_ptr(), q->data_ptr(), s->data_ptr(), z->data_ptr(), nullptr, 0, m, n, k, (int)group,
                   fold, x->stride(0), q->stride(0), out, zeroed, bytes,
                   tickets, num_tickets, swiglu, stream(device));
  }
  return rc ? failed(rc) : THPVariable_Wrap(std::move(y));
  FAST_END
}

// (x, weight) -> y
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t count) {
  ARGS(2)
  FAST_BEGIN
  const at::Tensor *x = plain(a[0]), *w = plain(a[1]);
  const int device = device_for(abi.linear, {x, w});
  if (device < 0) return none();
  const int code = half_code(*x);
  if (code < 0 || w->scalar_type() != x->scalar_type() || !tma_rows(*x) || !matrix(*w) || x->size(1) % 8 != 0 || x->size(1) != w->size(1))
    return none();
  const i64 m = x->size(0), n = w->size(0), k = w->size(1), bytes = abi.linear_workspace(m, n, k, 2);
  Kept& kp = kept()[device];
  if (!need_counters(device, a[0], kp)) return nullptr;
  void* tickets = kp.counters.data_ptr();
  const i64 num_tickets = kp.counters.numel();
  at::Tensor y, ws;
  int rc;
  {
    const Unlocked unlocked;
    y = at::empty({m, n}, x->options());
    if (bytes > 0) ws = at::empty({bytes}, x->options().dtype(at::kByte));
    rc = abi.linear(y.data_ptr(), x->data_ptr(), w->data_ptr(), nullptr, m, n, k, x->stride(0), w->stride(0), n,
                    bytes > 0 ? ws.data_ptr() : nullptr, bytes, tickets, num_tickets, code, stream(device));
  }
  return rc ? failed(rc) : THPVariable_Wrap(std::move(y));
  FAST_END
}

// (qa, a_scales, qweight, weight_scales [N] or [N, 1], bfloat16 out) -> y
PyObject* w8a8(PyObject*, PyObject* const* a, Py_ssize_t count) {
  ARGS(5)
  FAST_BEGIN
  const at::Tensor *x = plain(a[0]), *sa = plain(a[1]), *w = plain(a[2]), *sw = plain(a[3]);
  const int device = device_for(abi.w8a8, {x, sa, w, sw});
  if (device < 0) return none();
  const int bf16 = PyObject_IsTrue(a[4]);
  if (bf16 < 0) return nullptr;
  if (x->scalar_type() != at::kChar || w->scalar_type() != at::kChar || sa->scalar_type() != at::kFloat || sw->scalar_type() != at::kFloat)
    return none();
  if (!matrix(*x) || !matrix(*w) || x->size(1) != w->size(1) || x->size(1) % 16 != 0 || w->stride(0) % 16 != 0) return none();
  const i64 m = x->size(0), n = w->size(0), k = w->size(1);
  if (!sa->is_contiguous() || !sw->is_contiguous() || sw->dim() > 2 || (sw->dim() == 2 && sw->size(1) != 1)) return none();
  const i64 bytes = abi.linear_workspace(m, n, k, 1);
  Kept& kp = kept()[device];
  if (!need_counters(device, a[0], kp)) return nullptr;
  void* tickets = kp.counters.data_ptr();
  const i64 num_tickets = kp.counters.numel();
  at::Tensor y, ws;
  int rc;
  {
    const Unlocked unlocked;
    y = at::empty({m, n}, x->options().dtype(bf16 ? at::kBFloat16 : at::kHalf));
    if (bytes > 0) ws = at::empty({bytes}, x->options().dtype(at::kByte));
    rc = abi.w8a8(y.data_ptr(), x->data_ptr(), w->data_ptr(), sa->data_ptr(), sw->data_ptr(), nullptr, m, n, k, x->stride(0),
                  w->stride(0), n, bytes > 0 ? ws.data_ptr() : nullptr, bytes, tickets, num_tickets,
                  bf16, stream(device));
  }
  return rc ? failed(rc) : THPVariable_Wrap(std::move(y));
  FAST_END
}

PyObject* pair_of(at::Tensor a, at::Tensor b) {
  PyObject* r = PyTuple_New(2);
  if (!r) return nullptr;
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(a)));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(b)));
  return r;
}

// (a) -> (q, scales)
PyObject* quantize(PyObject*, PyObject* const* a, Py_ssize_t count) {
  ARGS(1)
  FAST_BEGIN
  const at::Tensor* x = plain(a[0]);
  const int device = device_for(abi.quantize, {x});
  if (device < 0) return none();
  const int code = half_code(*x);
  if (code < 0 || !matrix(*x)) return none();
  const i64 m = x->size(0), k = x->size(1);
  at::Tensor q, s;
  int rc;
  {
    const Unlocked unlocked;
    q = at::empty({m, k}, x->options().dtype(at::kChar));
    s = at::empty({m}, x->options().dtype(at::kFloat));
    rc = abi.quantize(q.data_ptr(), s.data_ptr(), x->data_ptr(), m, k, x->stride(0), k, code, stream(device));
  }
  return rc ? failed(rc) : pair_of(std::move(q), std::move(s));
  FAST_END
}

// rows of the norms: contiguous matrices that the results may alias
bool norm_rows(const at::Tensor& x, PyObject* res, const at::Tensor* r, const at::Tensor& w) {
  if (x.dim() != 2 || x.size(0) == 0 || x.size(1) == 0 || x.requires_grad() || !x.is_contiguous() || half_code(x) < 0) return false;
  if (w.scalar_type() != x.scalar_type() || !w.is_contiguous()) return false;
  if (res == Py_None) return true;
  return r && r->scalar_type() == x.scalar_type() && r->sizes() == x.sizes() && !r->requires_grad() && r->is_contiguous();
}

// (X, residual or None, weight, eps) -> (Y, residual or X)
PyObject* norm(PyObject*, PyObject* const* a, Py_ssize_t count) {
  ARGS(4)
  FAST_BEGIN
  const at::Tensor *x = plain(a[0]), *r = a[1] == Py_None ? nullptr : plain(a[1]), *w = plain(a[2]);
  const int device = r ? device_for(abi.norm, {x, w, r}) : device_for(abi.norm, {x, w});
  if (device < 0 || !PyFloat_CheckExact(a[3]) || !norm_rows(*x, a[1], r, *w)) return none();
  const i64 rows = x->size(0), n = x->size(1);
  at::Tensor y;
  int rc;
  {
    const Unlocked unlocked;
    y = at::empty({rows, n}, x->options());
    rc = abi.norm(y.data_ptr(), x->data_ptr(), r ? r->data_ptr() : nullptr, w->data_ptr(), rows, n, n, n, n,
                  (float)PyFloat_AS_DOUBLE(a[3]), half_code(*x), stream(device));
  }
  if (rc) return failed(rc);
  PyObject* out = PyTuple_New(2);
  if (!out) return nullptr;
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(std::move(y)));
  PyTuple_SET_ITEM(out, 1, Py_NewRef(r ? a[1] : a[0]));
  return out;
  FAST_END
}

// (X, residual or None, weight, eps) -> (q, scales)
PyObject* norm_quant(PyObject*, PyObject* const* a, Py_ssize_t count) {
  ARGS(4)
  FAST_BEGIN
  const at::Tensor *x = plain(a[0]), *r = a[1] == Py_None ? nullptr : plain(a[1]), *w = plain(a[2]);
  const int device = r ? device_for(abi.norm_quant, {x, w, r}) : device_for(abi.norm_quant, {x, w});
  if (device < 0 || !PyFloat_CheckExact(a[3]) || !norm_rows(*x, a[1], r, *w)) return none();
  const i64 rows = x->size(0), n = x->size(1);
  if (n % 8 != 0 || n > 16384) return none();
  at::Tensor q, s;
  int rc;
  {
    const Unlocked unlocked;
    q = at::empty({rows, n}, x->options().dtype(at::kChar));
    s = at::empty({rows}, x->options().dtype(at::kFloat));
    rc = abi.norm_quant(q.data_ptr(), s.data_ptr(), x->data_ptr(), r ? r->data_ptr() : nullptr, w->data_ptr(), rows, n, n, n, n,
                        (float)PyFloat_AS_DOUBLE(a[3]), half_code(*x), stream(device));
  }
  return rc ? failed(rc) : pair_of(std::move(q), std::move(s));
  FAST_END
}

// (a, b) -> silu(a) * b
PyObject* swiglu(PyObject*, PyObject* const* a, Py_ssize_t count) {
  ARGS(2)
  FAST_BEGIN
  const at::Tensor *g = plain(a[0]), *u = plain(a[1]);
  const int device = device_for(abi.swiglu, {g, u});
  if (device < 0) return none();
  const int code = g->scalar_type() == at::kFloat ? 2 : half_code(*g);
  if (code < 0 || u->scalar_type() != g->scalar_type() || !matrix(*g) || !matrix(*u) || g->sizes() != u->sizes()) return none();
  const i64 rows = g->size(0), n = g->size(1);
  at::Tensor y;
  int rc;
  {
    const Unlocked unlocked;
    y = at::empty({rows, n}, g->options());
    rc = abi.swiglu(y.data_ptr(), g->data_ptr(), u->data_ptr(), rows, n, g->stride(0), u->stride(0), n, code, stream(device));
  }
  return rc ? failed(rc) : THPVariable_Wrap(std::move(y));
  FAST_END
}

// (addresses of the C functions in the order of `abi`, zeroed_workspace, counters)
PyObject* init(PyObject*, PyObject* const* a, Py_ssize_t count) {
  constexpr Py_ssize_t n = sizeof(abi) / sizeof(void*);
  if (count != n + 2) { PyErr_SetString(PyExc_TypeError, "wrong number of arguments"); return nullptr; }
  for (Py_ssize_t i = 0; i < n; ++i) {
    void* p = PyLong_AsVoidPtr(a[i]);      // 0: not in this library
    if (!p && PyErr_Occurred()) return nullptr;
    reinterpret_cast<void**>(&abi)[i] = p;
  }
  py_zeroed = Py_NewRef(a[n]);
  py_counters = Py_NewRef(a[n + 1]);
  Py_RETURN_NONE;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(init), FAST(w8a16), FAST(w4a16_packed), FAST(linear), FAST(w8a8), FAST(quantize), FAST(norm),
                         FAST(norm_quant), FAST(swiglu), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fast", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__fast() {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "built_for", BUILT_FOR) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
