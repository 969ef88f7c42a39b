// The call path of the operators in native code: argument checks, data pointers, current stream, C ABI call.
//
// Through ctypes an operator call takes 9-12 us of Python (tensor checks one attribute at a time, argument conversion, stream
// lookup), several times what its kernel takes at batch 1: a decoder layer driven operator by operator was bound by that (113 us
// for ten calls; the kernels need about 35). Here a call takes under a microsecond besides the launch.
//
// Each operator is a callable that stands in for the method of the same name in ext.Ops and keeps that method as its fallback.
// It handles the calls whose arguments pass every check the method makes; for anything else - keywords it does not know, wrong
// types, shapes, a launch that was refused - it calls the method with the arguments as they came, which raises the error (or
// takes what only it takes). So there is one definition of every error.
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDAStream.h>

namespace {

constexpr int kMaxArgs = 16;
using Args = PyObject* const*;

struct Tensor {   // a tensor argument: what the checks look at, read once
  const at::Tensor* t = nullptr;
  explicit operator bool() const { return t != nullptr; }
  void* data() const { return t->data_ptr(); }
  int64_t numel() const { return t->numel(); }
  int64_t dim() const { return t->dim(); }
  int64_t size(int i) const { return t->size(i); }
  bool aligned16() const { return (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15u) == 0; }
};

// contiguous CUDA tensor of the type, or empty
Tensor get(PyObject* o, at::ScalarType type) {
  Tensor r;
  if (o && THPVariable_Check(o)) {
    const at::Tensor& t = THPVariable_Unpack(o);
    if (t.is_cuda() && t.scalar_type() == type && t.is_contiguous()) r.t = &t;
  }
  return r;
}
Tensor f16(PyObject* o) { return get(o, at::kHalf); }
Tensor f32(PyObject* o) { return get(o, at::kFloat); }
Tensor i32(PyObject* o) { return get(o, at::kInt); }
Tensor i64(PyObject* o) { return get(o, at::kLong); }

bool integer(PyObject* o, int* v) {
  if (!o || !PyLong_Check(o)) return false;
  int overflow = 0;
  const long long x = PyLong_AsLongLongAndOverflow(o, &overflow);
  if (overflow || x < INT_MIN || x > INT_MAX) return false;
  *v = (int)x;
  return true;
}
bool real(PyObject* o, float* v) {
  if (!o || !PyFloat_Check(o)) return false;
  *v = (float)PyFloat_AS_DOUBLE(o);
  return true;
}
bool flag(PyObject* o, int* v) {   // True or False; absent: False
  *v = o == Py_True;
  return !o || PyBool_Check(o);
}
int log2_exact(int64_t v) { return v > 0 && (v & (v - 1)) == 0 ? 63 - __builtin_clzll((unsigned long long)v) : -1; }
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
bool group_ok(int64_t n_q, int64_t n_kv) {
  if (n_kv <= 0 || n_q % n_kv) return false;
  const int64_t g = n_q / n_kv;
  return g == 1 || g == 2 || g == 4 || g == 8;
}

// An operator's C ABI entry point; it is bound by address, per operator object (the library may be any build of it).
// The call itself runs without the interpreter lock: a launch blocks while the device's queue is full.
template <typename... A>
bool call(void* fn, A... a) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = reinterpret_cast<int (*)(A...)>(fn)(a...);
  Py_END_ALLOW_THREADS
  return rc == 0;
}
#define CHECK(cond) \
  if (!(cond)) return false

bool op_gemv(void* fn, Args a) {   // stage, R, warps, pf, packed, sz, x, y, group
  int stage, R, warps, pf, group;
  CHECK(integer(a[0], &stage) && integer(a[1], &R) && integer(a[2], &warps) && integer(a[3], &pf) && integer(a[8], &group));
  const Tensor w = i32(a[4]), sz = f16(a[5]), x = f16(a[6]), y = f16(a[7]);
  CHECK(w && sz && x && y && w.dim() == 2 && sz.dim() >= 2);
  const int64_t N = w.size(0), K = w.size(1) * 8;
  CHECK(group >= 32 && K % 32 == 0 && K % group == 0 && K <= INT_MAX && N <= INT_MAX);
  CHECK(x.numel() == K && y.numel() == N && sz.size(0) == N && sz.size(1) == K / group && w.aligned16() && x.aligned16());
  const int lg = log2_exact(group);
  CHECK(lg >= 0);
  return call(fn, stage, R, warps, pf, w.data(), sz.data(), x.data(), y.data(), (int)N, (int)K, lg, stream());
}

bool op_tiled(void* fn, Args a) {   // tiled, x, y, N, K, swiglu
  int N, K, sw;
  const Tensor w = get(a[0], at::kByte), x = f16(a[1]), y = f16(a[2]);
  CHECK(w && x && y && integer(a[3], &N) && integer(a[4], &K) && flag(a[5], &sw) && x.numel() == K && y.numel() == N);
  return call(fn, w.data(), x.data(), y.data(), N, K, sw, stream());
}

bool op_tiled_norm(void* fn, Args a) {   // tiled, x_in, delta, norm_w, eps, x_out, y, N, K, swiglu
  int N, K, sw;
  float eps;
  const Tensor w = get(a[0], at::kByte), x = f16(a[1]), nw = f16(a[3]), xo = f16(a[5]), y = f16(a[6]);
  CHECK(w && x && nw && xo && y && real(a[4], &eps) && integer(a[7], &N) && integer(a[8], &K) && flag(a[9], &sw));
  CHECK(x.numel() == K && xo.numel() == K && nw.numel() == K && y.numel() == N);
  void* d = nullptr;
  if (a[2] != Py_None) {
    const Tensor t = f16(a[2]);
    CHECK(t);
    d = t.data();
  }
  return call(fn, w.data(), x.data(), d, nw.data(), eps, xo.data(), y.data(), N, K, sw, stream());
}

bool op_attn(void* fn, Args a) {   // q, kc, vc, bt, pos, part_size, o_part, m_part, l_part, out, version
  int part, version = 2;
  const Tensor q = f16(a[0]), kc = f16(a[1]), vc = f16(a[2]), bt = i32(a[3]), pos = i32(a[4]);
  const Tensor o = f32(a[6]), m = f32(a[7]), l = f32(a[8]), out = f16(a[9]);
  CHECK(q && kc && vc && bt && pos && o && m && l && out && integer(a[5], &part) && (!a[10] || integer(a[10], &version)));
  CHECK(kc.dim() == 4 && kc.size(3) == 64 && vc.t->sizes() == kc.t->sizes() && kc.aligned16() && vc.aligned16());
  const int64_t n_q = q.numel() / 64, n_kv = kc.size(1);
  const int lp = log2_exact(kc.size(2));
  CHECK(group_ok(n_q, n_kv) && part > 0 && version >= 1 && version <= 3 && lp >= 0);
  CHECK(o.dim() > 1 && m.dim() > 1 && l.dim() > 1);
  const int64_t S = o.size(1);
  CHECK(o.size(0) == n_q && m.size(1) == S && l.size(1) == S);
  return call(fn, version, q.data(), kc.data(), vc.data(), bt.data(), pos.data(), (int)n_q, (int)n_kv, lp, part, (int)S, o.data(),
              m.data(), l.data(), out.data(), stream());
}

bool op_attn_b(void* fn, Args a) {   // q, kc, vc, bt, pos, part_size, o_part, m_part, l_part, out, version
  int part, version = 0;
  const Tensor q = f16(a[0]), kc = f16(a[1]), vc = f16(a[2]), bt = i32(a[3]), pos = i32(a[4]);
  const Tensor o = f32(a[6]), m = f32(a[7]), l = f32(a[8]), out = f16(a[9]);
  CHECK(q && kc && vc && bt && pos && o && m && l && out && integer(a[5], &part) && (!a[10] || integer(a[10], &version)));
  CHECK(q.dim() == 3 && kc.dim() == 4 && vc.t->sizes() == kc.t->sizes() && kc.aligned16() && vc.aligned16());
  const int64_t B = q.size(0), n_q = q.size(1), D = q.size(2);
  const int lp = log2_exact(kc.size(2));
  CHECK(kc.size(3) == D && bt.dim() == 2 && bt.size(0) == B && pos.numel() == B && lp >= 0);
  CHECK(o.dim() == 4 && m.dim() == 3 && m.t->sizes() == l.t->sizes());
  const int64_t S = o.size(2);
  CHECK(o.size(0) == B && o.size(1) == n_q && o.size(3) == D && m.size(0) == B && m.size(1) == n_q && m.size(2) == S);
  return call(fn, version, q.data(), kc.data(), vc.data(), bt.data(), (int)bt.size(1), pos.data(), (int)B, (int)n_q,
              (int)kc.size(1), (int)D, lp, part, (int)S, o.data(), m.data(), l.data(), out.data(), stream());
}

bool op_rope_attn(void* fn, Args a) {   // qkv, cos_t, sin_t, pos, bt, kc, vc, n_q, n_kv, part_size, o_part, m_part, l_part, out, arrive
  int n_q, n_kv, part;
  const Tensor qkv = f16(a[0]), cs = f32(a[1]), sn = f32(a[2]), pos = i32(a[3]), bt = i32(a[4]), kc = f16(a[5]), vc = f16(a[6]);
  const Tensor o = f32(a[10]), m = f32(a[11]), l = f32(a[12]), out = f16(a[13]);
  CHECK(qkv && cs && sn && pos && bt && kc && vc && o && m && l && out);
  CHECK(integer(a[7], &n_q) && integer(a[8], &n_kv) && integer(a[9], &part) && kc.dim() == 4 && vc.t->sizes() == kc.t->sizes());
  const int64_t D = kc.size(3);
  const int lp = log2_exact(kc.size(2));
  CHECK(qkv.numel() == (n_q + 2 * (int64_t)n_kv) * D && kc.size(1) == n_kv && lp >= 0 && o.dim() == 3 && m.dim() == 2);
  const int64_t S = o.size(1);
  CHECK(o.size(0) == n_q && o.size(2) == D && m.size(0) == n_q && m.size(1) == S && m.t->sizes() == l.t->sizes());
  void* arrive = nullptr;
  if (a[14] && a[14] != Py_None) {
    const Tensor t = i32(a[14]);
    CHECK(t && t.numel() >= n_kv);
    arrive = t.data();
  }
  return call(fn, qkv.data(), cs.data(), sn.data(), kc.data(), vc.data(), bt.data(), pos.data(), n_q, n_kv, (int)D, lp, part,
              (int)S, o.data(), m.data(), l.data(), out.data(), arrive, stream());
}

bool op_norm(void* fn, Args a) {   // x, delta, w, out, eps
  float eps;
  const Tensor x = f16(a[0]), w = f16(a[2]), out = f16(a[3]);
  CHECK(x && w && out && real(a[4], &eps) && x.numel() % 8 == 0 && x.aligned16() && w.aligned16() && out.aligned16());
  void* d = nullptr;
  if (a[1] != Py_None) {
    const Tensor t = f16(a[1]);
    CHECK(t && t.aligned16());
    d = t.data();
  }
  return call(fn, x.data(), d, w.data(), out.data(), (int)x.numel(), eps, stream());
}

bool op_swiglu(void* fn, Args a) {   // gu, out
  const Tensor gu = f16(a[0]), out = f16(a[1]);
  CHECK(gu && out && out.numel() % 8 == 0 && gu.numel() == 2 * out.numel() && gu.aligned16() && out.aligned16());
  return call(fn, gu.data(), out.data(), (int)out.numel(), stream());
}

bool op_rope(void* fn, Args a) {   // qkv, cos_t, sin_t, pos, bt, kc, vc, n_q, n_kv
  int n_q, n_kv;
  const Tensor qkv = f16(a[0]), cs = f32(a[1]), sn = f32(a[2]), pos = i32(a[3]), bt = i32(a[4]), kc = f16(a[5]), vc = f16(a[6]);
  CHECK(qkv && cs && sn && pos && bt && kc && vc && integer(a[7], &n_q) && integer(a[8], &n_kv) && kc.dim() > 2 && cs.dim() > 1);
  const int lp = log2_exact(kc.size(2));
  CHECK(qkv.numel() == (n_q + 2 * (int64_t)n_kv) * 64 && cs.size(1) == 32 && lp >= 0);
  return call(fn, qkv.data(), cs.data(), sn.data(), pos.data(), bt.data(), kc.data(), vc.data(), n_q, n_kv, lp, stream());
}

bool op_rope_b(void* fn, Args a) {   // the same for rows qkv [B, (n_q + 2 n_kv) D], bt [B, max_pages]
  int n_q, n_kv;
  const Tensor qkv = f16(a[0]), cs = f32(a[1]), sn = f32(a[2]), pos = i32(a[3]), bt = i32(a[4]), kc = f16(a[5]), vc = f16(a[6]);
  CHECK(qkv && cs && sn && pos && bt && kc && vc && integer(a[7], &n_q) && integer(a[8], &n_kv));
  CHECK(qkv.dim() == 2 && cs.dim() > 1 && kc.dim() == 4 && bt.dim() == 2);
  const int64_t B = qkv.size(0), D = 2 * cs.size(1);
  const int lp = log2_exact(kc.size(2));
  CHECK(qkv.size(1) == (n_q + 2 * (int64_t)n_kv) * D && kc.size(3) == D && bt.size(0) == B && lp >= 0);
  return call(fn, qkv.data(), cs.data(), sn.data(), pos.data(), bt.data(), (int)bt.size(1), kc.data(), vc.data(), (int)B, n_q, n_kv,
              (int)D, lp, stream());
}

bool op_embed(void* fn, Args a) {   // emb, tok, x
  const Tensor emb = f16(a[0]), tok = i64(a[1]), x = f16(a[2]);
  CHECK(emb && tok && x && emb.dim() == 2 && emb.size(1) == x.numel());
  return call(fn, emb.data(), tok.data(), x.data(), (int)x.numel(), (int)emb.size(0), stream());
}

bool op_argmax(void* fn, Args a) {   // logits, tok, pos, history
  const Tensor lg = f16(a[0]), tok = i64(a[1]);
  CHECK(lg && tok);
  void *p = nullptr, *h = nullptr;
  if (a[2] && a[2] != Py_None) {
    const Tensor t = i32(a[2]);
    CHECK(t);
    p = t.data();
  }
  if (a[3] && a[3] != Py_None) {
    const Tensor t = i64(a[3]);
    CHECK(t);
    h = t.data();
  }
  return call(fn, lg.data(), (int)lg.numel(), tok.data(), p, h, stream());
}

struct OpDef {
  const char* name;
  bool (*fn)(void*, Args);
  const char* entry;   // the C function
  int required, total;
  const char* args[kMaxArgs];
};
const OpDef kOps[] = {
    {"gemv_w4a16", op_gemv, "b200_gemv_w4a16", 9, 9, {"stage", "R", "warps", "pf", "packed", "sz", "x", "y", "group"}},
    {"gemv_w4a16_tiled", op_tiled, "b200_gemv_w4a16_tiled", 5, 6, {"tiled", "x", "y", "N", "K", "swiglu"}},
    {"gemv_w4a16_tiled_norm", op_tiled_norm, "b200_gemv_w4a16_tiled_norm", 9, 10, {"tiled", "x_in", "delta", "norm_w", "eps", "x_out", "y", "N", "K", "swiglu"}},
    {"paged_attention", op_attn, "b200_paged_attention", 10, 11,
     {"q", "kc", "vc", "bt", "pos", "part_size", "o_part", "m_part", "l_part", "out", "version"}},
    {"paged_attention_batched", op_attn_b, "b200_paged_attention_batched_v", 10, 11,
     {"q", "kc", "vc", "bt", "pos", "part_size", "o_part", "m_part", "l_part", "out", "version"}},
    {"rope_paged_attention", op_rope_attn, "b200_rope_paged_attention", 14, 15,
     {"qkv", "cos_t", "sin_t", "pos", "bt", "kc", "vc", "n_q", "n_kv", "part_size", "o_part", "m_part", "l_part", "out", "arrive"}},
    {"add_rmsnorm", op_norm, "b200_add_rmsnorm", 5, 5, {"x", "delta", "w", "out", "eps"}},
    {"swiglu", op_swiglu, "b200_swiglu", 2, 2, {"gu", "out"}},
    {"rope_append", op_rope, "b200_rope_append", 9, 9, {"qkv", "cos_t", "sin_t", "pos", "bt", "kc", "vc", "n_q", "n_kv"}},
    {"rope_append_batched", op_rope_b, "b200_rope_append_batched", 9, 9, {"qkv", "cos_t", "sin_t", "pos", "bt", "kc", "vc", "n_q", "n_kv"}},
    {"embed_row", op_embed, "b200_embed_row", 3, 3, {"emb", "tok", "x"}},
    {"argmax", op_argmax, "b200_argmax", 2, 4, {"logits", "tok", "pos", "history"}},
};

struct OpObject {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  const OpDef* op;
  void* entry;
  PyObject* fallback;
};

PyObject* op_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  OpObject* o = reinterpret_cast<OpObject*>(self);
  const OpDef& op = *o->op;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf), nk = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
  PyObject* a[kMaxArgs] = {};
  bool ok = n <= op.total;
  for (Py_ssize_t i = 0; ok && i < n; ++i) a[i] = args[i];
  for (Py_ssize_t k = 0; ok && k < nk; ++k) {
    int at = -1;
    for (int i = 0; i < op.total && at < 0; ++i)
      if (PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, k), op.args[i]) == 0) at = i;
    ok = at >= 0 && !a[at];
    if (ok) a[at] = args[n + k];
  }
  for (int i = 0; ok && i < op.required; ++i) ok = a[i] != nullptr;
  try {
    if (ok && op.fn(o->entry, a)) Py_RETURN_NONE;
  } catch (const std::exception&) {   // a tensor without storage and the like: the method says what is wrong
  }
  return PyObject_Vectorcall(o->fallback, args, nargsf & ~PY_VECTORCALL_ARGUMENTS_OFFSET, kwnames);
}

void op_dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  Py_CLEAR(reinterpret_cast<OpObject*>(self)->fallback);
  Py_TYPE(self)->tp_free(self);
}
int op_traverse(PyObject* self, visitproc visit, void* arg) {
  Py_VISIT(reinterpret_cast<OpObject*>(self)->fallback);
  return 0;
}
int op_clear(PyObject* self) {
  Py_CLEAR(reinterpret_cast<OpObject*>(self)->fallback);
  return 0;
}
PyObject* op_doc(PyObject* self, void*) { return PyObject_GetAttrString(reinterpret_cast<OpObject*>(self)->fallback, "__doc__"); }
PyObject* op_wrapped(PyObject* self, void*) { return Py_NewRef(reinterpret_cast<OpObject*>(self)->fallback); }   // inspect.signature follows it
PyGetSetDef op_getset[] = {{"__doc__", op_doc, nullptr, nullptr, nullptr}, {"__wrapped__", op_wrapped, nullptr, nullptr, nullptr}, {}};

PyTypeObject OpType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// operator(name, address of its C function, fallback): the callable
PyObject* make_operator(PyObject*, PyObject* args) {
  const char* name;
  PyObject *address, *fallback;
  if (!PyArg_ParseTuple(args, "sOO", &name, &address, &fallback)) return nullptr;
  void* entry = PyLong_AsVoidPtr(address);
  if (!entry) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "%s: null address", name);
  for (const OpDef& d : kOps)
    if (strcmp(d.name, name) == 0) {
      OpObject* o = PyObject_GC_New(OpObject, &OpType);
      if (!o) return nullptr;
      o->vectorcall = op_call;
      o->op = &d;
      o->entry = entry;
      o->fallback = Py_NewRef(fallback);
      PyObject_GC_Track(o);
      return reinterpret_cast<PyObject*>(o);
    }
  return PyErr_Format(PyExc_KeyError, "%s", name);
}

PyObject* entries(PyObject*, PyObject*) {   // {operator: its C function}
  PyObject* o = PyDict_New();
  for (const OpDef& d : kOps) {
    PyObject* v = PyUnicode_FromString(d.entry);
    PyDict_SetItemString(o, d.name, v);
    Py_DECREF(v);
  }
  return o;
}
PyObject* names(PyObject*, PyObject*) {   // (C functions, {operator: (argument names, how many are required)})
  PyObject *f = PyList_New(0), *o = PyDict_New();
  for (const OpDef& d : kOps) {
    PyObject* s = PyUnicode_FromString(d.entry);
    PyList_Append(f, s);
    Py_DECREF(s);
    PyObject* args = PyTuple_New(d.total);
    for (int i = 0; i < d.total; ++i) PyTuple_SET_ITEM(args, i, PyUnicode_FromString(d.args[i]));
    PyObject* v = Py_BuildValue("(Ni)", args, d.required);
    PyDict_SetItemString(o, d.name, v);
    Py_DECREF(v);
  }
  return Py_BuildValue("(NN)", f, o);
}

PyMethodDef methods[] = {{"operator", make_operator, METH_VARARGS, nullptr}, {"entries", entries, METH_NOARGS, nullptr},
                         {"names", names, METH_NOARGS, nullptr}, {}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  OpType.tp_name = "llm_decode_kernels_b200._host.operator";
  OpType.tp_basicsize = sizeof(OpObject);
  OpType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_HAVE_GC;
  OpType.tp_vectorcall_offset = offsetof(OpObject, vectorcall);
  OpType.tp_call = PyVectorcall_Call;
  OpType.tp_dealloc = op_dealloc;
  OpType.tp_traverse = op_traverse;
  OpType.tp_clear = op_clear;
  OpType.tp_getset = op_getset;
  if (PyType_Ready(&OpType) < 0) return nullptr;
  return PyModule_Create(&module);
}
