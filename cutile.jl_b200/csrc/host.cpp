// Native call path of the Python package: one C function per entry point takes the tensors as they are, checks the
// ordinary form of the call (CUDA tensors of the expected types and shapes, no launch keywords) and enqueues it through
// the C ABI.
//
// What bounds the small calls is the host: in Python a softmax of 64 x 1000 elements spent about 9 us on reading
// shapes, strides, pointers and the current stream (torch.cuda.current_stream 1.2 us, a shape or stride 0.1-0.3 us) and
// on the ctypes conversion of 11 arguments (1.2 us), against 2.4-3.1 us for the launch itself.  The same through this
// file takes about 0.3 us on top of the launch.
//
// Every function returns None when a call is not of the ordinary form; the Python wrapper then runs its full argument
// checks, which either raise the precise error or make the call themselves.  A status other than CTB_OK raises CtbError
// (through the Python function installed by setup()).
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>

#include "../../include/cutile_b200.h"

namespace {

constexpr int kMaxDevices = 64;
ctb_ctx* g_ctx[kMaxDevices] = {};  // written under the GIL
PyObject* g_context = nullptr;     // _lib.context(device) -> c_void_p
PyObject* g_check = nullptr;       // _lib.check(status): raises CtbError

using at::Tensor;

const Tensor* cuda_tensor(PyObject* o) {
  if (!THPVariable_Check(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided ? &t : nullptr;
}

struct Call {  // device, context and current stream of a call; ok() is false with a Python error set
  ctb_ctx* ctx = nullptr;
  void* stream = nullptr;
  explicit Call(const Tensor& t) {
    const int dev = t.get_device();
    if (dev < 0 || dev >= kMaxDevices) return;
    if (!g_ctx[dev]) {
      PyObject* h = PyObject_CallFunction(g_context, "i", dev);
      PyObject* v = h ? PyObject_GetAttrString(h, "value") : nullptr;
      if (v) g_ctx[dev] = static_cast<ctb_ctx*>(PyLong_AsVoidPtr(v));
      Py_XDECREF(v);
      Py_XDECREF(h);
      if (!g_ctx[dev] && !PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "cutile_b200: no context");
    }
    ctx = g_ctx[dev];
    if (ctx) stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream();
  }
  bool ok() const { return ctx != nullptr; }
};

// Py_None ("not the ordinary form") and the result of a call with status s
PyObject* decline() { Py_RETURN_NONE; }
PyObject* done(int s, PyObject* result_owned) {
  if (s == CTB_OK) return result_owned;
  Py_XDECREF(result_owned);
  PyObject* r = PyObject_CallFunction(g_check, "i", s);  // raises
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "cutile_b200: call failed");
  return nullptr;
}
PyObject* yes() { Py_RETURN_TRUE; }

template <class F>
int without_gil(F f) {
  struct Release {  // the lock is taken again also when f throws: data_ptr() does for a tensor without storage (vmap, fake)
    PyThreadState* state = PyEval_SaveThread();
    ~Release() { PyEval_RestoreThread(state); }
  } release;
  return f();
}

bool as_int(PyObject* o, long long* v) {
  if (!PyLong_Check(o)) return false;
  int over = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &over);
  return over == 0 && *v >= INT32_MIN && *v <= INT32_MAX;
}
bool ints(PyObject* const* a, int n, long long* v) {
  for (int i = 0; i < n; ++i)
    if (!as_int(a[i], v + i)) return false;
  return true;
}
bool as_float(PyObject* o, float* v) {
  if (!PyFloat_Check(o)) return false;
  *v = (float)PyFloat_AS_DOUBLE(o);
  return true;
}
int dtype_of(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return CTB_F32;
    case at::kHalf: return CTB_F16;
    case at::kBFloat16: return CTB_BF16;
    default: return -1;
  }
}
// 2-D with contiguous rows -> leading dimension
bool rows(const Tensor& t, int64_t* ld, int64_t* m, int64_t* n) {
  if (t.dim() != 2) return false;
  *m = t.size(0);
  *n = t.size(1);
  if (*n > 1 && t.stride(1) != 1) return false;
  *ld = *m > 1 ? t.stride(0) : std::max<int64_t>(*n, t.stride(0));
  return true;
}
bool vec_f32(const Tensor* t, int64_t n) { return t && t->scalar_type() == at::kFloat && t->numel() == n && t->is_contiguous(); }

// softmax(output, input, variant, tile)
PyObject* softmax(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor *out, *in;
  long long v[2];
  int64_t ldo, mo, no, ldi, m, k;
  if (n != 4 || !(out = cuda_tensor(a[0])) || !(in = cuda_tensor(a[1])) || !ints(a + 2, 2, v) || !rows(*out, &ldo, &mo, &no) ||
      !rows(*in, &ldi, &m, &k) || mo != m || no != k || out->scalar_type() != in->scalar_type() || dtype_of(*in) < 0)
    return decline();
  Call c(*in);
  if (!c.ok()) return nullptr;
  const int s = without_gil([&] {
    return ctb_softmax(c.ctx, c.stream, out->data_ptr(), in->data_ptr(), k, m, ldo, ldi, (int)v[0], (int)v[1], dtype_of(*in));
  });
  return done(s, yes());
}

// vadd(a, b, c, tile_x, tile_y, gather, dims): dims = 1: dense 1-D arrays; 2: 2-D arrays with contiguous rows
PyObject* vadd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor* t[3];
  long long v[4];
  if (n != 7 || !ints(a + 3, 4, v)) return decline();
  int64_t ld[3], m = 1, k = 0;
  for (int i = 0; i < 3; ++i) {
    if (!(t[i] = cuda_tensor(a[i])) || t[i]->scalar_type() != t[0]->scalar_type() || t[i]->sizes() != t[0]->sizes() ||
        t[i]->dim() != v[3])
      return decline();
    if (v[3] == 1) {
      if (!t[i]->is_contiguous()) return decline();
      k = ld[i] = t[i]->numel();
    } else if (!rows(*t[i], ld + i, &m, &k)) {
      return decline();
    }
  }
  const int dt = dtype_of(*t[0]);
  if (dt < 0) return decline();
  Call c(*t[0]);
  if (!c.ok()) return nullptr;
  const int s = without_gil([&] {
    return ctb_vadd(c.ctx, c.stream, t[0]->data_ptr(), t[1]->data_ptr(), t[2]->data_ptr(), k, m, ld[0], ld[1], ld[2], (int)v[0],
                    (int)v[1], (int)v[2], dt);
  });
  return done(s, yes());
}

// transpose(x, y, tm, tn)
PyObject* transpose(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor *x, *y;
  long long v[2];
  int64_t ldx, N, M, ldy, My, Ny;
  if (n != 4 || !(x = cuda_tensor(a[0])) || !(y = cuda_tensor(a[1])) || !ints(a + 2, 2, v) || !rows(*x, &ldx, &N, &M) ||
      !rows(*y, &ldy, &My, &Ny) || My != M || Ny != N || x->scalar_type() != y->scalar_type() || dtype_of(*x) < 0)
    return decline();
  Call c(*x);
  if (!c.ok()) return nullptr;
  const int s = without_gil([&] {
    return ctb_transpose(c.ctx, c.stream, x->data_ptr(), y->data_ptr(), M, N, ldx, ldy, (int)v[0], (int)v[1], dtype_of(*x));
  });
  return done(s, yes());
}

// layernorm_fwd(X, W, B, Y, Mean, Rstd, eps, tile)
PyObject* layernorm_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor* t[6];
  if (n != 8) return decline();
  for (int i = 0; i < 6; ++i)
    if (!(t[i] = cuda_tensor(a[i]))) return decline();
  int64_t ldx, M, N, ldy, My, Ny;
  float eps;
  long long tile;
  if (t[0]->scalar_type() != at::kFloat || t[3]->scalar_type() != at::kFloat || !rows(*t[0], &ldx, &M, &N) ||
      !rows(*t[3], &ldy, &My, &Ny) || My != M || Ny != N || !vec_f32(t[1], N) || !vec_f32(t[2], N) || !vec_f32(t[4], M) ||
      !vec_f32(t[5], M) || !as_float(a[6], &eps) || !as_int(a[7], &tile))
    return decline();
  Call c(*t[0]);
  if (!c.ok()) return nullptr;
  auto p = [&](int i) { return static_cast<float*>(t[i]->data_ptr()); };
  const int s = without_gil([&] {
    return ctb_layernorm_fwd(c.ctx, c.stream, p(0), p(1), p(2), p(3), p(4), p(5), N, M, ldx, ldy, eps, (int)tile);
  });
  return done(s, yes());
}

// layernorm_bwd(DX, DY, DW, DB, X, W, Mean, Rstd, group_size_m, tile)
PyObject* layernorm_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor* t[8];
  if (n != 10) return decline();
  for (int i = 0; i < 8; ++i)
    if (!(t[i] = cuda_tensor(a[i])) || t[i]->scalar_type() != at::kFloat) return decline();
  int64_t ld[3], M, N, m, k;
  long long v[2];
  if (!ints(a + 8, 2, v) || !rows(*t[4], ld, &M, &N) || !rows(*t[1], ld + 1, &m, &k) || m != M || k != N ||
      !rows(*t[0], ld + 2, &m, &k) || m != M || k != N || !vec_f32(t[5], N) || !vec_f32(t[6], M) || !vec_f32(t[7], M))
    return decline();
  for (int i = 2; i < 4; ++i)
    if (t[i]->dim() != 2 || t[i]->size(0) != v[0] || t[i]->size(1) != N || !t[i]->is_contiguous()) return decline();
  Call c(*t[4]);
  if (!c.ok()) return nullptr;
  auto p = [&](int i) { return static_cast<float*>(t[i]->data_ptr()); };
  const int s = without_gil([&] {
    return ctb_layernorm_bwd_dx_partial_dwdb(c.ctx, c.stream, p(0), p(1), p(2), p(3), p(4), p(5), p(6), p(7), nullptr, N, M,
                                             ld[0], ld[1], ld[2], (int)v[0], (int)v[1]);
  });
  return done(s, yes());
}

// layernorm_dwdb(DW, DB, FINAL_DW, FINAL_DB, tile_m, tile_n)
PyObject* layernorm_dwdb(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor* t[4];
  long long v[2];
  if (n != 6 || !ints(a + 4, 2, v)) return decline();
  for (int i = 0; i < 4; ++i)
    if (!(t[i] = cuda_tensor(a[i])) || t[i]->scalar_type() != at::kFloat || !t[i]->is_contiguous()) return decline();
  if (t[0]->dim() != 2 || t[1]->sizes() != t[0]->sizes()) return decline();
  const int64_t G = t[0]->size(0), N = t[0]->size(1);
  if (t[2]->numel() != N || t[3]->numel() != N) return decline();
  Call c(*t[0]);
  if (!c.ok()) return nullptr;
  auto p = [&](int i) { return static_cast<float*>(t[i]->data_ptr()); };
  const int s = without_gil([&] {
    return ctb_layernorm_bwd_dwdb(c.ctx, c.stream, p(0), p(1), p(2), p(3), N, (int)G, (int)v[0], (int)v[1]);
  });
  return done(s, yes());
}

// matmul(A, B, C, tm, tn, tk): A [K, M], B [N, K], C [N, M]
PyObject* matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor* t[3];
  long long v[3];
  if (n != 6 || !ints(a + 3, 3, v)) return decline();
  int64_t ld[3], d0[3], d1[3];
  for (int i = 0; i < 3; ++i)
    if (!(t[i] = cuda_tensor(a[i])) || t[i]->scalar_type() != t[0]->scalar_type() || !rows(*t[i], ld + i, d0 + i, d1 + i))
      return decline();
  const int dt = dtype_of(*t[0]);
  const int64_t K = d0[0], M = d1[0], N = d0[1];
  if (dt < 0 || d1[1] != K || d0[2] != N || d1[2] != M) return decline();
  Call c(*t[0]);
  if (!c.ok()) return nullptr;
  const int s = without_gil([&] {
    return ctb_gemm(c.ctx, c.stream, t[0]->data_ptr(), t[1]->data_ptr(), t[2]->data_ptr(), M, N, K, ld[0], ld[1], ld[2], dt,
                    (int)v[0], (int)v[1], (int)v[2]);
  });
  return done(s, yes());
}

// batch_matmul(A, B, C, tm, tn, tk): A [batch, K, M], B [batch, N, K], C [batch, N, M]
PyObject* batch_matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor* t[3];
  long long v[3];
  if (n != 6 || !ints(a + 3, 3, v)) return decline();
  for (int i = 0; i < 3; ++i)
    if (!(t[i] = cuda_tensor(a[i])) || t[i]->scalar_type() != t[0]->scalar_type() || t[i]->dim() != 3 || t[i]->stride(2) != 1)
      return decline();
  const int dt = dtype_of(*t[0]);
  const int64_t nb = t[0]->size(0), K = t[0]->size(1), M = t[0]->size(2), N = t[1]->size(1);
  if (dt < 0 || t[1]->size(0) != nb || t[2]->size(0) != nb || t[1]->size(2) != K || t[2]->size(1) != N || t[2]->size(2) != M)
    return decline();
  Call c(*t[0]);
  if (!c.ok()) return nullptr;
  const int s = without_gil([&] {
    return ctb_gemm_batched(c.ctx, c.stream, t[0]->data_ptr(), t[1]->data_ptr(), t[2]->data_ptr(), M, N, K, nb, t[0]->stride(1),
                            t[1]->stride(1), t[2]->stride(1), t[0]->stride(0), t[1]->stride(0), t[2]->stride(0), dt, (int)v[0],
                            (int)v[1], (int)v[2]);
  });
  return done(s, yes());
}

// fmha(Q, K, V, Out or None, qk_scale or None, input_pos, tile_m, tile_n, group, causal) -> Out
PyObject* fmha(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor* t[3];
  long long v[4];
  if (n != 10 || !ints(a + 5, 4, v) || !PyBool_Check(a[9])) return decline();
  for (int i = 0; i < 3; ++i)
    if (!(t[i] = cuda_tensor(a[i])) || t[i]->dim() != 4 || !t[i]->is_contiguous() || t[i]->scalar_type() != t[0]->scalar_type())
      return decline();
  const Tensor &Q = *t[0], &K = *t[1], &V = *t[2];
  const int dt = dtype_of(Q);
  const int64_t B = Q.size(0), H = Q.size(1), Sq = Q.size(2), D = Q.size(3), KVH = K.size(1), Skv = K.size(2), Dv = V.size(3);
  if (dt < 0 || K.size(0) != B || K.size(3) != D || V.size(0) != B || V.size(1) != KVH || V.size(2) != Skv || D <= 0)
    return decline();
  float scale;
  if (a[4] == Py_None) scale = (float)(1.0 / std::sqrt((double)D));
  else if (!as_float(a[4], &scale)) return decline();
  const bool causal = a[9] == Py_True;
  Call c(Q);
  if (!c.ok()) return nullptr;
  Tensor made;
  const Tensor* out;
  if (a[3] == Py_None) {
    made = at::empty({B, H, Sq, Dv}, Q.options());
    out = &made;
  } else {
    if (!(out = cuda_tensor(a[3])) || out->scalar_type() != Q.scalar_type() || out->dim() != 4 || !out->is_contiguous() ||
        out->size(0) != B || out->size(1) != H || out->size(2) != Sq || out->size(3) != Dv)
      return decline();
  }
  const int s = without_gil([&] {
    return ctb_fmha_fwd(c.ctx, c.stream, Q.data_ptr(), K.data_ptr(), V.data_ptr(), out->data_ptr(), D, Dv, Sq, Skv, H, KVH, B,
                        scale, (int32_t)v[0], (int)v[1], (int)v[2], (int)v[3], causal ? 1 : 0, dt);
  });
  if (s != CTB_OK || a[3] != Py_None) return done(s, s == CTB_OK ? Py_NewRef(a[3]) : nullptr);
  return THPVariable_Wrap(std::move(made));
}

// moe_router(hidden, W_r, topk) -> (gates [topk, T] f16, ids [topk, T] int32)
PyObject* moe_router(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor *x, *w;
  long long topk;
  if (n != 3 || !(x = cuda_tensor(a[0])) || !(w = cuda_tensor(a[1])) || !as_int(a[2], &topk) || x->dim() != 2 || w->dim() != 2 ||
      x->scalar_type() != at::kHalf || w->scalar_type() != at::kHalf || !x->is_contiguous() || !w->is_contiguous() ||
      x->size(1) != w->size(1) || topk < 1)
    return decline();
  const int64_t T = x->size(0), H = x->size(1), E = w->size(0);
  Call c(*x);
  if (!c.ok()) return nullptr;
  Tensor ids = at::empty({topk, T}, x->options().dtype(at::kInt)), gates = at::empty({topk, T}, x->options());
  const int s = without_gil([&] {
    return ctb_moe_router(c.ctx, c.stream, x->data_ptr(), w->data_ptr(), static_cast<int32_t*>(ids.data_ptr()), gates.data_ptr(),
                          nullptr, T, H, E, (int)topk);
  });
  if (s != CTB_OK) return done(s, nullptr);
  PyObject* g = THPVariable_Wrap(std::move(gates));
  PyObject* i = g ? THPVariable_Wrap(std::move(ids)) : nullptr;
  PyObject* r = i ? PyTuple_Pack(2, g, i) : nullptr;
  Py_XDECREF(g);
  Py_XDECREF(i);
  return r;
}

// moe_ffn(hidden, w1, w2, gates, ids, tile_m, tile_n, tile_k) -> out [T, H] f16
PyObject* moe_ffn(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor* t[5];
  long long v[3];
  if (n != 8 || !ints(a + 5, 3, v)) return decline();
  for (int i = 0; i < 5; ++i)
    if (!(t[i] = cuda_tensor(a[i])) || !t[i]->is_contiguous() || (i < 4 && t[i]->scalar_type() != at::kHalf)) return decline();
  const Tensor &x = *t[0], &w1 = *t[1], &w2 = *t[2], &g = *t[3], &ids = *t[4];
  const int bits = ids.scalar_type() == at::kInt ? 32 : ids.scalar_type() == at::kLong ? 64 : 0;
  if (!bits || x.dim() != 2 || w1.dim() != 3 || w2.dim() != 3 || g.dim() != 2 || ids.dim() != 2) return decline();
  const int64_t T = x.size(0), H = x.size(1), E = w2.size(0), I = w2.size(2), topk = ids.size(0);
  if (w2.size(1) != H || w1.size(0) != E || w1.size(1) != 2 * I || w1.size(2) != H || ids.size(1) != T || g.size(0) != topk ||
      g.size(1) != T)
    return decline();
  Call c(x);
  if (!c.ok()) return nullptr;
  Tensor out = at::empty({T, H}, x.options());
  const int s = without_gil([&] {
    return ctb_moe_ffn(c.ctx, c.stream, x.data_ptr(), w1.data_ptr(), w2.data_ptr(), g.data_ptr(), ids.data_ptr(), bits,
                       out.data_ptr(), T, H, I, E, topk, (int)v[0], (int)v[1], (int)v[2]);
  });
  if (s != CTB_OK) return done(s, nullptr);
  return THPVariable_Wrap(std::move(out));
}

// ---- host-level array expressions ---------------------------------------------------------------------------------
// Expr and Tiled of the Python module `tiled` are the types below.  A fused expression is built of ten to twenty nodes
// per call; as Python classes a node cost 0.5-0.8 us (constructor, isinstance tests) and the walk that turns the tree
// into a program about 20 us, more than the kernel of an ordinary array.  As C types a node costs about 0.1 us and the
// walk about 1 us.
struct Node {
  PyObject_HEAD
  PyObject* node;    // ("leaf", tensor) | ("const", float) | (unary name, Expr) | (binary name, Expr, Expr)
  PyObject* tensor;  // Tiled only
  PyObject *dict, *weak;
};
PyTypeObject* g_expr = nullptr;
PyTypeObject* g_tiled = nullptr;
PyObject* g_leaf_error = nullptr;  // tiled._leaf_error(tensor): raises what is wrong with a leaf, or returns None
struct OpName { const char* name; int code; PyObject* str; };
OpName g_ops[] = {{"leaf", CTB_TILED_INPUT, nullptr}, {"const", CTB_TILED_CONST, nullptr}, {"identity", CTB_TILED_IDENTITY, nullptr},
                  {"neg", CTB_TILED_NEG, nullptr}, {"abs", CTB_TILED_ABS, nullptr}, {"sqrt", CTB_TILED_SQRT, nullptr},
                  {"exp", CTB_TILED_EXP, nullptr}, {"exp2", CTB_TILED_EXP2, nullptr}, {"log", CTB_TILED_LOG, nullptr},
                  {"log2", CTB_TILED_LOG2, nullptr}, {"sin", CTB_TILED_SIN, nullptr}, {"cos", CTB_TILED_COS, nullptr},
                  {"tanh", CTB_TILED_TANH, nullptr}, {"inv", CTB_TILED_INV, nullptr}, {"abs2", CTB_TILED_ABS2, nullptr},
                  {"add", CTB_TILED_ADD, nullptr}, {"sub", CTB_TILED_SUB, nullptr}, {"mul", CTB_TILED_MUL, nullptr},
                  {"div", CTB_TILED_DIV, nullptr}, {"max", CTB_TILED_MAX, nullptr}, {"min", CTB_TILED_MIN, nullptr},
                  {"pow", CTB_TILED_POW, nullptr}};
PyObject* op_str(int code) {
  for (auto& o : g_ops)
    if (o.code == code) return o.str;
  return nullptr;
}
int op_code(PyObject* name) {  // -1: not an operation
  for (auto& o : g_ops)
    if (o.str == name) return o.code;
  for (auto& o : g_ops)
    if (PyUnicode_Check(name) && PyUnicode_Compare(o.str, name) == 0) return o.code;
  return -1;
}

bool is_expr(PyObject* o) { return PyObject_TypeCheck(o, g_expr); }

PyObject* new_node(PyTypeObject* type, PyObject* tuple_owned, PyObject* tensor) {
  if (!tuple_owned) return nullptr;
  Node* n = reinterpret_cast<Node*>(type->tp_alloc(type, 0));
  if (!n) {
    Py_DECREF(tuple_owned);
    return nullptr;
  }
  n->node = tuple_owned;
  n->tensor = Py_XNewRef(tensor);
  return reinterpret_cast<PyObject*>(n);
}

int leaf_ok(PyObject* t) {  // 0 with a Python error set when the tensor cannot be a leaf
  try {
    const Tensor* c = cuda_tensor(t);
    if (c && c->dim() <= 3 && c->is_contiguous()) return 1;
  } catch (const std::exception& e) {  // type slots call this too: nothing may pass them
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return 0;
  }
  PyObject* r = PyObject_CallFunctionObjArgs(g_leaf_error, t, nullptr);
  Py_XDECREF(r);
  return r != nullptr;
}
PyObject* make_leaf(PyObject* t) {
  if (!leaf_ok(t)) return nullptr;
  return new_node(g_tiled, PyTuple_Pack(2, op_str(CTB_TILED_INPUT), t), t);
}

PyObject* wrap(PyObject* x) {  // new reference
  if (is_expr(x)) return Py_NewRef(x);
  if (THPVariable_Check(x)) return make_leaf(x);
  if (PyFloat_Check(x) || PyLong_Check(x)) {
    PyObject* f = PyNumber_Float(x);
    if (!f) return nullptr;
    PyObject* r = new_node(g_expr, PyTuple_Pack(2, op_str(CTB_TILED_CONST), f), nullptr);
    Py_DECREF(f);
    return r;
  }
  PyErr_Format(PyExc_TypeError, "a Tiled broadcast takes Tiled arrays and numbers, not %s", Py_TYPE(x)->tp_name);
  return nullptr;
}
PyObject* make_binary(int code, PyObject* a, PyObject* b) {
  PyObject* l = wrap(a);
  PyObject* r = l ? wrap(b) : nullptr;
  PyObject* out = r ? new_node(g_expr, PyTuple_Pack(3, op_str(code), l, r), nullptr) : nullptr;
  Py_XDECREF(l);
  Py_XDECREF(r);
  return out;
}
template <int CODE>
PyObject* nb_binary(PyObject* a, PyObject* b) { return make_binary(CODE, a, b); }
PyObject* nb_power(PyObject* a, PyObject* b, PyObject* mod) {
  if (!is_expr(a) || mod != Py_None) Py_RETURN_NOTIMPLEMENTED;
  return make_binary(CTB_TILED_POW, a, b);
}
template <int CODE>
PyObject* nb_unary(PyObject* a) { return new_node(g_expr, PyTuple_Pack(2, op_str(CODE), a), nullptr); }

int expr_init(PyObject* self, PyObject* args, PyObject* kw) {
  if (kw && PyDict_Size(kw)) {
    PyErr_SetString(PyExc_TypeError, "Expr takes no keyword arguments");
    return -1;
  }
  Py_XSETREF(reinterpret_cast<Node*>(self)->node, Py_NewRef(args));
  return 0;
}
int tiled_init(PyObject* self, PyObject* args, PyObject* kw) {
  static const char* names[] = {"tensor", nullptr};
  PyObject* t;
  if (!PyArg_ParseTupleAndKeywords(args, kw, "O", const_cast<char**>(names), &t) || !leaf_ok(t)) return -1;
  PyObject* n = PyTuple_Pack(2, op_str(CTB_TILED_INPUT), t);
  if (!n) return -1;
  Py_XSETREF(reinterpret_cast<Node*>(self)->node, n);
  Py_XSETREF(reinterpret_cast<Node*>(self)->tensor, Py_NewRef(t));
  return 0;
}
int node_traverse(PyObject* self, visitproc visit, void* arg) {
  Py_VISIT(Py_TYPE(self));
  Py_VISIT(reinterpret_cast<Node*>(self)->node);
  Py_VISIT(reinterpret_cast<Node*>(self)->tensor);
  Py_VISIT(reinterpret_cast<Node*>(self)->dict);
  return 0;
}
int node_clear(PyObject* self) {
  Py_CLEAR(reinterpret_cast<Node*>(self)->node);
  Py_CLEAR(reinterpret_cast<Node*>(self)->tensor);
  Py_CLEAR(reinterpret_cast<Node*>(self)->dict);
  return 0;
}
void node_dealloc(PyObject* self) {
  PyTypeObject* type = Py_TYPE(self);
  PyObject_GC_UnTrack(self);
  Py_TRASHCAN_BEGIN(self, node_dealloc)
  if (reinterpret_cast<Node*>(self)->weak) PyObject_ClearWeakRefs(self);
  node_clear(self);
  type->tp_free(self);
  Py_DECREF(type);
  Py_TRASHCAN_END
}
PyObject* expr_wrap(PyObject*, PyObject* x) { return wrap(x); }
// For copies and pickles: a new object of the type, its attributes, then the members above (no __init__ runs).
PyObject* node_reduce(PyObject* self, PyObject*) {
  Node* n = reinterpret_cast<Node*>(self);
  PyObject* module = PyImport_ImportModule("copyreg");
  PyObject* make = module ? PyObject_GetAttrString(module, "__newobj__") : nullptr;
  PyObject* members = make ? PyDict_New() : nullptr;
  bool ok = members && (!n->node || PyDict_SetItemString(members, "node", n->node) == 0) &&
            (!n->tensor || PyDict_SetItemString(members, "tensor", n->tensor) == 0);
  PyObject* r = ok ? Py_BuildValue("O(O)(OO)", make, Py_TYPE(self), n->dict ? n->dict : Py_None, members) : nullptr;
  Py_XDECREF(members);
  Py_XDECREF(make);
  Py_XDECREF(module);
  return r;
}
PyMemberDef kNodeMembers[] = {{"node", Py_T_OBJECT_EX, offsetof(Node, node), 0, "the operation and its operands"},
                              {"__dictoffset__", Py_T_PYSSIZET, offsetof(Node, dict), Py_READONLY, nullptr},
                              {"__weaklistoffset__", Py_T_PYSSIZET, offsetof(Node, weak), Py_READONLY, nullptr},
                              {nullptr, 0, 0, 0, nullptr}};
PyMemberDef kTiledMembers[] = {{"tensor", Py_T_OBJECT_EX, offsetof(Node, tensor), 0, "the array"}, {nullptr, 0, 0, 0, nullptr}};
PyGetSetDef kExprGetSet[] = {{"__dict__", PyObject_GenericGetDict, PyObject_GenericSetDict, nullptr, nullptr},
                             {nullptr, nullptr, nullptr, nullptr, nullptr}};
PyMethodDef kExprMethods[] = {{"__reduce__", node_reduce, METH_NOARGS, nullptr},
                              {"wrap", expr_wrap, METH_O | METH_STATIC, "an Expr of an Expr, a tensor or a number"},
                              {nullptr, nullptr, 0, nullptr}};
template <class F>
void* slot(F f) { return reinterpret_cast<void*>(f); }
PyType_Slot kExprSlots[] = {
    {Py_tp_doc, const_cast<char*>("A node of a broadcast expression: (\"leaf\", tensor) | (\"const\", value) | (unary name, Expr) | "
                                  "(binary name, Expr, Expr).")},
    {Py_tp_init, slot(expr_init)}, {Py_tp_dealloc, slot(node_dealloc)}, {Py_tp_traverse, slot(node_traverse)},
    {Py_tp_clear, slot(node_clear)}, {Py_tp_members, kNodeMembers}, {Py_tp_methods, kExprMethods}, {Py_tp_getset, kExprGetSet},
    {Py_nb_add, slot(nb_binary<CTB_TILED_ADD>)}, {Py_nb_subtract, slot(nb_binary<CTB_TILED_SUB>)},
    {Py_nb_multiply, slot(nb_binary<CTB_TILED_MUL>)}, {Py_nb_true_divide, slot(nb_binary<CTB_TILED_DIV>)},
    {Py_nb_power, slot(nb_power)}, {Py_nb_negative, slot(nb_unary<CTB_TILED_NEG>)},
    {Py_nb_absolute, slot(nb_unary<CTB_TILED_ABS>)}, {0, nullptr}};
PyType_Spec kExprSpec = {"cutile_b200.tiled.Expr", sizeof(Node), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC,
                         kExprSlots};
PyType_Slot kTiledSlots[] = {{Py_tp_doc, const_cast<char*>("``ct.Tiled(A)``: an array leaf.")}, {Py_tp_init, slot(tiled_init)},
                             {Py_tp_dealloc, slot(node_dealloc)}, {Py_tp_traverse, slot(node_traverse)},
                             {Py_tp_clear, slot(node_clear)}, {Py_tp_members, kTiledMembers}, {0, nullptr}};
PyType_Spec kTiledSpec = {"cutile_b200.tiled.Tiled", sizeof(Node), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC,
                          kTiledSlots};

// unary(name, x), binary(name, a, b): the function forms (sin, tmax, ...)
PyObject* unary(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "one argument expected");
    return nullptr;
  }
  PyObject* x = wrap(a[1]);
  if (!x) return nullptr;
  PyObject* t = PyTuple_Pack(2, a[0], x);
  Py_DECREF(x);
  return new_node(g_expr, t, nullptr);
}
PyObject* binary(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 3) {
    PyErr_SetString(PyExc_TypeError, "two arguments expected");
    return nullptr;
  }
  return make_binary(op_code(a[0]), a[1], a[2]);
}

// The tree as a postfix program over its distinct tensors and constants; false: more than the kernel takes (the Python
// path then reports it).
struct Walk {
  int32_t prog[2 * CTB_TILED_MAX_OPS];
  int n_ops = 0, n_in = 0, n_const = 0;
  PyObject* in[CTB_TILED_MAX_INPUTS];
  float consts[CTB_TILED_MAX_CONSTS];
  double exact[CTB_TILED_MAX_CONSTS];
  bool put(int op, int arg) {
    if (n_ops == CTB_TILED_MAX_OPS) return false;
    prog[2 * n_ops] = op;
    prog[2 * n_ops + 1] = arg;
    ++n_ops;
    return true;
  }
  bool walk(PyObject* e, int depth = 0) {
    PyObject* t = is_expr(e) ? reinterpret_cast<Node*>(e)->node : nullptr;
    if (!t || !PyTuple_Check(t) || PyTuple_GET_SIZE(t) < 2 || depth > CTB_TILED_MAX_OPS) return false;
    const int code = op_code(PyTuple_GET_ITEM(t, 0));
    const Py_ssize_t size = PyTuple_GET_SIZE(t);
    PyObject* x = PyTuple_GET_ITEM(t, 1);
    if (code == CTB_TILED_INPUT) {
      int i = 0;
      while (i < n_in && in[i] != x) ++i;
      if (i == CTB_TILED_MAX_INPUTS) return false;
      if (i == n_in) in[n_in++] = x;
      return put(CTB_TILED_INPUT, i);
    }
    if (code == CTB_TILED_CONST) {
      if (!PyFloat_Check(x)) return false;
      const double v = PyFloat_AS_DOUBLE(x);
      int i = 0;
      while (i < n_const && std::memcmp(&exact[i], &v, sizeof v)) ++i;  // 0.0 and -0.0 are two constants
      if (i == CTB_TILED_MAX_CONSTS) return false;
      if (i == n_const) {
        exact[n_const] = v;
        consts[n_const++] = (float)v;
      }
      return put(CTB_TILED_CONST, i);
    }
    if (code < 0 || size != (code >= CTB_TILED_ADD ? 3 : 2)) return false;
    for (Py_ssize_t k = 1; k < size; ++k)
      if (!walk(PyTuple_GET_ITEM(t, k), depth + 1)) return false;
    return put(code, 0);
  }
};
// Julia shape (first dimension contiguous) padded to three dimensions
void jshape(const Tensor& t, int64_t (&s)[3]) {
  const int d = (int)t.dim();
  for (int k = 0; k < 3; ++k) s[k] = k < d ? t.size(d - 1 - k) : 1;
}

// assign(dest, expr): dest .= expr
PyObject* assign(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor* dest;
  Walk w;
  if (n != 2 || !(dest = cuda_tensor(a[0])) || dest->dim() > 3 || !dest->is_contiguous() || dtype_of(*dest) < 0) return decline();
  PyObject* expr = wrap(a[1]);  // holds the operands until the call below is enqueued
  if (!expr) return nullptr;
  struct Hold {
    PyObject* o;
    ~Hold() { Py_DECREF(o); }
  } hold{expr};
  if (!w.walk(expr)) return decline();
  int64_t shape[3], strides[3 * CTB_TILED_MAX_INPUTS];
  const void* ptrs[CTB_TILED_MAX_INPUTS];
  jshape(*dest, shape);
  for (int i = 0; i < w.n_in; ++i) {
    const Tensor* t = cuda_tensor(w.in[i]);
    if (!t || t->dim() > 3 || !t->is_contiguous() || t->scalar_type() != dest->scalar_type() || t->device() != dest->device())
      return decline();
    int64_t s[3], run = 1;
    jshape(*t, s);
    for (int k = 0; k < 3; ++k) {
      if (s[k] != 1 && s[k] != shape[k]) return decline();
      strides[3 * i + k] = s[k] == 1 ? 0 : run;
      run *= s[k];
    }
    ptrs[i] = t->data_ptr();
  }
  Call c(*dest);
  if (!c.ok()) return nullptr;
  const int s = without_gil([&] {
    return ctb_tiled_broadcast(c.ctx, c.stream, dest->data_ptr(), shape, ptrs, strides, w.n_in, w.prog, w.n_ops, w.consts,
                               w.n_const, dtype_of(*dest));
  });
  return done(s, yes());
}

// mapreduce(f, op, tensor or Tiled, dims: None, int or tuple) -> the reduced tensor
PyObject* mapreduce(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4) return decline();
  PyObject* src = PyObject_TypeCheck(a[2], g_tiled) ? reinterpret_cast<Node*>(a[2])->tensor : a[2];
  const Tensor* t = src ? cuda_tensor(src) : nullptr;
  const int f = op_code(a[0]), op = op_code(a[1]);
  if (!t || t->dim() > 3 || !t->is_contiguous() || dtype_of(*t) < 0 || f < CTB_TILED_IDENTITY || f > CTB_TILED_ABS2 ||
      op < CTB_TILED_ADD)
    return decline();
  const int d = (int)t->dim();
  int mask = 0;
  long long v;
  auto add = [&](PyObject* o) {
    if (!as_int(o, &v) || v < 1) return false;
    if (v <= d) mask |= 1 << (v - 1);
    return true;
  };
  if (a[3] == Py_None) {
    mask = (1 << d) - 1;
  } else if (PyTuple_Check(a[3])) {
    for (Py_ssize_t k = 0; k < PyTuple_GET_SIZE(a[3]); ++k)
      if (!add(PyTuple_GET_ITEM(a[3], k))) return decline();
  } else if (!add(a[3])) {
    return decline();
  }
  int64_t shape[3], out[3];
  jshape(*t, shape);
  for (int k = 0; k < d; ++k) out[d - 1 - k] = (mask >> k) & 1 ? 1 : shape[k];
  Call c(*t);
  if (!c.ok()) return nullptr;
  Tensor dest = a[3] == Py_None ? at::empty({}, t->options()) : at::empty(at::IntArrayRef(out, d), t->options());
  const int s = without_gil([&] {
    return ctb_tiled_mapreduce(c.ctx, c.stream, dest.data_ptr(), t->data_ptr(), shape, mask, f, op, dtype_of(*t));
  });
  if (s != CTB_OK) return done(s, nullptr);
  return THPVariable_Wrap(std::move(dest));
}

// fft(x complex64 [batch, N], out or None, (W0, W1, W2, T0, T1) of make_twiddles, N, F0, F1, F2, D) -> out
PyObject* fft(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const Tensor *x, *out, *tab[2];
  long long v[5];
  if (n != 8 || !(x = cuda_tensor(a[0])) || !PyTuple_Check(a[2]) || PyTuple_GET_SIZE(a[2]) != 5 || !ints(a + 3, 5, v))
    return decline();
  const int64_t N = v[0], F0 = v[1], F1 = v[2], F2 = v[3];
  if (x->scalar_type() != at::kComplexFloat || x->dim() != 2 || x->size(1) != N || !x->is_contiguous() || x->is_conj())
    return decline();
  const int64_t want[2] = {2 * F0 * F1 * F2, 2 * F1 * F2};
  for (int i = 0; i < 2; ++i)
    if (!(tab[i] = cuda_tensor(PyTuple_GET_ITEM(a[2], 3 + i))) || !vec_f32(tab[i], want[i])) return decline();
  Tensor made;
  if (a[1] == Py_None) {
    made = at::empty(x->sizes(), x->options());
    out = &made;
  } else if (!(out = cuda_tensor(a[1])) || out->scalar_type() != at::kComplexFloat || out->sizes() != x->sizes() ||
             !out->is_contiguous() || out->is_conj()) {
    return decline();
  }
  Call c(*x);
  if (!c.ok()) return nullptr;
  const int s = without_gil([&] {
    return ctb_fft_plan(c.ctx, c.stream, x->data_ptr(), out->data_ptr(), tab[0]->data_ptr(), tab[1]->data_ptr(), N, (int)F0,
                        (int)F1, (int)F2, x->size(0), 1, (int)v[4]);
  });
  if (s != CTB_OK || a[1] != Py_None) return done(s, s == CTB_OK ? Py_NewRef(a[1]) : nullptr);
  return THPVariable_Wrap(std::move(made));
}

PyObject* setup(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 3) {
    PyErr_SetString(PyExc_TypeError, "setup(context, check, leaf_error)");
    return nullptr;
  }
  Py_XSETREF(g_context, Py_NewRef(a[0]));
  Py_XSETREF(g_check, Py_NewRef(a[1]));
  Py_XSETREF(g_leaf_error, Py_NewRef(a[2]));
  Py_RETURN_NONE;
}

// A C++ exception (out of memory from the allocator, say) becomes the Python exception torch raises for it.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(self, a, n);
  END_HANDLE_TH_ERRORS
}
#define CTB_METHOD(name) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {CTB_METHOD(setup),         CTB_METHOD(softmax),        CTB_METHOD(vadd),
                          CTB_METHOD(transpose),     CTB_METHOD(layernorm_fwd),  CTB_METHOD(layernorm_bwd),
                          CTB_METHOD(layernorm_dwdb), CTB_METHOD(matmul),        CTB_METHOD(batch_matmul),
                          CTB_METHOD(fmha),          CTB_METHOD(moe_router),     CTB_METHOD(moe_ffn),
                          CTB_METHOD(unary),         CTB_METHOD(binary),         CTB_METHOD(assign),
                          CTB_METHOD(mapreduce),     CTB_METHOD(fft),
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "Native call path of cutile_b200.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  for (auto& o : g_ops)
    if (!(o.str = PyUnicode_InternFromString(o.name))) return nullptr;
  PyObject* m = PyModule_Create(&kModule);
  if (!m) return nullptr;
  g_expr = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&kExprSpec));
  g_tiled = g_expr ? reinterpret_cast<PyTypeObject*>(PyType_FromSpecWithBases(&kTiledSpec, reinterpret_cast<PyObject*>(g_expr)))
                   : nullptr;
  if (!g_tiled || PyModule_AddStringConstant(m, "TORCH_VERSION", CTB_TORCH_VERSION) < 0 ||
      PyModule_AddObjectRef(m, "Expr", reinterpret_cast<PyObject*>(g_expr)) < 0 ||
      PyModule_AddObjectRef(m, "Tiled", reinterpret_cast<PyObject*>(g_tiled)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
