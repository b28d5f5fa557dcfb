/* The Python side of the smallest qf.* calls, in C: the checks of quark_b200/functional on QuarkTensor slots, then the call into
 * the kernel library.  A kernel of two to four microseconds is otherwise bound by the interpreter (checks and ctypes: 2.7 us for a
 * norm, 3.3 us for a GEMM).
 *
 * Every function returns None for a call it does not take (an output to be allocated, a tensor of another type, any argument that
 * fails a check), and the Python function then goes its own way, which also words the error; otherwise the status of the library
 * call.  bind() receives the tensor class and the addresses of the library's entry points. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include "../../include/quark_b200.h"

static PyTypeObject* g_tensor = NULL;
static Py_ssize_t g_ptr, g_numel, g_nbytes, g_dtype, g_shape; /* slot offsets */
static PyObject* g_names[4];                                  /* bf16, e4m3, f32, s32: the codes of qb_dtype */

typedef int32_t (*gemm_fn)(const void*, const void*, void*, const void*, const void*, const void*, const qb_gemm_params*, void*, size_t, void*);
typedef size_t (*gemm_ws_fn)(const qb_gemm_params*);
typedef int32_t (*ada_fn)(const void*, const void*, const void*, void*, void*, int32_t, int32_t, int32_t, float, int32_t, void*);
typedef int32_t (*rms_fn)(const void*, void*, int32_t, int32_t, float, void*);
typedef int32_t (*head_fn)(const void*, void*, int32_t, int32_t, int32_t, int32_t, float, void*);
typedef int32_t (*gate_fn)(const void*, const void*, const void*, void*, int32_t, int32_t, int32_t, void*);
typedef int32_t (*silu_fn)(const void*, void*, void*, size_t, void*);
typedef int32_t (*add_fn)(const void*, const void*, void*, size_t, void*);
typedef int32_t (*euler_fn)(const void*, const void*, const float*, void*, size_t, void*);
typedef int32_t (*quant_fn)(const void*, void*, size_t, int32_t, void*);
typedef int32_t (*dequant_fn)(const void*, void*, size_t, void*);
typedef int32_t (*append_fn)(const void*, const int32_t*, const int32_t*, void*, void*, int32_t*, int32_t*, const float*, const qb_kv_params*, void*);
typedef int32_t (*append_kv_fn)(const void*, const void*, const int32_t*, const int32_t*, void*, void*, int32_t*, int32_t*, const float*, const qb_kv_params*, void*);
typedef size_t (*attn_ws_fn)(const qb_attn_params*);
typedef int32_t (*attn_fn)(const void*, const void*, const void*, const int32_t*, const int32_t*, const int32_t*, void*, void*, const float*, const qb_attn_params*, void*,
                           size_t, void*);

static struct {
  gemm_fn gemm;
  gemm_ws_fn gemm_ws;
  ada_fn ada;
  ada_fn ada_chained;
  rms_fn rms;
  head_fn head;
  gate_fn gate;
  silu_fn silu;
  add_fn add;
  euler_fn euler;
  quant_fn quant;
  dequant_fn dequant;
  append_fn append;
  append_kv_fn append_kv;
  attn_ws_fn attn_ws;
  attn_fn attn;
} g_lib;

typedef struct {
  void* ptr;
  long long numel, nbytes;
  int dtype; /* qb_dtype, -1 for any other */
  PyObject* shape;
} Tensor;

static int dtype_code(PyObject* name) {
  for (int i = 0; i < 4; ++i)
    if (name == g_names[i]) return i;
  if (name != NULL && PyUnicode_Check(name))
    for (int i = 0; i < 4; ++i)
      if (PyUnicode_Compare(name, g_names[i]) == 0) return i;
  return -1;
}
static PyObject* slot(PyObject* o, Py_ssize_t at) { return *(PyObject**)((char*)o + at); }

static int tensor(PyObject* o, Tensor* t) {
  if (g_tensor == NULL || Py_TYPE(o) != g_tensor) return 0;
  PyObject *p = slot(o, g_ptr), *n = slot(o, g_numel), *b = slot(o, g_nbytes), *s = slot(o, g_shape);
  if (p == NULL || n == NULL || b == NULL || s == NULL || !PyLong_CheckExact(p) || !PyLong_CheckExact(n) || !PyLong_CheckExact(b) || !PyTuple_CheckExact(s)) return 0;
  t->ptr = (void*)(uintptr_t)PyLong_AsUnsignedLongLong(p);
  t->numel = PyLong_AsLongLong(n);
  t->nbytes = PyLong_AsLongLong(b);
  t->dtype = dtype_code(slot(o, g_dtype));
  t->shape = s;
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return 0;
  }
  return 1;
}
static int tensor_or_none(PyObject* o, Tensor* t) {
  if (o == Py_None) {
    memset(t, 0, sizeof(*t));
    return 1;
  }
  return tensor(o, t);
}
static int as_ll(PyObject* o, long long* v) {
  if (!PyLong_Check(o)) return 0;
  *v = PyLong_AsLongLong(o);
  if (*v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return 0;
  }
  return 1;
}
static int as_float(PyObject* o, float* v) {
  if (!PyFloat_Check(o)) return 0;
  *v = (float)PyFloat_AS_DOUBLE(o);
  return 1;
}
static int stream_of(PyObject* o, void** s) {
  long long v;
  if (!as_ll(o, &v)) return 0;
  *s = (void*)(uintptr_t)v;
  return 1;
}
static long long dim(const Tensor* t, Py_ssize_t i) {
  const Py_ssize_t n = PyTuple_GET_SIZE(t->shape);
  long long v;
  if (i < 0) i += n;
  if (i < 0 || i >= n || !as_ll(PyTuple_GET_ITEM(t->shape, i), &v)) return -1;
  return v;
}
/* 0 for None, 1 for "silu", -1 for anything else */
static int activation_of(PyObject* o) {
  if (o == Py_None) return 0;
  return PyUnicode_Check(o) && PyUnicode_CompareWithASCIIString(o, "silu") == 0 ? 1 : -1;
}
#define SMALL(x) ((x) > 0 && (x) <= 0x7fffffffll)
#define RUN(call)                      \
  do {                                 \
    int32_t rc_;                       \
    Py_BEGIN_ALLOW_THREADS rc_ = call; \
    Py_END_ALLOW_THREADS return PyLong_FromLong(rc_); \
  } while (0)

/* (A, B, out_dtype, compute_dtype, activation, bias, gate, residual, gate_groups, out, a_scale, w_scale, split_k, tile_n, flags, workspace, stream) */
static PyObject* fast_gemm(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor A, B, C, bias, gate, res, sa, sw, ws;
  long long groups, split, tile, flags;
  void* st;
  if (n != 17 || g_lib.gemm == NULL || !tensor(a[0], &A) || !tensor(a[1], &B) || !tensor(a[9], &C) || !tensor_or_none(a[5], &bias) ||
      !tensor_or_none(a[6], &gate) || !tensor_or_none(a[7], &res) || !tensor_or_none(a[10], &sa) || !tensor_or_none(a[11], &sw) ||
      !tensor_or_none(a[15], &ws) || !as_ll(a[8], &groups) || !as_ll(a[12], &split) || !as_ll(a[13], &tile) || !as_ll(a[14], &flags) || !stream_of(a[16], &st))
    Py_RETURN_NONE;
  const int act = activation_of(a[4]);
  if (act < 0 || PyTuple_GET_SIZE(A.shape) < 2 || PyTuple_GET_SIZE(B.shape) != 2 || A.dtype < 0 || A.dtype > 1 || B.dtype < 0 || B.dtype > 1 || C.dtype < 0) Py_RETURN_NONE;
  const int cd = a[3] == Py_None ? (B.dtype == QB_E4M3 ? QB_E4M3 : A.dtype) : dtype_code(a[3]);
  if (cd != QB_BF16 && cd != QB_E4M3) Py_RETURN_NONE;
  if (a[2] != Py_None && dtype_code(a[2]) != C.dtype) Py_RETURN_NONE;
  const long long K = dim(&A, -1), N = dim(&B, 0);
  if (!SMALL(K) || !SMALL(N) || dim(&B, 1) != K) Py_RETURN_NONE;
  const long long M = A.numel / K;
  if (!SMALL(M) || C.numel != M * N || (bias.ptr != NULL && bias.numel != N) || (gate.ptr == NULL) != (res.ptr == NULL) || !SMALL(groups)) Py_RETURN_NONE;
  if (gate.ptr != NULL && (gate.numel != groups * N || res.numel != M * N || M % groups != 0)) Py_RETURN_NONE;
  qb_gemm_params p;
  p.M = (int32_t)M; p.N = (int32_t)N; p.K = (int32_t)K;
  p.a_dtype = A.dtype; p.b_dtype = B.dtype; p.c_dtype = C.dtype;
  p.compute_dtype = cd; p.activation = act; p.gate_groups = (int32_t)groups;
  p.split_k = (int32_t)split; p.tile_n = (int32_t)tile; p.reserved = (int32_t)flags;
  p.a_scale = (const float*)sa.ptr; p.w_scale = (const float*)sw.ptr;
  if (g_lib.gemm_ws(&p) > (size_t)ws.nbytes) Py_RETURN_NONE;
  RUN(g_lib.gemm(A.ptr, B.ptr, C.ptr, bias.ptr, gate.ptr, res.ptr, &p, ws.ptr, (size_t)ws.nbytes, st));
}

/* (X, scale, bias, eps, activation, out, out_q, only_q, chained, stream) */
static PyObject* fast_ada_rmsnorm(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor X, sc, bi, out, oq;
  float eps;
  void* st;
  if (n != 10 || g_lib.ada == NULL || !tensor(a[0], &X) || !tensor(a[1], &sc) || !tensor(a[2], &bi) || !as_float(a[3], &eps) || !tensor_or_none(a[5], &out) ||
      !tensor_or_none(a[6], &oq) || !stream_of(a[9], &st))
    Py_RETURN_NONE;
  const int act = activation_of(a[4]), only_q = a[7] == Py_True;
  if ((a[7] != Py_True && a[7] != Py_False) || (a[8] != Py_True && a[8] != Py_False)) Py_RETURN_NONE;
  if (only_q) out.ptr = NULL;
  if (act < 0 || (only_q ? oq.ptr == NULL : out.ptr == NULL) || X.dtype != QB_BF16 || sc.dtype != QB_BF16 || bi.dtype != QB_BF16) Py_RETURN_NONE;
  const long long D = dim(&X, -1);
  if (!SMALL(D)) Py_RETURN_NONE;
  const long long rows = X.numel / D, G = sc.numel / D;
  if (!SMALL(rows) || !SMALL(G) || sc.numel != G * D || bi.numel != G * D || rows % G != 0) Py_RETURN_NONE;
  if (out.ptr != NULL && (out.numel != X.numel || out.dtype != X.dtype)) Py_RETURN_NONE;
  if (oq.ptr != NULL && (oq.numel != X.numel || oq.dtype != QB_E4M3)) Py_RETURN_NONE;
  const ada_fn call = a[8] == Py_True ? g_lib.ada_chained : g_lib.ada;
  RUN(call(X.ptr, sc.ptr, bi.ptr, out.ptr, oq.ptr, (int32_t)rows, (int32_t)D, (int32_t)G, eps, act, st));
}

/* (X, eps, out, stream) */
static PyObject* fast_rmsnorm(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor X, out;
  float eps;
  void* st;
  if (n != 4 || g_lib.rms == NULL || !tensor(a[0], &X) || !as_float(a[1], &eps) || !tensor(a[2], &out) || !stream_of(a[3], &st)) Py_RETURN_NONE;
  const long long D = dim(&X, -1);
  if (X.dtype != QB_BF16 || out.dtype != QB_BF16 || out.numel != X.numel || !SMALL(D) || !SMALL(X.numel / D)) Py_RETURN_NONE;
  RUN(g_lib.rms(X.ptr, out.ptr, (int32_t)(X.numel / D), (int32_t)D, eps, st));
}

/* (X, n_q_heads, n_kv_heads, Dh, eps, out, stream) */
static PyObject* fast_head_rmsnorm(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor X, out;
  long long nq, nk, Dh;
  float eps;
  void* st;
  if (n != 7 || g_lib.head == NULL || !tensor(a[0], &X) || !as_ll(a[1], &nq) || !as_ll(a[2], &nk) || !as_ll(a[3], &Dh) || !as_float(a[4], &eps) ||
      !tensor(a[5], &out) || !stream_of(a[6], &st))
    Py_RETURN_NONE;
  if (X.dtype != QB_BF16 || out.dtype != QB_BF16 || out.numel != X.numel || PyTuple_GET_SIZE(X.shape) != 2 || nq < 0 || nk < 0 || !SMALL(nq + nk) ||
      !SMALL(Dh) || dim(&X, 1) != (nq + 2 * nk) * Dh || !SMALL(dim(&X, 0)))
    Py_RETURN_NONE;
  RUN(g_lib.head(X.ptr, out.ptr, (int32_t)dim(&X, 0), (int32_t)nq, (int32_t)nk, (int32_t)Dh, eps, st));
}

/* (X, Y, gate, out, stream) */
static PyObject* fast_gate_residual(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor X, Y, g, out;
  void* st;
  if (n != 5 || g_lib.gate == NULL || !tensor(a[0], &X) || !tensor(a[1], &Y) || !tensor(a[2], &g) || !tensor(a[3], &out) || !stream_of(a[4], &st)) Py_RETURN_NONE;
  const long long D = dim(&X, -1);
  if (X.dtype != QB_BF16 || Y.dtype != QB_BF16 || g.dtype != QB_BF16 || out.dtype != QB_BF16 || !SMALL(D) || Y.numel != X.numel || out.numel != X.numel) Py_RETURN_NONE;
  const long long rows = X.numel / D, G = g.numel / D;
  if (!SMALL(rows) || !SMALL(G) || g.numel != G * D || rows % G != 0) Py_RETURN_NONE;
  RUN(g_lib.gate(X.ptr, Y.ptr, g.ptr, out.ptr, (int32_t)rows, (int32_t)D, (int32_t)G, st));
}

/* (X, out, out_q, stream) */
static PyObject* fast_silu(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor X, out, oq;
  void* st;
  if (n != 4 || g_lib.silu == NULL || !tensor(a[0], &X) || !tensor(a[1], &out) || !tensor_or_none(a[2], &oq) || !stream_of(a[3], &st)) Py_RETURN_NONE;
  if (X.dtype != QB_BF16 || out.dtype != QB_BF16 || out.numel != X.numel || (oq.ptr != NULL && (oq.dtype != QB_E4M3 || oq.numel != X.numel))) Py_RETURN_NONE;
  RUN(g_lib.silu(X.ptr, out.ptr, oq.ptr, (size_t)X.numel, st));
}

/* (X, Y, out, stream) */
static PyObject* fast_add(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor X, Y, out;
  void* st;
  if (n != 4 || g_lib.add == NULL || !tensor(a[0], &X) || !tensor(a[1], &Y) || !tensor(a[2], &out) || !stream_of(a[3], &st)) Py_RETURN_NONE;
  if (X.dtype != QB_BF16 || Y.dtype != QB_BF16 || out.dtype != QB_BF16 || Y.numel != X.numel || out.numel != X.numel) Py_RETURN_NONE;
  RUN(g_lib.add(X.ptr, Y.ptr, out.ptr, (size_t)X.numel, st));
}

/* (X, V, Dsig, out, stream) */
static PyObject* fast_euler_step(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor X, V, D, out;
  void* st;
  if (n != 5 || g_lib.euler == NULL || !tensor(a[0], &X) || !tensor(a[1], &V) || !tensor(a[2], &D) || !tensor(a[3], &out) || !stream_of(a[4], &st)) Py_RETURN_NONE;
  if (X.dtype != QB_BF16 || V.dtype != QB_BF16 || out.dtype != QB_BF16 || D.dtype != QB_F32 || V.numel != X.numel || out.numel != X.numel) Py_RETURN_NONE;
  RUN(g_lib.euler(X.ptr, V.ptr, (const float*)D.ptr, out.ptr, (size_t)X.numel, st));
}

/* (X, out, stream) */
static PyObject* fast_quantize(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor X, out;
  void* st;
  if (n != 3 || g_lib.quant == NULL || !tensor(a[0], &X) || !tensor(a[1], &out) || !stream_of(a[2], &st)) Py_RETURN_NONE;
  if ((X.dtype != QB_BF16 && X.dtype != QB_F32) || out.dtype != QB_E4M3 || out.numel != X.numel) Py_RETURN_NONE;
  RUN(g_lib.quant(X.ptr, out.ptr, (size_t)X.numel, X.dtype, st));
}
static PyObject* fast_dequantize(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor X, out;
  void* st;
  if (n != 3 || g_lib.dequant == NULL || !tensor(a[0], &X) || !tensor(a[1], &out) || !stream_of(a[2], &st)) Py_RETURN_NONE;
  if (X.dtype != QB_E4M3 || out.dtype != QB_BF16 || out.numel != X.numel) Py_RETURN_NONE;
  RUN(g_lib.dequant(X.ptr, out.ptr, (size_t)X.numel, st));
}

/* The geometry that the append and the attention share, and the cache tensors' shapes against it. */
typedef struct {
  long long nk, H, W, nb, pd, segs, qf, qo, tpf;
  int packed;
} Geometry;
static int geometry(Geometry* g, PyObject* B, PyObject* nk, PyObject* H, PyObject* W, PyObject* nb, PyObject* pd, PyObject* segs, PyObject* packed, PyObject* qf, PyObject* qo,
                    const Tensor* K, const Tensor* Vt, const Tensor* seg, const Tensor* nseg) {
  long long b;
  if (!as_ll(B, &b) || b != 1 || !as_ll(nk, &g->nk) || !as_ll(H, &g->H) || !as_ll(W, &g->W) || !as_ll(nb, &g->nb) || !as_ll(pd, &g->pd) || !as_ll(segs, &g->segs) ||
      !as_ll(qf, &g->qf) || !as_ll(qo, &g->qo) || (packed != Py_True && packed != Py_False))
    return 0;
  g->packed = packed == Py_True;
  if (g->nk <= 0 || g->nk > 65536 || g->H <= 0 || g->H > 65536 || g->W <= 0 || g->W > 65536 || g->nb <= 0 || g->nb > (1 << 24) || !SMALL(g->pd) || g->segs <= 0 ||
      g->segs > 65536 || g->qf < 1 || g->qf > 65536 || (g->qf & (g->qf - 1)) != 0 || g->qo < 0 || g->qo >= g->qf)
    return 0;
  g->tpf = g->H * g->W;
  if (g->tpf % g->qf != 0) return 0;
  const long long cap = (g->nb + 1) * (g->tpf / g->qf);
  return PyTuple_GET_SIZE(K->shape) == 2 && dim(K, 0) == g->nk * cap && dim(K, 1) == 64 && PyTuple_GET_SIZE(Vt->shape) == 2 && dim(Vt, 0) == g->nk * 64 && dim(Vt, 1) == cap &&
         dim(seg, 0) == g->segs * 2 && dim(nseg, 0) == 1 && K->dtype == Vt->dtype && (K->dtype == QB_BF16 || K->dtype == QB_E4M3);
}
/* per-head scales: None, or f32 of one value per KV head */
static int head_scale(PyObject* o, long long nk, const float** p) {
  Tensor t;
  if (!tensor_or_none(o, &t) || (t.ptr != NULL && (t.dtype != QB_F32 || t.numel != nk))) return 0;
  *p = (const float*)t.ptr;
  return 1;
}

/* (K, V, frame_t, frozen, Vt_cache, segments, n_segments, K_cache, B, n_kv_heads, H, W, num_buckets, pinned_dilation, kv_dtype, max_segments, packed, n_q_heads,
 *  quilt_factor, quilt_offset, k_scale, v_scale, rope table, stream) */
static PyObject* fast_kv_cache_update(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor K, V, ft, fz, Vc, seg, nseg, Kc, rope;
  Geometry g;
  long long nq;
  qb_kv_params p;
  void* st;
  if (n != 24 || g_lib.append == NULL || !tensor(a[0], &K) || !tensor(a[2], &ft) || !tensor(a[3], &fz) || !tensor(a[4], &Vc) || !tensor(a[5], &seg) || !tensor(a[6], &nseg) ||
      !tensor(a[7], &Kc) || !tensor(a[22], &rope) || !as_ll(a[17], &nq) || !stream_of(a[23], &st) ||
      !geometry(&g, a[8], a[9], a[10], a[11], a[12], a[13], a[15], a[16], a[18], a[19], &Kc, &Vc, &seg, &nseg) || !head_scale(a[20], g.nk, &p.k_scale) ||
      !head_scale(a[21], g.nk, &p.v_scale))
    Py_RETURN_NONE;
  if (nq < 0 || nq > (1 << 20) || K.dtype != QB_BF16 || PyTuple_GET_SIZE(K.shape) != 2 || (a[14] != Py_None && dtype_code(a[14]) != Kc.dtype)) Py_RETURN_NONE;
  if (g.packed ? dim(&K, 0) != g.tpf || dim(&K, 1) != (nq + 2 * g.nk) * 64 : dim(&K, 0) != g.nk * g.tpf || dim(&K, 1) != 64) Py_RETURN_NONE;
  if (!g.packed && (!tensor(a[1], &V) || V.dtype != QB_BF16 || PyTuple_GET_SIZE(V.shape) != 2 || dim(&V, 0) != dim(&K, 0) || dim(&V, 1) != 64)) Py_RETURN_NONE;
  p.n_q_heads = (int32_t)nq; p.n_kv_heads = (int32_t)g.nk; p.H_spatial = (int32_t)g.H; p.W_spatial = (int32_t)g.W;
  p.num_buckets = (int32_t)g.nb; p.pinned_dilation = (int32_t)g.pd; p.kv_dtype = Kc.dtype; p.max_segments = (int32_t)g.segs;
  p.quilt_factor = (int32_t)g.qf; p.packed_qkv = g.packed; p.quilt_offset = (int32_t)g.qo;
  if (g.packed) RUN(g_lib.append(K.ptr, ft.ptr, fz.ptr, Kc.ptr, Vc.ptr, seg.ptr, nseg.ptr, rope.ptr, &p, st));
  RUN(g_lib.append_kv(K.ptr, V.ptr, ft.ptr, fz.ptr, Kc.ptr, Vc.ptr, seg.ptr, nseg.ptr, rope.ptr, &p, st));
}

/* (Q, K_cache, Vt_cache, segments, n_segments, B, n_kv_heads, gqa_ratio, H, W, num_buckets, pinned_dilation, out_dtype, compute_dtype, max_segments, packed,
 *  quilt_factor, quilt_offset, frame_t, out, out_q, k_scale, v_scale, kv_splits, rope table, workspace, stream) */
static PyObject* fast_owl_attn(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  Tensor Q, Kc, Vc, seg, nseg, ft, out, oq, rope, ws;
  Geometry g;
  long long gqa, splits;
  qb_attn_params p;
  void* st;
  if (n != 27 || g_lib.attn == NULL || !tensor(a[0], &Q) || !tensor(a[1], &Kc) || !tensor(a[2], &Vc) || !tensor(a[3], &seg) || !tensor(a[4], &nseg) || !tensor(a[18], &ft) ||
      !tensor(a[19], &out) || !tensor_or_none(a[20], &oq) || !tensor(a[24], &rope) || !tensor_or_none(a[25], &ws) || !as_ll(a[7], &gqa) || !as_ll(a[23], &splits) ||
      !stream_of(a[26], &st) || !geometry(&g, a[5], a[6], a[8], a[9], a[10], a[11], a[14], a[15], a[16], a[17], &Kc, &Vc, &seg, &nseg) ||
      !head_scale(a[21], g.nk, &p.k_scale) || !head_scale(a[22], g.nk, &p.v_scale))
    Py_RETURN_NONE;
  /* a cache of another dtype than the compute dtype is cast first: Python's way */
  if ((a[13] == Py_None ? QB_BF16 : dtype_code(a[13])) != Kc.dtype || (a[12] != Py_None && dtype_code(a[12]) != QB_BF16) || gqa <= 0 || gqa > 65536 || splits < 0 ||
      splits > 16 || Q.dtype != QB_BF16 || out.dtype != QB_BF16 || PyTuple_GET_SIZE(Q.shape) != 2)
    Py_RETURN_NONE;
  const long long nq = g.nk * gqa;
  if (g.packed ? dim(&Q, 0) != g.tpf || dim(&Q, 1) != (nq + 2 * g.nk) * 64 : dim(&Q, 0) != nq * g.tpf || dim(&Q, 1) != 64) Py_RETURN_NONE;
  if (out.numel != g.tpf * nq * 64 || (oq.ptr != NULL && (oq.dtype != QB_E4M3 || oq.numel != out.numel))) Py_RETURN_NONE;
  p.n_kv_heads = (int32_t)g.nk; p.gqa_ratio = (int32_t)gqa; p.H_spatial = (int32_t)g.H; p.W_spatial = (int32_t)g.W;
  p.num_buckets = (int32_t)g.nb; p.pinned_dilation = (int32_t)g.pd; p.kv_dtype = p.compute_dtype = Kc.dtype; p.max_segments = (int32_t)g.segs;
  p.packed_qkv = g.packed; p.quilt_factor = (int32_t)g.qf; p.kv_splits = (int32_t)splits;
  const size_t need = g_lib.attn_ws(&p);
  if (need > (size_t)ws.nbytes) Py_RETURN_NONE;
  RUN(g_lib.attn(Q.ptr, Kc.ptr, Vc.ptr, seg.ptr, nseg.ptr, ft.ptr, out.ptr, oq.ptr, rope.ptr, &p, need > 0 ? ws.ptr : NULL, need > 0 ? (size_t)ws.nbytes : 0, st));
}

/* (tensor class, {entry point: address}) */
static PyObject* fast_bind(PyObject* self, PyObject* args) {
  PyObject *cls, *table;
  if (!PyArg_ParseTuple(args, "O!O!", &PyType_Type, &cls, &PyDict_Type, &table)) return NULL;
  static const char* const members[5] = {"_ptr", "numel", "nbytes", "dtype", "shape"};
  Py_ssize_t* const at[5] = {&g_ptr, &g_numel, &g_nbytes, &g_dtype, &g_shape};
  for (int i = 0; i < 5; ++i) {
    PyObject* d = PyDict_GetItemString(((PyTypeObject*)cls)->tp_dict, members[i]);
    if (d == NULL || Py_TYPE(d) != &PyMemberDescr_Type) {
      PyErr_Format(PyExc_TypeError, "bind: %s is not a slot of the tensor class", members[i]);
      return NULL;
    }
    *at[i] = ((PyMemberDescrObject*)d)->d_member->offset;
  }
  static const char* const names[16] = {"qb_gemm", "qb_gemm_workspace_bytes", "qb_ada_rmsnorm", "qb_ada_rmsnorm_chained", "qb_rmsnorm", "qb_head_rmsnorm", "qb_ada_gate_residual",
                                        "qb_silu", "qb_add", "qb_euler_step", "qb_quantize_e4m3", "qb_dequantize_e4m3", "qb_kv_cache_update",
                                        "qb_kv_cache_update_kv", "qb_owl_attn_scratch_bytes", "qb_owl_attn"};
  void** const fn = (void**)&g_lib;
  for (int i = 0; i < 16; ++i) {
    PyObject* v = PyDict_GetItemString(table, names[i]);
    if (v == NULL) {
      PyErr_Format(PyExc_KeyError, "bind: %s", names[i]);
      return NULL;
    }
    fn[i] = PyLong_AsVoidPtr(v);
    if (fn[i] == NULL && PyErr_Occurred()) return NULL;
  }
  Py_INCREF(cls);
  Py_XDECREF((PyObject*)g_tensor);
  g_tensor = (PyTypeObject*)cls;
  Py_RETURN_NONE;
}

#define F(name) {#name, (PyCFunction)(void (*)(void))fast_##name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {{"bind", fast_bind, METH_VARARGS, NULL}, F(gemm), F(ada_rmsnorm), F(rmsnorm), F(head_rmsnorm), F(gate_residual), F(silu),
                                F(add), F(euler_step), F(quantize), F(dequantize), F(kv_cache_update), F(owl_attn), {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void) {
  static const char* const names[4] = {"bf16", "e4m3", "f32", "s32"};
  for (int i = 0; i < 4; ++i) {
    g_names[i] = PyUnicode_InternFromString(names[i]);
    if (g_names[i] == NULL) return NULL;
  }
  return PyModule_Create(&module);
}
