// CPython binding of the C ABI: what `ops.py` and the cache classes call on every decode step.
//
// One call per operator takes torch tensors positionally, fills the pk_tensor descriptors, allocates the outputs,
// picks torch's current stream and calls the library, all natively.  The same work in Python (a ctypes structure per
// tensor, filled element by element) measured 2 us a tensor on the B200 hosts, 100 - 160 us for the four launches of a
// layer's decode step, which the GPU runs in 45 - 60 us: eager decoding was bound by it.  Plain METH_FASTCALL
// functions, not pybind11 or dispatcher ops: those cost a microsecond or more per call themselves.
// The C ABI stays free of torch types; this module is one of its callers.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/pariskv_b200.h"

namespace {

// A tensor argument: descriptor for the C ABI, null for None.
struct Arg {
  pk_tensor d = {};
  const at::Tensor* t = nullptr;
  const pk_tensor* p() const { return t ? &d : nullptr; }
};

int dtype_tag(at::ScalarType s) {
  switch (s) {
    case at::kByte: return PK_U8;
    case at::kInt: return PK_I32;
    case at::kLong: return PK_I64;
    case at::kFloat: return PK_F32;
    case at::kBFloat16: return PK_BF16;
    default: return -1;
  }
}

bool describe(const at::Tensor& t, pk_tensor* d) {
  const int64_t n = t.dim();
  if (n > PK_MAX_DIMS) {
    PyErr_SetString(PyExc_ValueError, "too many dimensions");
    return false;
  }
  d->dtype = dtype_tag(t.scalar_type());
  if (d->dtype < 0) {
    PyErr_Format(PyExc_TypeError, "unsupported dtype %s", at::toString(t.scalar_type()));
    return false;
  }
  d->data = t.data_ptr();
  d->ndim = (int32_t)n;
  const auto sz = t.sizes();
  const auto st = t.strides();
  for (int64_t i = 0; i < n; i++) d->shape[i] = sz[i], d->stride[i] = st[i];
  return true;
}

// What a tensor argument must be.
enum Want { ANY, CUDA };

bool take(PyObject* o, Arg* a, Want want) {
  if (o == Py_None) return true;
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "expected a tensor or None, got %s", Py_TYPE(o)->tp_name);
    return false;
  }
  a->t = &THPVariable_Unpack(o);
  if (want == CUDA && !a->t->is_cuda()) {
    PyErr_SetString(PyExc_RuntimeError, "pariskv_b200 ops need CUDA tensors; there is no CPU fallback");
    return false;
  }
  return describe(*a->t, &a->d);
}

bool need(PyObject* o, Arg* a, Want want) {
  if (o == Py_None) {
    PyErr_SetString(PyExc_RuntimeError, "pariskv_b200: a required tensor is None");
    return false;
  }
  return take(o, a, want);
}

bool to_i64(PyObject* o, int64_t* v) {
  *v = PyLong_AsLongLong(o);
  return !(*v == -1 && PyErr_Occurred());
}
bool to_f64(PyObject* o, double* v) {
  *v = PyFloat_AsDouble(o);
  return !(*v == -1.0 && PyErr_Occurred());
}

bool arity(Py_ssize_t n, Py_ssize_t want, const char* name) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, n);
  return false;
}

void* stream_of(const at::Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

at::Tensor empty_on(const at::Tensor& like, at::IntArrayRef shape, at::ScalarType dt) {
  return at::detail::empty_cuda(shape, dt, like.device(), std::nullopt);
}

PyObject* raise(int rc) {
  PyErr_Format(PyExc_RuntimeError, "pariskv_b200 error %d: %s", rc, pk_last_error());
  return nullptr;
}

// An output: the tensor passed in, or a fresh one of this shape.
bool output(PyObject* o, Arg* a, at::Tensor* own, const at::Tensor& like, at::IntArrayRef shape, at::ScalarType dt) {
  if (o != Py_None) return take(o, a, CUDA);
  *own = empty_on(like, shape, dt);
  a->t = own;
  return describe(*own, &a->d);
}
PyObject* give(PyObject* o, const Arg& a) {   // the output as the caller's object, or a new reference to a fresh tensor
  if (o != Py_None) return Py_NewRef(o);
  return THPVariable_Wrap(*a.t);
}

// Runs a library call without the GIL (a launch can block on a full queue).
template <typename F>
int without_gil(F&& f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  return rc;
}

// torch.OutOfMemoryError, looked up once.
PyObject* oom_class() {
  static PyObject* cls = nullptr;
  if (!cls) {
    PyObject* m = PyImport_ImportModule("torch");
    cls = m ? PyObject_GetAttrString(m, "OutOfMemoryError") : nullptr;
    Py_XDECREF(m);
    if (!cls) {
      PyErr_Clear();
      cls = PyExc_RuntimeError;
    }
  }
  return cls;
}

// C++ exceptions (an out-of-memory error of the allocator) become Python ones.
#define PK_PY_BEGIN try {
#define PK_PY_END                                       \
  }                                                     \
  catch (const c10::OutOfMemoryError& e) {              \
    PyErr_SetString(oom_class(), e.what_without_backtrace()); \
    return nullptr;                                     \
  }                                                     \
  catch (const std::exception& e) {                     \
    PyErr_SetString(PyExc_RuntimeError, e.what());      \
    return nullptr;                                     \
  }

// Whether the arguments are tensors that the dispatcher would take straight to the CUDA implementation: torch.Tensor or
// Parameter, without gradient, conjugate or negative bit or a wrapper of a transform, and no transform, tracer, dispatch
// or function mode active on this thread.
PyObject* py_plain(PyObject*, PyObject* const* a, Py_ssize_t n) {
  using c10::DispatchKey;
  static const c10::DispatchKeySet modes({DispatchKey::FuncTorchDynamicLayerFrontMode, DispatchKey::FuncTorchDynamicLayerBackMode,
                                          DispatchKey::FuncTorchVmapMode, DispatchKey::VmapMode, DispatchKey::Functionalize,
                                          DispatchKey::Tracer, DispatchKey::PreDispatch, DispatchKey::PythonDispatcher,
                                          DispatchKey::Python, DispatchKey::PythonTLSSnapshot});
  static const c10::DispatchKeySet wrappers({DispatchKey::Python, DispatchKey::PythonTLSSnapshot, DispatchKey::FuncTorchBatched,
                                             DispatchKey::FuncTorchGradWrapper, DispatchKey::BatchedNestedTensor, DispatchKey::Batched,
                                             DispatchKey::Functionalize, DispatchKey::Conjugate, DispatchKey::Negative,
                                             DispatchKey::ZeroTensor});
  if (c10::impl::tls_local_dispatch_key_set().included_.has_any(modes) || at::impl::torch_function_mode_enabled()) Py_RETURN_FALSE;
  for (Py_ssize_t i = 0; i < n; i++) {
    if (!THPVariable_CheckExact(a[i])) Py_RETURN_FALSE;
    const at::Tensor& t = THPVariable_Unpack(a[i]);
    if (t.requires_grad() || t.key_set().has_any(wrappers)) Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
}

PyObject* py_append_encode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 18, "append_encode")) return nullptr;
  PK_PY_BEGIN
  Arg t[16];
  for (int i = 0; i < 16; i++)
    if (!take(a[i], &t[i], (i == 0 || i == 1 || i == 3 || i == 4 || i == 15) ? CUDA : ANY)) return nullptr;
  int64_t sink, interval;
  if (!to_i64(a[16], &sink) || !to_i64(a[17], &interval)) return nullptr;
  if (!t[3].t) return PyErr_SetString(PyExc_TypeError, "window_k is None"), nullptr;
  void* st = stream_of(*t[3].t);
  const int rc = without_gil([&] {
    return pk_append_encode(t[0].p(), t[1].p(), t[2].p(), t[3].p(), t[4].p(), t[5].p(), t[6].p(), t[7].p(), t[8].p(),
                            t[9].p(), t[10].p(), t[11].p(), t[12].p(), t[13].p(), t[14].p(), t[15].p(), sink, interval, st);
  });
  if (rc) return raise(rc);
  Py_RETURN_NONE;
  PK_PY_END
}

// (queries, window_k, window_v, n_window, n_window_dev, n_window_add, store_k, store_v, selected, n_sel, index_offset,
//  scale, out, lse, workspace) -> out
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 15, "sparse_attention")) return nullptr;
  PK_PY_BEGIN
  Arg q, wk, wv, nwd, sk, sv, sel, ns, out, lse, ws;
  at::Tensor own;
  int64_t n_window, n_add, off;
  double scale;
  if (!need(a[0], &q, CUDA) || !take(a[1], &wk, CUDA) || !take(a[2], &wv, CUDA) || !to_i64(a[3], &n_window) ||
      !take(a[4], &nwd, ANY) || !to_i64(a[5], &n_add) || !take(a[6], &sk, ANY) || !take(a[7], &sv, ANY) ||
      !take(a[8], &sel, CUDA) || !take(a[9], &ns, ANY) || !to_i64(a[10], &off) || !to_f64(a[11], &scale) ||
      !output(a[12], &out, &own, *q.t, q.t->sizes(), q.t->scalar_type()) || !take(a[13], &lse, ANY) ||
      !need(a[14], &ws, CUDA))
    return nullptr;
  void* st = stream_of(*q.t);
  const int rc = without_gil([&] {
    return pk_sparse_attention(q.p(), wk.p(), wv.p(), n_window, nwd.p(), n_add, sk.p(), sv.p(), sel.p(), ns.p(), off,
                               (float)scale, out.p(), lse.p(), ws.d.data, (int64_t)ws.t->nbytes(), st);
  });
  if (rc) return raise(rc);
  return give(a[12], out);
  PK_PY_END
}

// (queries, signs, mag_centers, codebook, key_block_weight, key_4bit, cluster_key_counts, C, K, tier_counts or None,
//  kv_len, schedule address or 0, phase, local_hist, shard_hist, world, rank, final, n_sel, cand, n_cand, scores,
//  q_blocks, q_norm, query_avg, workspace, queries_settled)
// -> (final, n_sel); final and n_sel are made here when they are None, K > 0 and phase != 1.
PyObject* py_retrieve(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 27, "retrieve_ex")) return nullptr;
  PK_PY_BEGIN
  Arg t[7], kv, lh, sh, fin, ns, cand, nc, sc, qb, qn, qa, ws;
  at::Tensor own_f, own_n;
  for (int i = 0; i < 7; i++)
    if (!need(a[i], &t[i], (i == 0 || i >= 3) ? CUDA : ANY)) return nullptr;
  int64_t C, K, sched, phase, world, rank, settled, tiers[8];
  int n_tiers = 0;
  if (!to_i64(a[7], &C) || !to_i64(a[8], &K)) return nullptr;
  if (a[9] != Py_None) {
    PyObject* seq = PySequence_Fast(a[9], "tier_counts must be a sequence");
    if (!seq) return nullptr;
    const Py_ssize_t m = PySequence_Fast_GET_SIZE(seq);
    bool ok = true;
    for (Py_ssize_t i = 0; i < m && i < 8 && ok; i++) ok = to_i64(PySequence_Fast_GET_ITEM(seq, i), &tiers[i]);
    Py_DECREF(seq);
    if (!ok) return nullptr;
    n_tiers = (int)m;
  }
  if (!take(a[10], &kv, ANY) || !to_i64(a[11], &sched) || !to_i64(a[12], &phase) || !take(a[13], &lh, ANY) ||
      !take(a[14], &sh, ANY) || !to_i64(a[15], &world) || !to_i64(a[16], &rank))
    return nullptr;
  const bool selects = K > 0 && phase != 1;
  if (t[3].d.ndim != 4) return PyErr_SetString(PyExc_ValueError, "codebook must be [bs,H,16,N]"), nullptr;
  const int64_t bs = t[3].d.shape[0], H = t[3].d.shape[1];
  if (selects) {
    if (!output(a[17], &fin, &own_f, *t[3].t, {bs, H, K}, at::kLong) || !output(a[18], &ns, &own_n, *t[3].t, {bs, H}, at::kInt))
      return nullptr;
  } else if (!take(a[17], &fin, ANY) || !take(a[18], &ns, ANY)) {
    return nullptr;
  }
  if (!take(a[19], &cand, ANY) || !take(a[20], &nc, ANY) || !take(a[21], &sc, ANY) || !take(a[22], &qb, ANY) ||
      !take(a[23], &qn, ANY) || !take(a[24], &qa, ANY) || !need(a[25], &ws, CUDA) || !to_i64(a[26], &settled))
    return nullptr;
  pk_retrieve_args r = {};
  r.queries = t[0].p(), r.signs = t[1].p(), r.mag_centers = t[2].p(), r.codebook = t[3].p(), r.key_block_weight = t[4].p();
  r.key_4bit = t[5].p(), r.cluster_key_counts = t[6].p();
  r.tier_counts = a[9] != Py_None ? tiers : nullptr, r.n_tiers = n_tiers;
  r.phase = (int32_t)phase, r.C = C, r.K = K, r.kv_len = kv.p();
  r.schedule = reinterpret_cast<const pk_zone_schedule*>((uintptr_t)sched);
  r.local_hist = lh.p(), r.shard_hist = sh.p(), r.world = (int32_t)world, r.rank = (int32_t)rank;
  r.final_indices = fin.p(), r.n_sel = ns.p(), r.cand = cand.p(), r.n_cand = nc.p(), r.scores_f32 = sc.p();
  r.q_blocks = qb.p(), r.q_norm = qn.p(), r.query_avg = qa.p();
  r.workspace = ws.d.data, r.workspace_bytes = (int64_t)ws.t->nbytes();
  r.queries_settled = settled != 0;
  void* st = stream_of(*t[3].t);
  const int rc = without_gil([&] { return pk_retrieve_ex(&r, st); });
  if (rc) return raise(rc);
  PyObject* f = fin.t ? give(a[17], fin) : Py_NewRef(Py_None);
  PyObject* s = ns.t ? give(a[18], ns) : Py_NewRef(Py_None);
  PyObject* both = f && s ? PyTuple_Pack(2, f, s) : nullptr;
  Py_XDECREF(f);
  Py_XDECREF(s);
  return both;
  PK_PY_END
}

// k, v, signs, window_k, window_v, win_codes, win_weight, win_4bit, win_vnorm, codebook, block_weight, packed_4bit,
// value_norm, cluster_counts, rows, state, b, sink, local
PyObject* py_prefill_sample(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 19, "prefill_sample")) return nullptr;
  PK_PY_BEGIN
  Arg t[16];
  for (int i = 0; i < 16; i++)
    if (!take(a[i], &t[i], i == 12 || i == 14 ? ANY : CUDA)) return nullptr;
  int64_t b, sink, local;
  if (!to_i64(a[16], &b) || !to_i64(a[17], &sink) || !to_i64(a[18], &local)) return nullptr;
  if (!t[0].t) return PyErr_SetString(PyExc_TypeError, "k is None"), nullptr;
  void* st = stream_of(*t[0].t);
  const int rc = without_gil([&] {
    return pk_prefill_sample(t[0].p(), t[1].p(), t[2].p(), t[3].p(), t[4].p(), t[5].p(), t[6].p(), t[7].p(), t[8].p(), t[9].p(),
                             t[10].p(), t[11].p(), t[12].p(), t[13].p(), t[14].p(), t[15].p(), b, sink, local, st);
  });
  if (rc) return raise(rc);
  Py_RETURN_NONE;
  PK_PY_END
}

// src (device), dst (device or pinned host)
PyObject* py_copy_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 2, "copy_rows")) return nullptr;
  PK_PY_BEGIN
  Arg src, dst;
  if (!need(a[0], &src, CUDA) || !need(a[1], &dst, ANY)) return nullptr;
  void* st = stream_of(*src.t);
  const int rc = without_gil([&] { return pk_copy_rows(src.p(), dst.p(), st); });
  if (rc) return raise(rc);
  Py_RETURN_NONE;
  PK_PY_END
}

// keys, signs, codebook, block_weight, packed_4bit, cluster_counts
PyObject* py_encode_keys(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 6, "encode_keys")) return nullptr;
  PK_PY_BEGIN
  Arg t[6];
  for (int i = 0; i < 6; i++)
    if (!take(a[i], &t[i], i < 2 ? CUDA : ANY)) return nullptr;
  if (!t[0].t) return PyErr_SetString(PyExc_TypeError, "keys is None"), nullptr;
  void* st = stream_of(*t[0].t);
  const int rc = without_gil([&] { return pk_encode_keys(t[0].p(), t[1].p(), t[2].p(), t[3].p(), t[4].p(), t[5].p(), st); });
  if (rc) return raise(rc);
  Py_RETURN_NONE;
  PK_PY_END
}

// queries, kv_heads, signs, want_avg -> (q_blocks, q_norm) or (q_blocks, q_norm, query_avg)
PyObject* py_query_prep(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 4, "query_prep")) return nullptr;
  PK_PY_BEGIN
  Arg q, s, qb, qn, qa;
  at::Tensor tb, tn, ta;
  int64_t H, avg;
  if (!need(a[0], &q, CUDA) || !to_i64(a[1], &H) || !need(a[2], &s, CUDA) || !to_i64(a[3], &avg)) return nullptr;
  const int64_t bs = q.d.shape[0];
  if (!output(Py_None, &qb, &tb, *q.t, {bs, H, 16, 8}, at::kBFloat16) || !output(Py_None, &qn, &tn, *q.t, {bs, H, 1}, at::kBFloat16) ||
      (avg && !output(Py_None, &qa, &ta, *q.t, {bs, H, 128}, at::kBFloat16)))
    return nullptr;
  void* st = stream_of(*q.t);
  const int rc = without_gil([&] { return pk_query_prep(q.p(), s.p(), qb.p(), qn.p(), qa.p(), st); });
  if (rc) return raise(rc);
  if (avg) return Py_BuildValue("(NNN)", THPVariable_Wrap(tb), THPVariable_Wrap(tn), THPVariable_Wrap(ta));
  return Py_BuildValue("(NN)", THPVariable_Wrap(tb), THPVariable_Wrap(tn));
  PK_PY_END
}

PyObject* py_rank_clusters(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 1, "rank_clusters")) return nullptr;
  PK_PY_BEGIN
  Arg q, o;
  at::Tensor own;
  if (!need(a[0], &q, CUDA)) return nullptr;
  if (!output(Py_None, &o, &own, *q.t, {q.d.shape[0], q.d.shape[1], 16, 256}, at::kLong)) return nullptr;
  void* st = stream_of(*q.t);
  const int rc = without_gil([&] { return pk_rank_clusters(q.p(), o.p(), st); });
  if (rc) return raise(rc);
  return THPVariable_Wrap(own);
  PK_PY_END
}

// sorted_cluster_ids, cluster_key_counts, codebook, tier_counts, cache_cnt or None, workspace -> cache_cnt
PyObject* py_collision_fused(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 6, "collision_fused")) return nullptr;
  PK_PY_BEGIN
  Arg ids, cnt, cb, out, ws;
  at::Tensor own;
  if (!need(a[0], &ids, CUDA) || !need(a[1], &cnt, CUDA) || !need(a[2], &cb, CUDA)) return nullptr;
  if (cb.d.ndim != 4) return PyErr_SetString(PyExc_ValueError, "codebook must be [bs,H,B,N]"), nullptr;
  if (!output(a[4], &out, &own, *cb.t, {cb.d.shape[0], cb.d.shape[1], cb.d.shape[3]}, at::kInt) || !need(a[5], &ws, CUDA))
    return nullptr;
  PyObject* seq = PySequence_Fast(a[3], "tier_counts must be a sequence");
  if (!seq) return nullptr;
  const Py_ssize_t m = PySequence_Fast_GET_SIZE(seq);
  int64_t tiers[8] = {};
  bool ok = true;
  for (Py_ssize_t i = 0; i < m && i < 8 && ok; i++) ok = to_i64(PySequence_Fast_GET_ITEM(seq, i), &tiers[i]);
  Py_DECREF(seq);
  if (!ok) return nullptr;
  void* st = stream_of(*cb.t);
  const int rc = without_gil([&] {
    return pk_collision_fused(ids.p(), cnt.p(), cb.p(), tiers, (int)m, out.p(), ws.d.data, (int64_t)ws.t->nbytes(), st);
  });
  if (rc) return raise(rc);
  return give(a[4], out);
  PK_PY_END
}

// input [rows, L], k, order -> [rows, k]
PyObject* py_topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 3, "topk")) return nullptr;
  PK_PY_BEGIN
  Arg x, o;
  at::Tensor own;
  int64_t k, order;
  if (!need(a[0], &x, CUDA) || !to_i64(a[1], &k) || !to_i64(a[2], &order)) return nullptr;
  // any number of leading dimensions: the rows of a contiguous tensor are the rows of its 2-D view
  pk_tensor x2 = x.d;
  at::DimVector shape(x.t->sizes());
  if (x.d.ndim < 1) return PyErr_SetString(PyExc_ValueError, "input must have a dimension to select from"), nullptr;
  if (x.d.ndim != 2) {
    int64_t rows = 1;
    for (int i = 0; i + 1 < x.d.ndim; i++) rows *= x.d.shape[i];
    x2.ndim = 2;
    x2.shape[0] = rows, x2.shape[1] = x.d.shape[x.d.ndim - 1];
    x2.stride[0] = x2.shape[1], x2.stride[1] = x.d.stride[x.d.ndim - 1];
  }
  shape.back() = k < 0 ? 0 : k;
  if (!output(Py_None, &o, &own, *x.t, shape, at::kLong)) return nullptr;
  pk_tensor o2 = o.d;
  o2.ndim = 2;
  o2.shape[0] = x2.shape[0], o2.shape[1] = shape.back(), o2.stride[0] = shape.back(), o2.stride[1] = 1;
  void* st = stream_of(*x.t);
  const int rc = without_gil([&] { return pk_topk(&x2, k, &o2, (int)order, st); });
  if (rc) return raise(rc);
  return THPVariable_Wrap(own);
  PK_PY_END
}

PyObject* py_final_topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 3, "final_topk")) return nullptr;
  PK_PY_BEGIN
  Arg s, c, o;
  at::Tensor own;
  int64_t K;
  if (!need(a[0], &s, CUDA) || !need(a[1], &c, CUDA) || !to_i64(a[2], &K)) return nullptr;
  if (!output(Py_None, &o, &own, *s.t, {s.d.shape[0], s.d.shape[1], K}, at::kLong)) return nullptr;
  void* st = stream_of(*s.t);
  const int rc = without_gil([&] { return pk_final_topk(s.p(), c.p(), K, o.p(), st); });
  if (rc) return raise(rc);
  return THPVariable_Wrap(own);
  PK_PY_END
}

// sl_logits, cand_scores, cand_scale, sl_vnorm, cand_indices, cand_vnorm, value_norm, sink, threshold, K_out, min_k,
// max_k, adaptive_k or None, topk_indices or None -> (adaptive_k, topk_indices)
PyObject* py_adaptive_topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 14, "adaptive_topk")) return nullptr;
  PK_PY_BEGIN
  Arg sl, sc, slv, ci, cv, vn, ak, ti;
  at::Tensor oa, ot;
  double scale, thr;
  int64_t sink, K, lo, hi;
  if (!need(a[0], &sl, CUDA) || !need(a[1], &sc, CUDA) || !to_f64(a[2], &scale) || !need(a[3], &slv, CUDA) ||
      !need(a[4], &ci, CUDA) || !take(a[5], &cv, ANY) || !take(a[6], &vn, ANY) || !to_i64(a[7], &sink) ||
      !to_f64(a[8], &thr) || !to_i64(a[9], &K) || !to_i64(a[10], &lo) || !to_i64(a[11], &hi))
    return nullptr;
  const int64_t bs = sl.d.shape[0], H = sl.d.shape[1];
  if (!output(a[12], &ak, &oa, *sl.t, {bs, H}, at::kLong) || !output(a[13], &ti, &ot, *sl.t, {bs, H, K}, at::kLong)) return nullptr;
  void* st = stream_of(*sl.t);
  const int rc = without_gil([&] {
    return pk_adaptive_topk(sl.p(), sc.p(), (float)scale, slv.p(), ci.p(), cv.p(), vn.p(), sink, (float)thr, K, lo, hi,
                            ak.p(), ti.p(), st);
  });
  if (rc) return raise(rc);
  return Py_BuildValue("(NN)", give(a[12], ak), give(a[13], ti));
  PK_PY_END
}

// query_avg, window_k, n_window or None, S, cand_scores, n_cand or None, scale, sl_vnorm, cand_indices, value_norm,
// threshold, K_out, min_k, max_k -> (adaptive_k, topk_indices, n_sel, sl_logits)
PyObject* py_adaptive_select(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 14, "adaptive_select")) return nullptr;
  PK_PY_BEGIN
  Arg qa, wk, nw, sl, sc, nc, slv, ci, vn, ak, ti, ns;
  at::Tensor oa, ot, os, ol;
  double scale, thr;
  int64_t S, K, lo, hi;
  if (!need(a[0], &qa, CUDA) || !need(a[1], &wk, CUDA) || !take(a[2], &nw, CUDA) || !to_i64(a[3], &S) ||
      !need(a[4], &sc, CUDA) || !take(a[5], &nc, CUDA) || !to_f64(a[6], &scale) || !need(a[7], &slv, CUDA) ||
      !need(a[8], &ci, CUDA) || !need(a[9], &vn, CUDA) || !to_f64(a[10], &thr) || !to_i64(a[11], &K) ||
      !to_i64(a[12], &lo) || !to_i64(a[13], &hi))
    return nullptr;
  const int64_t bs = qa.d.shape[0], H = qa.d.shape[1];
  if (!output(Py_None, &ak, &oa, *qa.t, {bs, H}, at::kLong) || !output(Py_None, &ti, &ot, *qa.t, {bs, H, K}, at::kLong) ||
      !output(Py_None, &ns, &os, *qa.t, {bs, H}, at::kInt) || !output(Py_None, &sl, &ol, *qa.t, {bs, H, S}, at::kFloat))
    return nullptr;
  void* st = stream_of(*qa.t);
  const int rc = without_gil([&] {
    return pk_adaptive_select(qa.p(), wk.p(), nw.p(), sl.p(), sc.p(), nc.p(), (float)scale, slv.p(), ci.p(), vn.p(), (float)thr, K,
                              lo, hi, ak.p(), ti.p(), ns.p(), st);
  });
  if (rc) return raise(rc);
  return Py_BuildValue("(NNNN)", give(Py_None, ak), give(Py_None, ti), give(Py_None, ns), give(Py_None, sl));
  PK_PY_END
}

// coarse_indices, key_4bit, key_block_weight, q_blocks, q_norm, mag_centers, approx or None (made here), scores_f32,
// v4b -> approx
PyObject* py_rerank(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 9, "rerank")) return nullptr;
  PK_PY_BEGIN
  Arg t[6], ap, s32, v4;
  at::Tensor own;
  for (int i = 0; i < 6; i++)
    if (!need(a[i], &t[i], CUDA)) return nullptr;
  if (!output(a[6], &ap, &own, *t[0].t, t[0].t->sizes(), at::kBFloat16) || !take(a[7], &s32, ANY) || !take(a[8], &v4, ANY))
    return nullptr;
  void* st = stream_of(*t[0].t);
  const int rc = without_gil([&] {
    return pk_rerank(t[0].p(), t[1].p(), t[2].p(), t[3].p(), t[4].p(), t[5].p(), ap.p(), s32.p(), v4.p(), st);
  });
  if (rc) return raise(rc);
  return give(a[6], ap);
  PK_PY_END
}

// src_k, src_v (host or device), selected_indices, dst_k, dst_v
PyObject* py_h2d_gather_kv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 5, "h2d_gather_kv")) return nullptr;
  PK_PY_BEGIN
  Arg t[5];
  for (int i = 0; i < 5; i++)
    if (!need(a[i], &t[i], i >= 2 ? CUDA : ANY)) return nullptr;
  void* st = stream_of(*t[3].t);
  const int rc = without_gil([&] { return pk_h2d_gather_kv(t[0].p(), t[1].p(), t[2].p(), t[3].p(), t[4].p(), st); });
  if (rc) return raise(rc);
  Py_RETURN_NONE;
  PK_PY_END
}

// qkv, weight, cos, sin, eps, out or None -> out [B, heads, 128]
PyObject* py_qk_norm_rope(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 6, "qk_norm_rope")) return nullptr;
  PK_PY_BEGIN
  Arg x, w, c, s, o;
  at::Tensor own;
  double eps;
  if (!need(a[0], &x, CUDA) || !need(a[1], &w, CUDA) || !need(a[2], &c, CUDA) || !need(a[3], &s, CUDA) || !to_f64(a[4], &eps))
    return nullptr;
  if (!output(a[5], &o, &own, *x.t, {x.d.shape[0], w.d.shape[0], 128}, at::kBFloat16)) return nullptr;
  void* st = stream_of(*x.t);
  const int rc = without_gil([&] { return pk_qk_norm_rope(x.p(), w.p(), c.p(), s.p(), o.p(), eps, st); });
  if (rc) return raise(rc);
  return give(a[5], o);
  PK_PY_END
}

// a, residual or None, weight, eps -> (h, x)
PyObject* py_add_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 4, "add_rmsnorm")) return nullptr;
  PK_PY_BEGIN
  Arg x, r, w, h, y;
  at::Tensor th, ty;
  double eps;
  if (!need(a[0], &x, CUDA) || !take(a[1], &r, ANY) || !need(a[2], &w, CUDA) || !to_f64(a[3], &eps)) return nullptr;
  if (!output(Py_None, &h, &th, *x.t, x.t->sizes(), x.t->scalar_type()) ||
      !output(Py_None, &y, &ty, *x.t, x.t->sizes(), x.t->scalar_type()))
    return nullptr;
  void* st = stream_of(*x.t);
  const int rc = without_gil([&] { return pk_add_rmsnorm(x.p(), r.p(), w.p(), h.p(), y.p(), eps, st); });
  if (rc) return raise(rc);
  return Py_BuildValue("(NN)", THPVariable_Wrap(th), THPVariable_Wrap(ty));
  PK_PY_END
}

PyObject* py_silu_mul(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 1, "silu_mul")) return nullptr;
  PK_PY_BEGIN
  Arg x, o;
  at::Tensor own;
  if (!need(a[0], &x, CUDA)) return nullptr;
  if (x.d.ndim != 2) return PyErr_SetString(PyExc_ValueError, "gate_up must be [B, 2F]"), nullptr;
  if (!output(Py_None, &o, &own, *x.t, {x.d.shape[0], x.d.shape[1] / 2}, at::kBFloat16)) return nullptr;
  void* st = stream_of(*x.t);
  const int rc = without_gil([&] { return pk_silu_mul(x.p(), o.p(), st); });
  if (rc) return raise(rc);
  return THPVariable_Wrap(own);
  PK_PY_END
}

// weight, x, gated -> [1, O] or [1, O / 2]
PyObject* py_gemv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 3, "gemv")) return nullptr;
  PK_PY_BEGIN
  Arg w, x, o;
  at::Tensor own;
  int64_t gated;
  if (!need(a[0], &w, CUDA) || !need(a[1], &x, CUDA) || !to_i64(a[2], &gated)) return nullptr;
  const int64_t O = w.d.ndim > 0 ? w.d.shape[0] : 0;
  if (!output(Py_None, &o, &own, *x.t, {1, gated ? O / 2 : O}, at::kBFloat16)) return nullptr;
  void* st = stream_of(*x.t);
  const int rc = without_gil([&] { return pk_gemv(w.p(), x.p(), o.p(), gated != 0, st); });
  if (rc) return raise(rc);
  return THPVariable_Wrap(own);
  PK_PY_END
}

PyObject* py_attention_workspace_bytes(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 3, "attention_workspace_bytes")) return nullptr;
  int64_t v[3];
  for (int i = 0; i < 3; i++)
    if (!to_i64(a[i], &v[i])) return nullptr;
  return PyLong_FromLongLong(pk_attention_workspace_bytes(v[0], v[1], v[2]));
}

PyObject* py_retrieve_workspace_bytes(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 4, "retrieve_workspace_bytes")) return nullptr;
  int64_t v[4];
  for (int i = 0; i < 4; i++)
    if (!to_i64(a[i], &v[i])) return nullptr;
  return PyLong_FromLongLong(pk_retrieve_workspace_bytes(v[0], v[1], v[2], v[3]));
}

#define PK_METHOD(name, fn) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    PK_METHOD("plain", py_plain),
    PK_METHOD("append_encode", py_append_encode),
    PK_METHOD("sparse_attention", py_attention),
    PK_METHOD("retrieve_ex", py_retrieve),
    PK_METHOD("prefill_sample", py_prefill_sample),
    PK_METHOD("copy_rows", py_copy_rows),
    PK_METHOD("encode_keys", py_encode_keys),
    PK_METHOD("query_prep", py_query_prep),
    PK_METHOD("rank_clusters", py_rank_clusters),
    PK_METHOD("collision_fused", py_collision_fused),
    PK_METHOD("topk", py_topk),
    PK_METHOD("final_topk", py_final_topk),
    PK_METHOD("adaptive_topk", py_adaptive_topk),
    PK_METHOD("adaptive_select", py_adaptive_select),
    PK_METHOD("rerank", py_rerank),
    PK_METHOD("h2d_gather_kv", py_h2d_gather_kv),
    PK_METHOD("qk_norm_rope", py_qk_norm_rope),
    PK_METHOD("add_rmsnorm", py_add_rmsnorm),
    PK_METHOD("silu_mul", py_silu_mul),
    PK_METHOD("gemv", py_gemv),
    PK_METHOD("attention_workspace_bytes", py_attention_workspace_bytes),
    PK_METHOD("retrieve_workspace_bytes", py_retrieve_workspace_bytes),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Native binding of libpariskv_b200.so.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};
}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
