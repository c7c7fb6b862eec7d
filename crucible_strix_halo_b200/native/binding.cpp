// _binding: the per-call host path of layers.py in C++.  A step of one session reads some forty tensor addresses and
// attributes; through ctypes that, the stream look-up and the outputs took 15 us per GDN call and 24 us per QSA call, three
// times their launches.  Here the same objects (weights, sessions, plans, span dicts) are read with the CPython API and the
// argument structs of include/crucible_attn.h are filled on the stack.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>
#include <vector>
#include "../../include/crucible_attn.h"

namespace {

// ---- names, interned once ---------------------------------------------------------------------------------------
#define NAMES(X)                                                                                                        \
  X(g) X(conv) X(A_log) X(dt_bias) X(gamma) X(ab) X(suh) X(state) X(hist) X(pend) X(pend_rows) X(session) X(qkv) X(z) X(x) X(pos0) \
  X(replay) X(commit) X(q) X(k) X(v) X(idx) X(q_norm1) X(k_norm1) X(iq_norm1) X(ik_norm1) X(rope) X(ik_raw) X(ik_pool) X(raw_slots) \
  X(scores) X(sstride) X(sel) X(nsel) X(w) X(fmt) X(scratch) X(workspace) X(out) X(raw_y) X(in_dtype) X(q_hi) X(data_ptr)
#define DECLARE(n) PyObject* s_##n;
NAMES(DECLARE)

struct Error {};                                     // a Python exception is set

// A new reference that is dropped at the end of the scope.
struct Ref {
  PyObject* p;
  explicit Ref(PyObject* o) : p(o) { if (!p) throw Error(); }
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  operator PyObject*() const { return p; }
};

PyObject* item(PyObject* dict, PyObject* name) {     // borrowed; a missing key is a KeyError
  PyObject* o = PyDict_GetItemWithError(dict, name);
  if (!o) {
    if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, name);
    throw Error();
  }
  return o;
}
long as_long(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw Error();
  return v;
}
long long_attr(PyObject* o, PyObject* name) { Ref r(PyObject_GetAttr(o, name)); return as_long(r); }
long item_or(PyObject* dict, PyObject* name, long otherwise) {
  PyObject* o = PyDict_GetItemWithError(dict, name);
  if (!o) { if (PyErr_Occurred()) throw Error(); return otherwise; }
  return as_long(o);
}
// Address of a tensor (or of anything with data_ptr()); None is null.
void* address(PyObject* o) {
  if (o == Py_None) return nullptr;
  if (THPVariable_Check(o)) return THPVariable_Unpack(o).data_ptr();
  Ref r(PyObject_CallMethodNoArgs(o, s_data_ptr));
  void* p = PyLong_AsVoidPtr(r);
  if (!p && PyErr_Occurred()) throw Error();
  return p;
}
template <typename T>
void attr(T*& to, PyObject* o, PyObject* name) { Ref r(PyObject_GetAttr(o, name)); to = static_cast<T*>(address(r)); }
const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) { PyErr_SetString(PyExc_TypeError, "a torch tensor is needed"); throw Error(); }
  return THPVariable_Unpack(o);
}
cr_geometry geometry(PyObject* w) {                  // w.g, a ctypes structure
  Ref g(PyObject_GetAttr(w, s_g));
  Py_buffer b;
  if (PyObject_GetBuffer(g, &b, PyBUF_SIMPLE) != 0) throw Error();
  cr_geometry out{};
  if (b.len == (Py_ssize_t)sizeof(out)) out = *static_cast<const cr_geometry*>(b.buf);
  PyBuffer_Release(&b);
  if (!out.kv_heads) { PyErr_SetString(PyExc_TypeError, "weights need a Geometry"); throw Error(); }
  return out;
}
// A call into the library, without the interpreter lock: other host threads go on meanwhile, on streams or GPUs of their own.
// The argument structs are filled and nothing of Python is touched until the lock is back, also when `f` throws.
template <typename F>
cr_status unlocked(F&& f) {
  struct Lock {
    PyThreadState* state = PyEval_SaveThread();
    ~Lock() { PyEval_RestoreThread(state); }
  } released;
  return f();
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }   // throws without a usable GPU
at::ScalarType out_type(long fmt) {
  return fmt == CR_OUT_RAW_F32 ? at::kFloat : fmt == CR_OUT_RAW_BF16 ? at::kBFloat16 : at::kHalf;
}
PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
void check(cr_status s) {
  if (s == CR_OK) return;
  Ref capi(PyImport_ImportModule("crucible_strix_halo_b200.capi")), type(PyObject_GetAttrString(capi, "CrError"));
  Ref e(PyObject_CallFunction(type, "is", (int)s, cr_last_error()));
  PyErr_SetObject(type, e);
  throw Error();
}
// The i-th output: given by the caller, or new.  The list takes it.
void* output(PyObject* list, PyObject* given, Py_ssize_t i, at::IntArrayRef shape, at::ScalarType type, const at::Tensor& like) {
  PyObject* o;
  if (given != Py_None) {
    o = PySequence_GetItem(given, i);
    if (!o) throw Error();
  } else {
    o = wrap(at::empty(shape, at::TensorOptions().dtype(type).device(like.device())));
  }
  PyList_SET_ITEM(list, i, o);
  return address(o);
}

template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const Error&) {
    return nullptr;
  } catch (...) {                                    // the exception that torch's own functions give for it
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

// ---- argument structs --------------------------------------------------------------------------------------------
void gdn_weights(cr_gdn_args& a, PyObject* w) {
  attr(a.ab, w, s_ab); attr(a.conv, w, s_conv); attr(a.A_log, w, s_A_log); attr(a.dt_bias, w, s_dt_bias);
  attr(a.gamma, w, s_gamma); attr(a.suh_out, w, s_suh);
}
void gdn_session(cr_gdn_args& a, PyObject* s) { attr(a.hist, s, s_hist); attr(a.state, s, s_state); attr(a.pend, s, s_pend); }

void qsa_weights(cr_qsa_args& a, PyObject* w) {
  attr(a.q_norm1, w, s_q_norm1); attr(a.k_norm1, w, s_k_norm1); attr(a.iq_norm1, w, s_iq_norm1); attr(a.ik_norm1, w, s_ik_norm1);
  attr(a.suh_o, w, s_suh); attr(a.rope, w, s_rope);
}
void qsa_session(cr_qsa_args& a, PyObject* s) {
  attr(a.c.k, s, s_k); attr(a.c.v, s, s_v); attr(a.c.ik_raw, s, s_ik_raw); attr(a.c.ik_pool, s, s_ik_pool);
  a.c.raw_slots = (int)long_attr(s, s_raw_slots);
  attr(a.scores, s, s_scores); attr(a.sel, s, s_sel); attr(a.nsel, s, s_nsel);
  a.sstride = (int)long_attr(s, s_sstride);
}

// ---- calls ---------------------------------------------------------------------------------------------------------
PyObject* gdn_step(PyObject*, PyObject* args) {      // (weights, spans, fmt, outs or None) -> outputs
  return guarded([&]() -> PyObject* {
    PyObject *w, *spans, *given;
    int fmt;
    if (!PyArg_ParseTuple(args, "OOiO", &w, &spans, &fmt, &given)) throw Error();
    Ref list(PySequence_Fast(spans, "spans must be a sequence"));
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(list.p);
    const cr_geometry g = geometry(w);
    const int64_t W = (int64_t)g.gdn_vheads * 128;
    cr_gdn_args base{};
    gdn_weights(base, w);
    std::vector<cr_gdn_args> a(n, base);
    Ref outs(PyList_New(n));
    long pend_rows = 0;
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* sp = PySequence_Fast_GET_ITEM(list.p, i);
      PyObject* s = item(sp, s_session);
      const at::Tensor& qkv = tensor(item(sp, s_qkv));
      const int64_t R = qkv.size(0);
      if (i == 0) pend_rows = long_attr(s, s_pend_rows);
      a[i].qkv = qkv.data_ptr();
      a[i].z = address(item(sp, s_z));
      a[i].x = static_cast<const float*>(address(item(sp, s_x)));
      gdn_session(a[i], s);
      a[i].pos0 = (int)as_long(item(sp, s_pos0));
      a[i].R = (int)R;
      a[i].replay = (int)item_or(sp, s_replay, 0);
      a[i].commit = (int)item_or(sp, s_commit, R);
      a[i].out = output(outs, given, i, {R, W}, out_type(fmt), qkv);
    }
    void* const st = stream();
    check(unlocked([&] { return cr_gdn_step(&g, a.data(), (int)n, (int)pend_rows, (cr_out_format)fmt, st); }));
    Py_INCREF(outs.p);
    return outs.p;
  });
}

PyObject* qsa_step(PyObject*, PyObject* args) {      // (plan, spans, want_context, outs or None) -> outputs or (outputs, contexts)
  return guarded([&]() -> PyObject* {
    PyObject *plan, *spans, *given;
    int want;
    if (!PyArg_ParseTuple(args, "OOpO", &plan, &spans, &want, &given)) throw Error();
    Ref list(PySequence_Fast(spans, "spans must be a sequence"));
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(list.p);
    Ref w(PyObject_GetAttr(plan, s_w));
    const cr_geometry g = geometry(w);
    const long fmt = long_attr(plan, s_fmt);
    cr_qsa_args base{};
    qsa_weights(base, w);
    std::vector<cr_qsa_args> a(n, base);
    Ref outs(PyList_New(n)), contexts(PyList_New(want ? n : 0));
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* sp = PySequence_Fast_GET_ITEM(list.p, i);
      const at::Tensor& q = tensor(item(sp, s_q));
      const int64_t R = q.size(0);
      a[i].q = static_cast<float*>(q.data_ptr());
      a[i].k = static_cast<const float*>(address(item(sp, s_k)));
      a[i].v = static_cast<const float*>(address(item(sp, s_v)));
      a[i].idx = static_cast<float*>(address(item(sp, s_idx)));
      qsa_session(a[i], item(sp, s_session));
      a[i].pos0 = (int)as_long(item(sp, s_pos0));
      a[i].R = (int)R;
      a[i].out = output(outs, given, i, {R, (int64_t)g.q_heads * 256}, out_type(fmt), q);
      if (want) a[i].context = static_cast<float*>(output(contexts, Py_None, i, {R, (int64_t)g.q_heads, 256}, at::kFloat, q));
    }
    Ref scratch(PyObject_GetAttr(plan, s_scratch));
    const at::Tensor& sc = tensor(scratch);
    void *const st = stream(), *const at = sc.data_ptr();
    const size_t bytes = (size_t)sc.numel();
    check(unlocked([&] { return cr_qsa_step(&g, a.data(), (int)n, at, bytes, (cr_out_format)fmt, st); }));
    if (want) return PyTuple_Pack(2, outs.p, contexts.p);
    Py_INCREF(outs.p);
    return outs.p;
  });
}

PyObject* gdn_prefill(PyObject*, PyObject* args) {   // (plan, session, qkv, z, ab_logits, pos0, algo)
  return guarded([&]() -> PyObject* {
    PyObject *plan, *s, *qkv, *z, *ab;
    int pos0, algo;
    if (!PyArg_ParseTuple(args, "OOOOOii", &plan, &s, &qkv, &z, &ab, &pos0, &algo)) throw Error();
    Ref w(PyObject_GetAttr(plan, s_w)), ws(PyObject_GetAttr(plan, s_workspace));
    const cr_geometry g = geometry(w);
    cr_gdn_prefill_args a{};
    gdn_weights(a.input, w);
    gdn_session(a.input, s);
    const at::Tensor& t = tensor(qkv);
    a.input.qkv = t.data_ptr();
    a.input.z = address(z);
    a.input.pos0 = pos0;
    a.input.R = a.input.commit = (int)t.size(0);
    attr(a.input.out, plan, s_out);
    a.ab_logits = address(ab);
    a.in_dtype = (cr_in_dtype)long_attr(plan, s_in_dtype);
    const at::Tensor& wst = tensor(ws);
    a.workspace = wst.data_ptr();
    a.workspace_bytes = (size_t)wst.numel();
    attr(a.raw_y, plan, s_raw_y);
    const cr_out_format fmt = (cr_out_format)long_attr(plan, s_fmt);
    void* const st = stream();
    check(unlocked([&] { return cr_gdn_prefill(&g, &a, (cr_gdn_algo)algo, fmt, st); }));
    return PyObject_GetAttr(plan, s_out);
  });
}

PyObject* qsa_prefill(PyObject*, PyObject* args) {   // (plan, session, q, k, v, idx, pos0, skip, context or None)
  return guarded([&]() -> PyObject* {
    PyObject *plan, *s, *q, *k, *v, *idx, *context;
    int pos0, skip;
    if (!PyArg_ParseTuple(args, "OOOOOOiiO", &plan, &s, &q, &k, &v, &idx, &pos0, &skip, &context)) throw Error();
    Ref w(PyObject_GetAttr(plan, s_w)), scratch(PyObject_GetAttr(plan, s_scratch)), out(PyObject_GetAttr(plan, s_out));
    const cr_geometry g = geometry(w);
    cr_qsa_prefill_args a{};
    qsa_weights(a.input, w);
    qsa_session(a.input, s);
    const at::Tensor& qt = tensor(q);
    a.input.q = static_cast<float*>(qt.data_ptr());
    a.input.k = static_cast<const float*>(address(k));
    a.input.v = static_cast<const float*>(address(v));
    a.input.idx = static_cast<float*>(address(idx));
    a.input.out = address(out);
    a.input.context = static_cast<float*>(address(context));
    a.input.pos0 = pos0;
    a.input.R = (int)qt.size(0);
    attr(a.q_hi, plan, s_q_hi);
    const at::Tensor& sc = tensor(scratch);
    a.scratch = sc.data_ptr();
    a.scratch_bytes = (size_t)sc.numel();
    const cr_out_format fmt = (cr_out_format)long_attr(plan, s_fmt);
    void* const st = stream();
    check(unlocked([&] { return cr_qsa_prefill(&g, &a, skip, fmt, st); }));
    return wrap(tensor(out).narrow(0, 0, qt.size(0)));
  });
}

PyObject* proj_gemm(PyObject*, PyObject* args) {     // (x, w, outs)
  return guarded([&]() -> PyObject* {
    PyObject *x, *w, *outs;
    if (!PyArg_ParseTuple(args, "OOO", &x, &w, &outs)) throw Error();
    const at::Tensor &xt = tensor(x), &wt = tensor(w);
    if (xt.dim() != 2) { PyErr_SetString(PyExc_ValueError, "x must be a matrix [rows, inner]"); throw Error(); }
    Ref list(PySequence_Fast(outs, "outs must be a sequence"));
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(list.p);
    std::vector<cr_proj_out> o(n);
    int col = 0;
    for (Py_ssize_t i = 0; i < n; ++i) {
      const at::Tensor& t = tensor(PySequence_Fast_GET_ITEM(list.p, i));
      if (t.dim() != 2 && t.size(0) == 0) { PyErr_SetString(PyExc_IndexError, "an output that is not a matrix needs a first row"); throw Error(); }
      const int cols = (int)(t.dim() == 2 ? t.size(1) : t.numel() / t.size(0));
      o[i] = cr_proj_out{t.data_ptr(), col, cols, cols, t.scalar_type() == at::kFloat ? 1 : 0};
      col += cols;
    }
    const void *const xp = xt.data_ptr(), *const wp = wt.data_ptr();
    const int R = (int)xt.size(0), K = (int)xt.size(1), N = (int)wt.size(0);
    void* const st = stream();
    check(unlocked([&] { return cr_proj_gemm(xp, wp, R, K, N, o.data(), (int)n, st); }));
    Py_INCREF(outs);
    return outs;
  });
}

PyObject* current_stream(PyObject*, PyObject*) {
  return guarded([] { return PyLong_FromVoidPtr(stream()); });
}

PyMethodDef methods[] = {{"current_stream", current_stream, METH_NOARGS, nullptr},
                         {"gdn_step", gdn_step, METH_VARARGS, nullptr},       {"qsa_step", qsa_step, METH_VARARGS, nullptr},
                         {"gdn_prefill", gdn_prefill, METH_VARARGS, nullptr}, {"qsa_prefill", qsa_prefill, METH_VARARGS, nullptr},
                         {"proj_gemm", proj_gemm, METH_VARARGS, nullptr},     {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding() {
#define INTERN(n) s_##n = PyUnicode_InternFromString(#n); if (!s_##n) return nullptr;
  NAMES(INTERN)
  return PyModule_Create(&module);
}
