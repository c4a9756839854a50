// The per-call work of the Python front end in native code: argument checks, the result tensor, the current stream
// and the C entry point, without a Python-level loop or a ctypes marshalling pass in between.
//
// Every function here either does the whole call or returns None, and then the Python code behind it runs: for
// anything out of the ordinary (an `out=` tensor of another kind, a tensor subclass or wrapper, a tensor that is not
// contiguous or not on a GPU, a shape or type that does not fit, an error code of the entry point) that code is the one
// that converts, accepts or raises.  So what is accepted and what is refused is decided in one place.
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/torch.h>

#include <cstring>
#include <string>
#include <vector>

namespace {

using at::Tensor;

// ---- entry points of libantares_b200.so, bound by address --------------------------------------------------------------
typedef int (*GemvFn)(const void *, const void *, const void *, void *, int, int, int, int, int, void *);
typedef int (*SigmoidFn)(const void *, void *, size_t, int, void *);
typedef int (*SoftmaxFn)(const void *, void *, int, int, int, void *);
typedef int (*RmsnormFn)(const void *, int, const void *, void *, int, int, float, void *);
typedef int (*RmsnormVsumFn)(const void *, const void *, const void *, void *, size_t, float, float, int, void *);
typedef int (*RopeFn)(const void *, const void *, const void *, void *, int, int, int, int, void *);
typedef int (*RopeAtFn)(const void *, const void *, int, void *, int, int, int, void *);
typedef int (*AttendAtFn)(const void *, const void *, const void *, void *, int, int, int, long, const void *, int, void *);
typedef int (*EltwiseFn)(const void *, const void *, int, const void *, int, const void *, const void *, int, void *, int, size_t, void *);
typedef int (*RowFn)(const void *, const void *, const void *, const void *, int, const void *, int, const void *, const void *, int, const void *, const void *,
                     int, void *, int, int, int, void *);
struct Entries {
  GemvFn gemv, gemm;
  SigmoidFn sigmoid;
  SoftmaxFn softmax;
  RmsnormFn rmsnorm;
  RmsnormVsumFn rmsnorm_vsum;
  RopeFn rope;
  RopeAtFn rope_at;
  AttendAtFn attend_at;
  EltwiseFn eltwise;
  RowFn row;
} E;

#define NOT_HERE Py_RETURN_NONE

// A plain tensor on a GPU, contiguous, that no wrapper or mode has a say in; else nullptr.
inline const Tensor *plain(PyObject *o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const Tensor &t = THPVariable_Unpack(o);
  if (!t.is_cuda() || !t.is_contiguous() || !t.has_storage()) return nullptr;
  constexpr c10::DispatchKeySet odd({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                     c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate, c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
  return t.key_set().has_any(odd) ? nullptr : &t;
}
inline int code_of(const Tensor &t) { return t.scalar_type() == at::kHalf ? 0 : t.scalar_type() == at::kFloat ? 1 : -1; }
inline void *stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
inline Tensor fresh(at::IntArrayRef shape, at::ScalarType type, const Tensor &like) { return at::empty(shape, at::TensorOptions().dtype(type).device(like.device())); }

template <class F>
inline int enter(F f) {  // like ctypes: other threads run during the call
  int rc;
  Py_BEGIN_ALLOW_THREADS rc = f();
  Py_END_ALLOW_THREADS return rc;
}
#define GUARDED(...)                \
  try {                             \
    __VA_ARGS__                     \
  } catch (const std::exception &) { \
    PyErr_Clear();                  \
    NOT_HERE;                       \
  }

// x . dequant(q, s); which 0 = by the number of rows, 1 = decode kernels, 2 = tensor-core GEMM; group 0 = what the scales' shape says
PyObject *project(long which, const Tensor &x, const Tensor &q, const Tensor &s, int64_t group) {
  const int code = code_of(x);
  if (code < 0 || s.scalar_type() != x.scalar_type() || q.scalar_type() != at::kInt || q.dim() != 2 || s.dim() != 2 || x.dim() < 1) NOT_HERE;
  const int64_t K = q.size(0) * 8, N = q.size(1), G = s.size(0);
  if (K <= 0 || N <= 0 || G <= 0 || K % G || (group && G * group != K) || s.size(1) != N || x.size(-1) != K || x.numel() <= 0) NOT_HERE;
  const int64_t M = x.numel() / K;
  if (M > INT32_MAX || K > INT32_MAX || N > INT32_MAX) NOT_HERE;
  if (which == 0) which = M <= 16 ? 1 : 2;
  c10::SmallVector<int64_t, 6> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = N;
  Tensor out = fresh(shape, x.scalar_type(), x);
  const GemvFn f = which == 1 ? E.gemv : E.gemm;
  const void *xp = x.data_ptr(), *qp = q.data_ptr(), *sp = s.data_ptr();
  void *op = out.data_ptr(), *st = stream();
  if (enter([&] { return f(xp, qp, sp, op, (int)M, (int)K, (int)N, (int)(K / G), code, st); })) NOT_HERE;
  return THPVariable_Wrap(std::move(out));
}
PyObject *sigmoid_of(const Tensor &x) {
  const int code = code_of(x);
  if (code < 0) NOT_HERE;
  Tensor out = fresh(x.sizes(), x.scalar_type(), x);
  const void *xp = x.data_ptr();
  void *op = out.data_ptr(), *st = stream();
  const size_t count = x.numel();
  if (enter([&] { return E.sigmoid(xp, op, count, code, st); })) NOT_HERE;
  return THPVariable_Wrap(std::move(out));
}
PyObject *softmax_of(const Tensor &x) {  // over the last axis
  const int code = code_of(x);
  if (code < 0 || x.dim() < 1 || x.numel() <= 0) NOT_HERE;
  const int64_t cols = x.size(-1), rows = x.numel() / cols;
  if (rows > INT32_MAX || cols > INT32_MAX) NOT_HERE;
  Tensor out = fresh(x.sizes(), x.scalar_type(), x);
  const void *xp = x.data_ptr();
  void *op = out.data_ptr(), *st = stream();
  if (enter([&] { return E.softmax(xp, op, (int)rows, (int)cols, code, st); })) NOT_HERE;
  return THPVariable_Wrap(std::move(out));
}

// w4a16(which, x, qweight, scales), sigmoid(x), softmax(x)
PyObject *py_w4a16(PyObject *, PyObject *const *a, Py_ssize_t n) {
  GUARDED({
    const Tensor *x, *q, *s;
    if (n != 4 || !(x = plain(a[1])) || !(q = plain(a[2])) || !(s = plain(a[3]))) NOT_HERE;
    return project(PyLong_AsLong(a[0]), *x, *q, *s, 0);
  })
}
PyObject *py_sigmoid(PyObject *, PyObject *o) {
  GUARDED({
    const Tensor *x = plain(o);
    if (!x) NOT_HERE;
    return sigmoid_of(*x);
  })
}
PyObject *py_softmax(PyObject *, PyObject *o) {
  GUARDED({
    const Tensor *x = plain(o);
    if (!x) NOT_HERE;
    return softmax_of(*x);
  })
}

// rmsnorm(x, weight, eps) -> fp16
PyObject *py_rmsnorm(PyObject *, PyObject *const *a, Py_ssize_t n) {
  GUARDED({
    const Tensor *x, *w;
    int code;
    if (n != 3 || !(x = plain(a[0])) || !(w = plain(a[1])) || (code = code_of(*x)) < 0 || w->scalar_type() != at::kHalf || x->dim() < 1 || x->numel() <= 0) NOT_HERE;
    const int64_t cols = x->size(-1), rows = x->numel() / cols;
    if (w->numel() < cols || rows > INT32_MAX || cols > INT32_MAX || !PyFloat_Check(a[2])) NOT_HERE;
    const float eps = (float)PyFloat_AS_DOUBLE(a[2]);
    Tensor out = fresh(x->sizes(), at::kHalf, *x);
    const void *xp = x->data_ptr(), *wp = w->data_ptr();
    void *op = out.data_ptr(), *st = stream();
    if (enter([&] { return E.rmsnorm(xp, code, wp, op, (int)rows, (int)cols, eps, st); })) NOT_HERE;
    return THPVariable_Wrap(std::move(out));
  })
}

// rmsnorm_vsum(x, vsum, weight, inv_n, eps)
PyObject *py_rmsnorm_vsum(PyObject *, PyObject *const *a, Py_ssize_t n) {
  GUARDED({
    const Tensor *x, *v, *w;
    int code;
    if (n != 5 || !(x = plain(a[0])) || !(v = plain(a[1])) || !(w = plain(a[2])) || (code = code_of(*x)) < 0) NOT_HERE;
    if (v->scalar_type() != at::kFloat || v->numel() != 1 || w->scalar_type() != x->scalar_type() || w->numel() < x->numel() || x->numel() <= 0) NOT_HERE;
    const float inv_n = (float)PyFloat_AsDouble(a[3]), eps = (float)PyFloat_AsDouble(a[4]);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      NOT_HERE;
    }
    Tensor out = fresh(x->sizes(), x->scalar_type(), *x);
    const void *xp = x->data_ptr(), *vp = v->data_ptr(), *wp = w->data_ptr();
    void *op = out.data_ptr(), *st = stream();
    const size_t count = x->numel();
    if (enter([&] { return E.rmsnorm_vsum(xp, vp, wp, op, count, inv_n, eps, code, st); })) NOT_HERE;
    return THPVariable_Wrap(std::move(out));
  })
}

// rope(x [rows, H, D], pos [rows], inv_freq)
PyObject *py_rope(PyObject *, PyObject *const *a, Py_ssize_t n) {
  GUARDED({
    const Tensor *x, *pos, *f;
    int code;
    if (n != 3 || !(x = plain(a[0])) || !(pos = plain(a[1])) || !(f = plain(a[2])) || (code = code_of(*x)) < 0 || x->dim() != 3 || x->numel() <= 0) NOT_HERE;
    if (pos->scalar_type() != at::kInt || f->scalar_type() != at::kFloat || pos->numel() < x->size(0)) NOT_HERE;
    const int64_t rows = x->size(0), H = x->size(1), D = x->size(2);
    if (rows > INT32_MAX || H > INT32_MAX || D > INT32_MAX) NOT_HERE;
    Tensor out = fresh(x->sizes(), x->scalar_type(), *x);
    const void *xp = x->data_ptr(), *fp = f->data_ptr(), *pp = pos->data_ptr();
    void *op = out.data_ptr(), *st = stream();
    if (enter([&] { return E.rope(xp, fp, pp, op, (int)rows, (int)H, (int)D, code, st); })) NOT_HERE;
    return THPVariable_Wrap(std::move(out));
  })
}

// rope_at(dtype code, x [H, ...], inv_freq, out or None, position): one row, its position from the host
PyObject *py_rope_at(PyObject *, PyObject *const *a, Py_ssize_t n) {
  GUARDED({
    const Tensor *x, *f, *given = nullptr;
    if (n != 5 || !(x = plain(a[1])) || !(f = plain(a[2])) || (a[3] != Py_None && !(given = plain(a[3])))) NOT_HERE;
    const int code = code_of(*x);
    if (code < 0 || code != PyLong_AsLong(a[0]) || f->scalar_type() != at::kFloat || x->dim() < 1 || x->numel() <= 0 || !PyLong_Check(a[4])) NOT_HERE;
    if (given && (given->scalar_type() != x->scalar_type() || given->numel() != x->numel())) NOT_HERE;
    const long pos = PyLong_AsLong(a[4]);
    const int64_t H = x->size(0), D = x->numel() / H;
    if (PyErr_Occurred() || pos < INT32_MIN || pos > INT32_MAX || H > INT32_MAX || D > INT32_MAX) {
      PyErr_Clear();
      NOT_HERE;
    }
    Tensor out = given ? *given : fresh({H, D}, x->scalar_type(), *x);
    const void *xp = x->data_ptr(), *fp = f->data_ptr();
    void *op = out.data_ptr(), *st = stream();
    if (enter([&] { return E.rope_at(xp, fp, (int)pos, op, (int)H, (int)D, code, st); })) NOT_HERE;
    if (given) {
      Py_INCREF(a[3]);
      return a[3];
    }
    return THPVariable_Wrap(std::move(out));
  })
}

// attend_at(dtype code, q [H, D], k, v [S, H, D] with one row stride, scale: fp32 on the GPU)
PyObject *py_attend_at(PyObject *, PyObject *const *a, Py_ssize_t n) {
  GUARDED({
    const Tensor *q, *k, *v, *f;
    if (n != 5 || !(q = plain(a[1])) || !(k = plain(a[2])) || !(v = plain(a[3])) || !(f = plain(a[4]))) NOT_HERE;
    const int code = code_of(*q);
    if (code < 0 || code != PyLong_AsLong(a[0]) || q->dim() != 2 || k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type()) NOT_HERE;
    const int64_t H = q->size(0), D = q->size(1), S = k->dim() > 0 ? k->size(0) : 0;
    if (S <= 0 || f->scalar_type() != at::kFloat || f->numel() < 1 || k->numel() != S * H * D || v->numel() != S * H * D || S > INT32_MAX || H > INT32_MAX) NOT_HERE;
    const long stride = k->stride(0);
    Tensor out = fresh(q->sizes(), q->scalar_type(), *q);
    const void *qp = q->data_ptr(), *kp = k->data_ptr(), *vp = v->data_ptr(), *fp = f->data_ptr();
    void *op = out.data_ptr(), *st = stream();
    if (enter([&] { return E.attend_at(qp, kp, vp, op, (int)S, (int)H, (int)D, stride, fp, code, st); })) NOT_HERE;
    return THPVariable_Wrap(std::move(out));
  })
}

// ---- exported programs ----------------------------------------------------------------------------------------------
enum { KIND_W4A16 = 0, KIND_SIGMOID, KIND_SOFTMAX, KIND_ELTWISE, KIND_ROWS };
struct Input {
  at::ScalarType type;
  std::vector<int64_t> bound;
  std::vector<char> dyn;  // the declared extent is an upper bound
};
struct Program {
  int kind;
  std::vector<Input> inputs;
  // element-wise / row programs: postfix code, operands as indices into the inputs.  The others: mats holds the operands in
  // the entry point's order, group the group size that the statements name.
  int group = 0;
  std::vector<unsigned char> ops, args;
  std::vector<int> lens, kinds, mats, cols;
  std::vector<float> consts;
};

void drop(PyObject *capsule) { delete static_cast<Program *>(PyCapsule_GetPointer(capsule, "antares_b200.program")); }

template <class T>
bool ints(PyObject *seq, std::vector<T> &v) {
  PyObject *f = PySequence_Fast(seq, "a sequence of numbers");
  if (!f) return false;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(f); ++i) v.push_back((T)PyLong_AsLongLong(PySequence_Fast_GET_ITEM(f, i)));
  Py_DECREF(f);
  return !PyErr_Occurred();
}

// program(kind, [(type, bounds, dyn)], group, ops, args, lens, kinds, consts, mats, cols)
PyObject *py_program(PyObject *, PyObject *args) {
  int kind, group;
  PyObject *ins, *ops, *opargs, *lens, *kinds, *consts, *mats, *cols;
  if (!PyArg_ParseTuple(args, "iOiOOOOOOO", &kind, &ins, &group, &ops, &opargs, &lens, &kinds, &consts, &mats, &cols)) return nullptr;
  auto p = std::make_unique<Program>();
  p->kind = kind, p->group = group;
  PyObject *f = PySequence_Fast(ins, "a sequence of inputs");
  if (!f) return nullptr;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(f); ++i) {
    int type;
    PyObject *bound, *dyn;
    std::vector<int64_t> b;
    std::vector<char> d;
    if (!PyArg_ParseTuple(PySequence_Fast_GET_ITEM(f, i), "iOO", &type, &bound, &dyn) || !ints(bound, b) || !ints(dyn, d) || b.size() != d.size()) {
      Py_DECREF(f);
      return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "an input needs as many flags as bounds");
    }
    p->inputs.push_back(Input{type == 0 ? at::kHalf : type == 1 ? at::kFloat : at::kInt, b, d});
  }
  Py_DECREF(f);
  std::vector<int> o, oa;
  if (!ints(ops, o) || !ints(opargs, oa) || !ints(lens, p->lens) || !ints(kinds, p->kinds) || !ints(mats, p->mats) || !ints(cols, p->cols)) return nullptr;
  p->ops.assign(o.begin(), o.end());
  p->args.assign(oa.begin(), oa.end());
  f = PySequence_Fast(consts, "a sequence of constants");
  if (!f) return nullptr;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(f); ++i) p->consts.push_back((float)PyFloat_AsDouble(PySequence_Fast_GET_ITEM(f, i)));
  Py_DECREF(f);
  if (PyErr_Occurred()) return nullptr;
  return PyCapsule_New(p.release(), "antares_b200.program", drop);
}

constexpr size_t MAX_INPUTS = 8;

// run(program, tensor, ...)
PyObject *py_run(PyObject *, PyObject *const *a, Py_ssize_t n) {
  GUARDED({
    Program *p = n >= 2 ? static_cast<Program *>(PyCapsule_GetPointer(a[0], "antares_b200.program")) : nullptr;
    if (!p) {
      PyErr_Clear();
      NOT_HERE;
    }
    const size_t count = p->inputs.size();
    if ((size_t)n - 1 != count || count > MAX_INPUTS) NOT_HERE;
    const Tensor *t[MAX_INPUTS];
    for (size_t i = 0; i < count; ++i) {
      const Input &in = p->inputs[i];
      if (!(t[i] = plain(a[i + 1])) || t[i]->scalar_type() != in.type || (size_t)t[i]->dim() != in.bound.size() || t[i]->numel() <= 0) NOT_HERE;
      for (size_t d = 0; d < in.bound.size(); ++d)
        if (t[i]->size(d) > in.bound[d] || (!in.dyn[d] && t[i]->size(d) != in.bound[d])) NOT_HERE;
    }
    if (p->kind == KIND_W4A16) return project(0, *t[p->mats[0]], *t[p->mats[1]], *t[p->mats[2]], p->group);
    if (p->kind == KIND_SIGMOID) return sigmoid_of(*t[p->mats[0]]);
    if (p->kind == KIND_SOFTMAX) return softmax_of(*t[p->mats[0]]);
    void *st = stream();
    bool wide = false;
    const void *mp[MAX_INPUTS], *cp[MAX_INPUTS];
    int md[MAX_INPUTS], cd[MAX_INPUTS];
    const Tensor &x = *t[p->mats[0]];
    const int64_t ncols = x.dim() > 0 ? x.size(-1) : 1;
    for (size_t i = 0; i < p->mats.size(); ++i) {
      const Tensor &m = *t[p->mats[i]];
      if (m.sizes() != x.sizes() || (md[i] = code_of(m)) < 0) NOT_HERE;
      mp[i] = m.data_ptr();
      wide = wide || md[i] == 1;
    }
    for (size_t i = 0; i < p->cols.size(); ++i) {
      const Tensor &c = *t[p->cols[i]];
      if (c.numel() != ncols || (cd[i] = code_of(c)) < 0) NOT_HERE;
      cp[i] = c.data_ptr();
      wide = wide || cd[i] == 1;
    }
    Tensor out = fresh(x.sizes(), wide ? at::kFloat : at::kHalf, x);
    void *op = out.data_ptr();
    const size_t total = x.numel();
    const int n_consts = (int)p->consts.size();
    int rc;
    if (p->kind == KIND_ELTWISE) {
      rc = enter([&] { return E.eltwise(p->ops.data(), p->args.data(), (int)p->ops.size(), p->consts.data(), n_consts, mp, md, (int)p->mats.size(), op, wide, total, st); });
    } else {
      if (total / ncols > INT32_MAX || ncols > INT32_MAX) NOT_HERE;
      rc = enter([&] {
        return E.row(p->ops.data(), p->args.data(), p->lens.data(), p->kinds.data(), (int)p->lens.size(), p->consts.data(), n_consts, mp, md, (int)p->mats.size(), cp, cd,
                     (int)p->cols.size(), op, wide, (int)(total / ncols), (int)ncols, st);
      });
    }
    if (rc) NOT_HERE;
    return THPVariable_Wrap(std::move(out));
  })
}

// bind({name: address})
PyObject *py_bind(PyObject *, PyObject *d) {
  auto get = [&](const char *name, auto &slot) {
    PyObject *v = PyDict_GetItemString(d, name);
    void *addr = v ? PyLong_AsVoidPtr(v) : nullptr;
    std::memcpy(&slot, &addr, sizeof addr);
    return addr != nullptr;
  };
  if (!PyDict_Check(d) || !get("ab200_w4a16_gemv", E.gemv) || !get("ab200_w4a16_gemm", E.gemm) || !get("ab200_sigmoid", E.sigmoid) || !get("ab200_softmax", E.softmax) ||
      !get("ab200_rmsnorm", E.rmsnorm) || !get("ab200_rmsnorm_vsum", E.rmsnorm_vsum) || !get("ab200_rope", E.rope) || !get("ab200_rope_at", E.rope_at) ||
      !get("ab200_attention_decode_at", E.attend_at) || !get("ab200_eltwise_vm", E.eltwise) || !get("ab200_rowreduce_vm", E.row))
    return PyErr_Format(PyExc_KeyError, "bind: an entry point is missing");
  Py_RETURN_NONE;
}

// what this file was compiled against; another torch or Python must not use it
PyObject *py_built_for(PyObject *, PyObject *) { return PyUnicode_FromString(AB200_BUILT_FOR); }

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"bind", py_bind, METH_O, nullptr},
                         {"built_for", py_built_for, METH_NOARGS, nullptr},
                         {"program", py_program, METH_VARARGS, nullptr},
                         {"sigmoid", py_sigmoid, METH_O, nullptr},
                         {"softmax", py_softmax, METH_O, nullptr},
                         FAST(w4a16),
                         FAST(rmsnorm),
                         FAST(rmsnorm_vsum),
                         FAST(rope),
                         FAST(rope_at),
                         FAST(attend_at),
                         FAST(run),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall() { return PyModule_Create(&module); }
