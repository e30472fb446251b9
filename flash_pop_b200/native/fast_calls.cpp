// The host side of the operator calls, natively: argument checks, allocation of the results and of scratch memory, and the
// call into the C ABI.  In Python the same steps cost 50 to 65 us a call (measured), several times what most kernels of
// small and medium calls take.
//
// Every function here takes the ordinary call only - strided CUDA tensors of exactly torch.Tensor or Parameter type with the
// dtypes, shapes and strides the kernels read in place, no dispatch mode - and returns None for anything else, errors
// included; the caller then goes through the Python path, which copies, converts or raises.  A nonzero status of the C ABI
// comes back as an int.  Nothing is kept between calls but the addresses of the C ABI's entry points.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/TensorBody.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/autograd/python_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/flash_pop_b200.h"

namespace {

struct Entry {
  decltype(&fpb_retention_fwd) retention_fwd;
  decltype(&fpb_retention_bwd) retention_bwd;
  decltype(&fpb_pop_retention_fwd) pop_fwd;
  decltype(&fpb_pop_retention_bwd) pop_bwd;
  decltype(&fpb_pop_suffix_fwd) suffix_fwd;
  decltype(&fpb_pop_suffix_bwd) suffix_bwd;
  decltype(&fpb_retention_step) step;
  decltype(&fpb_workspace_bytes) workspace_bytes;
  decltype(&fpb_rotary) rotary;
  decltype(&fpb_groupnorm_gate_fwd) gate_fwd;
  decltype(&fpb_groupnorm_gate_bwd) gate_bwd;
  decltype(&fpb_layernorm_fwd) norm_fwd;
  decltype(&fpb_layernorm_bwd) norm_bwd;
  decltype(&fpb_column_sums) column_sums;
} entry;
constexpr int ENTRIES = sizeof(Entry) / sizeof(void*), MAX_HEADS = 256;

struct NotOurs {};                               // thrown where a call is left to the Python path
#define NEED(cond) do { if (!(cond)) throw NotOurs{}; } while (0)

// A tensor the kernels may read through its address: exact type, strided CUDA memory, no lazy negation or conjugation.
at::Tensor tensor(PyObject* o) {
  NEED(THPVariable_CheckExact(o));
  const at::Tensor& t = THPVariable_Unpack(o);
  NEED(t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.has_storage() && !t.is_neg() && !t.is_conj() && t.numel() > 0);
  return t;
}
at::Tensor maybe(PyObject* o) { return o == Py_None ? at::Tensor() : tensor(o); }
bool real(at::ScalarType t) { return t == at::kBFloat16 || t == at::kFloat; }
int32_t code(at::ScalarType t) { return t == at::kFloat ? FPB_F32 : FPB_BF16; }

// unit inner stride, and no row folded onto another (as _lib.unit_inner)
bool in_place(const at::Tensor& t) {
  const int n = (int)t.dim();
  if (t.is_contiguous()) return true;
  if (n == 0 || n > 6 || (t.stride(n - 1) != 1 && t.size(n - 1) != 1)) return false;
  int64_t st[6], sz[6];
  int m = 0;
  for (int i = 0; i < n - 1; ++i) {
    if (t.size(i) <= 1) continue;
    int j = m++;
    for (; j > 0 && st[j - 1] > t.stride(i); --j) { st[j] = st[j - 1]; sz[j] = sz[j - 1]; }
    st[j] = t.stride(i); sz[j] = t.size(i);
  }
  int64_t span = t.size(n - 1);
  for (int i = 0; i < m; ++i) {
    if (st[i] < span) return false;
    span = st[i] * sz[i];
  }
  return true;
}
bool aligned(const at::Tensor& t, int64_t bytes) {
  const int64_t vec = bytes / t.element_size();
  if ((uintptr_t)t.data_ptr() % bytes) return false;
  for (int64_t i = 0; i + 1 < t.dim(); ++i)
    if (t.stride(i) % vec) return false;
  return t.stride(t.dim() - 1) == 1;
}
bool state_ok(const at::Tensor& s) { return (s.stride(3) == 1 || s.size(3) == 1) && (s.stride(2) == s.size(3) || s.size(2) == 1); }

fpb_seq seq(const at::Tensor& t) {
  if (!t.defined()) return {nullptr, 0, 0, 0};
  return {t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)};
}
fpb_seq seq3(const at::Tensor& t) { return {t.data_ptr(), t.stride(0), 0, t.stride(1)}; }      // (B, H, d): one token
fpb_state state(const at::Tensor& t) {
  if (!t.defined()) return {nullptr, 0, 0};
  return {t.data_ptr(), t.stride(0), t.stride(1)};
}

struct Decays {
  double g[MAX_HEADS];
  Decays(PyObject* o, int64_t heads) {
    NEED(PyTuple_Check(o) && PyTuple_GET_SIZE(o) == heads && heads <= MAX_HEADS);
    for (int64_t h = 0; h < heads; ++h) {
      PyObject* f = PyTuple_GET_ITEM(o, h);
      NEED(PyFloat_Check(f));
      g[h] = PyFloat_AS_DOUBLE(f);
    }
  }
};

at::Tensor make(at::IntArrayRef shape, const at::Tensor& like, at::ScalarType t) { return at::empty(shape, like.options().dtype(t).requires_grad(false)); }
at::Tensor make_like(const at::Tensor& t) { return at::empty_like(t, t.options().requires_grad(false)); }

// a call on t's device and its current stream
struct Place {
  c10::cuda::CUDAGuard guard;
  fpb_stream_t stream;
  explicit Place(const at::Tensor& t) : guard(t.device()), stream((fpb_stream_t)c10::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
};

struct Dims {
  fpb_dims d{};
  at::Tensor scratch;
  Dims(const at::Tensor& q, int64_t T, int64_t H, int64_t dk, int64_t dv, const Decays& g, int64_t block, int64_t flags, int64_t batch) {
    d.dtype = code(q.scalar_type()); d.B = (int32_t)batch; d.T = (int32_t)T; d.H = (int32_t)H; d.dk = (int32_t)dk; d.dv = (int32_t)dv;
    d.block_size = (int32_t)block; d.flags = (int32_t)flags; d.head_decays = g.g;
  }
  void with_scratch(const at::Tensor& q) {
    const int64_t need = entry.workspace_bytes(&d);
    if (need > 0) {
      scratch = at::empty({need}, q.options().dtype(at::kByte).requires_grad(false));
      d.workspace = scratch.data_ptr(); d.workspace_bytes = need;
    }
  }
};

at::ScalarType state_dtype(PyObject* asked, const at::Tensor& q, const at::Tensor& s) {
  at::ScalarType t = s.defined() ? s.scalar_type() : q.scalar_type();
  if (asked != Py_None) {
    NEED(THPDtype_Check(asked));
    t = reinterpret_cast<THPDtype*>(asked)->scalar_type;
  }
  NEED(t == q.scalar_type() || (t == at::kFloat && q.scalar_type() == at::kBFloat16));
  return t;
}

int64_t integer(PyObject* o) {
  NEED(PyLong_Check(o));
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); throw NotOurs{}; }
  return v;
}
PyObject* wrap(const at::Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
PyObject* tuple_of(std::initializer_list<at::Tensor> ts) {
  PyObject* r = PyTuple_New((Py_ssize_t)ts.size());
  if (!r) return nullptr;
  Py_ssize_t i = 0;
  for (const at::Tensor& t : ts) {
    PyObject* o = wrap(t);
    if (!o) { Py_DECREF(r); return nullptr; }
    PyTuple_SET_ITEM(r, i++, o);
  }
  return r;
}

template <typename F> int unlocked(F f) {
  int r;
  Py_BEGIN_ALLOW_THREADS
  r = f();
  Py_END_ALLOW_THREADS
  return r;
}
// body with the exceptions of this file and of ATen turned into Python's
template <typename F> PyObject* guarded(Py_ssize_t got, Py_ssize_t want, F body) {
  if (got != want) { PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got); return nullptr; }
  try {
    if (!entry.step || c10::impl::TorchDispatchModeTLS::any_modes_set()) Py_RETURN_NONE;
    return body();
  } catch (const NotOurs&) {
    Py_RETURN_NONE;
  } catch (const c10::OutOfMemoryError& e) {
    // (the Python path raises the allocator's own exception type with its message)
    Py_RETURN_NONE;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

void check_qkv(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& s) {
  NEED(q.dim() == 4 && v.dim() == 4 && k.sizes() == q.sizes() && v.size(0) == q.size(0) && v.size(1) == q.size(1) && v.size(2) == q.size(2));
  NEED(real(q.scalar_type()) && k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type());
  NEED(k.device() == q.device() && v.device() == q.device() && in_place(q) && in_place(k) && in_place(v));
  if (s.defined())
    NEED(s.dim() == 4 && s.size(0) == q.size(0) && s.size(1) == q.size(2) && s.size(2) == q.size(3) && s.size(3) == v.size(3) &&
         s.device() == q.device() && state_ok(s));
}

// step(q, k, v, decays, prev_state, state_dtype, in_place) -> (o, state)
PyObject* step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 7, [&]() -> PyObject* {
    const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), prev = maybe(a[4]);
    NEED(q.dim() == 3 && v.dim() == 3 && k.sizes() == q.sizes() && v.size(0) == q.size(0) && v.size(1) == q.size(1));
    NEED(real(q.scalar_type()) && k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type());
    NEED(k.device() == q.device() && v.device() == q.device() && in_place(q) && in_place(k) && in_place(v));
    const int64_t B = q.size(0), H = q.size(1), dk = q.size(2), dv = v.size(2);
    const Decays g(a[3], H);
    at::ScalarType sdt = prev.defined() ? prev.scalar_type() : q.scalar_type();
    if (a[5] != Py_None) { NEED(THPDtype_Check(a[5])); sdt = reinterpret_cast<THPDtype*>(a[5])->scalar_type; }
    NEED(real(sdt));
    if (prev.defined())
      NEED(prev.dim() == 4 && prev.size(0) == B && prev.size(1) == H && prev.size(2) == dk && prev.size(3) == dv && prev.scalar_type() == sdt &&
           prev.device() == q.device() && state_ok(prev));
    const bool reuse = prev.defined() && a[6] == Py_True;
    Place here(q);
    const at::Tensor o = make({B, H, dv}, q, q.scalar_type()), out = reuse ? prev : make({B, H, dk, dv}, q, sdt);
    const Dims d(q, 1, H, dk, dv, g, 0, 0, B);
    const fpb_seq sq = seq3(q), sk = seq3(k), sv = seq3(v), so = seq3(o);
    const fpb_state s0 = state(prev), s1 = state(out);
    const int r = unlocked([&] { return entry.step(&d.d, code(sdt), &sq, &sk, &sv, &s0, &so, &s1, here.stream); });
    if (r) return PyLong_FromLong(r);
    PyObject* po = wrap(o);
    PyObject* ps = reuse ? Py_NewRef(a[4]) : wrap(out);
    return po && ps ? Py_BuildValue("(NN)", po, ps) : nullptr;
  });
}

// forward(q, k, v, s, decays, state_dtype, flags, block_size) -> (o, s_out) or, with block_size > 0, (o, block_states)
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 8, [&]() -> PyObject* {
    const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), s = maybe(a[3]);
    check_qkv(q, k, v, s);
    const int64_t B = q.size(0), T = q.size(1), H = q.size(2), dk = q.size(3), dv = v.size(3);
    const Decays g(a[4], H);
    const at::ScalarType sdt = state_dtype(a[5], q, s);
    NEED(!s.defined() || s.scalar_type() == sdt);
    const int64_t block = integer(a[7]), flags = integer(a[6]) | (sdt != q.scalar_type() ? FPB_FLAG_STATE_F32 : 0);
    NEED(block >= 0 && block <= INT32_MAX);
    Place here(q);
    const at::Tensor o = make({B, T, H, dv}, q, q.scalar_type());
    const at::Tensor end = block ? make({B, T / block, H, dk, dv}, q, sdt) : make({B, H, dk, dv}, q, sdt);
    Dims d(q, T, H, dk, dv, g, block, flags, B);
    d.with_scratch(q);
    const fpb_seq sq = seq(q), sk = seq(k), sv = seq(v), so = seq(o);
    const fpb_state s0 = state(s), s1 = block ? fpb_state{nullptr, 0, 0} : state(end);
    void* blocks = block && end.numel() > 0 ? end.data_ptr() : nullptr;
    const int r = unlocked([&] {
      return block ? entry.pop_fwd(&d.d, &sq, &sk, &sv, &s0, &so, blocks, here.stream)
                   : entry.retention_fwd(&d.d, &sq, &sk, &sv, &s0, &so, &s1, here.stream);
    });
    return r ? PyLong_FromLong(r) : tuple_of({o, end});
  });
}

// backward(q, k, v, s, dO, d_end, decays, state_dtype, flags, block_size, need_q, need_kv, need_s) -> (dQ, dK, dV, dS)
PyObject* backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 13, [&]() -> PyObject* {
    const at::Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), s = maybe(a[3]), dO = tensor(a[4]), dE = maybe(a[5]);
    check_qkv(q, k, v, s);
    const int64_t B = q.size(0), T = q.size(1), H = q.size(2), dk = q.size(3), dv = v.size(3);
    const Decays g(a[6], H);
    NEED(THPDtype_Check(a[7]));
    const at::ScalarType sdt = reinterpret_cast<THPDtype*>(a[7])->scalar_type;
    const int64_t block = integer(a[9]);
    const bool need_q = a[10] == Py_True, need_kv = a[11] == Py_True, need_s = a[12] == Py_True;
    NEED((need_q || need_kv) && block >= 0 && block <= INT32_MAX);
    NEED(dO.sizes() == v.sizes() && dO.scalar_type() == q.scalar_type() && dO.device() == q.device() && in_place(dO));
    if (dE.defined()) {
      NEED(dE.scalar_type() == sdt && dE.device() == q.device());
      if (block) NEED(dE.is_contiguous() && dE.dim() == 5 && dE.size(0) == B && dE.size(1) == T / block && dE.size(2) == H && dE.size(3) == dk && dE.size(4) == dv);
      else NEED(dE.dim() == 4 && dE.size(0) == B && dE.size(1) == H && dE.size(2) == dk && dE.size(3) == dv && state_ok(dE) &&
                (B == 1 || dE.stride(0) >= dk * dv) && (H == 1 || dE.stride(1) >= dk * dv));
    }
    const int64_t flags = integer(a[8]) | (need_q ? 0 : FPB_FLAG_SKIP_DQ) | (need_kv ? 0 : FPB_FLAG_SKIP_DKDV);
    Place here(q);
    const at::Tensor dQ = need_q ? make_like(q) : at::Tensor(), dK = need_kv ? make_like(k) : at::Tensor(),
                     dV = need_kv ? make_like(v) : at::Tensor(), dS = need_s ? make({B, H, dk, dv}, q, sdt) : at::Tensor();
    Dims d(q, T, H, dk, dv, g, block, flags, B);
    d.with_scratch(q);
    const fpb_seq sq = seq(q), sk = seq(k), sv = seq(v), so = seq(dO), gq = seq(dQ), gk = seq(dK), gv = seq(dV);
    const fpb_state s0 = state(s), s1 = block ? fpb_state{nullptr, 0, 0} : state(dE), gs = state(dS);
    const int r = unlocked([&] {
      return block ? entry.pop_bwd(&d.d, &sq, &sk, &sv, &s0, &so, dE.defined() ? dE.data_ptr() : nullptr, &gq, &gk, &gv, &gs, here.stream)
                   : entry.retention_bwd(&d.d, &sq, &sk, &sv, &s0, &so, &s1, &gq, &gk, &gv, &gs, here.stream);
    });
    return r ? PyLong_FromLong(r) : tuple_of({dQ, dK, dV, dS});
  });
}

// (B, M, P, H, d) as (B M, P, H, d) in place
at::Tensor rows_of(const at::Tensor& t) {
  NEED(t.dim() == 5 && (t.size(0) == 1 || t.size(1) == 1 || t.stride(0) == t.size(1) * t.stride(1)));
  const at::Tensor f = t.flatten(0, 1);
  NEED(f.data_ptr() == t.data_ptr() && in_place(f));
  return f;
}

// suffix_forward(sq, sk, sv, s, block_states, decays, flags) -> (o, fq, fk, fv)
PyObject* suffix_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 7, [&]() -> PyObject* {
    const at::Tensor sq = tensor(a[0]), sk = tensor(a[1]), sv = tensor(a[2]), s = maybe(a[3]), bs = tensor(a[4]);
    NEED(sq.dim() == 5 && sv.dim() == 5 && sk.sizes() == sq.sizes() && sv.sizes().slice(0, 4) == sq.sizes().slice(0, 4));
    const int64_t B = sq.size(0), M = sq.size(1), P = sq.size(2), H = sq.size(3), dk = sq.size(4), dv = sv.size(4);
    const at::ScalarType sdt = bs.scalar_type();
    NEED(real(sq.scalar_type()) && sk.scalar_type() == sq.scalar_type() && sv.scalar_type() == sq.scalar_type() &&
         (sdt == sq.scalar_type() || (sdt == at::kFloat && sq.scalar_type() == at::kBFloat16)));
    NEED(sk.device() == sq.device() && sv.device() == sq.device() && bs.device() == sq.device() && bs.dim() == 5 && bs.is_contiguous());
    NEED(bs.size(0) == B && M <= bs.size(1) + 1 && bs.size(2) == H && bs.size(3) == dk && bs.size(4) == dv && B * M <= INT32_MAX);
    if (s.defined())
      NEED(s.dim() == 4 && s.size(0) == B && s.size(1) == H && s.size(2) == dk && s.size(3) == dv && s.scalar_type() == sdt &&
           s.device() == sq.device() && state_ok(s));
    const Decays g(a[5], H);
    const at::Tensor fq = rows_of(sq), fk = rows_of(sk), fv = rows_of(sv);
    const int64_t flags = integer(a[6]) | (sdt != sq.scalar_type() ? FPB_FLAG_STATE_F32 : 0);
    Place here(fq);
    const at::Tensor o = make({B, M, P, H, dv}, sq, sq.scalar_type());
    const Dims d(fq, P, H, dk, dv, g, 0, flags, B);
    const fpb_seq q4 = seq(fq), k4 = seq(fk), v4 = seq(fv), o4{o.data_ptr(), P * H * dv, H * dv, dv};
    const fpb_state s0 = state(s);
    const int r = unlocked([&] {
      return entry.suffix_fwd(&d.d, (int32_t)M, (int32_t)bs.size(1), &q4, &k4, &v4, &s0, bs.data_ptr(), &o4, here.stream);
    });
    return r ? PyLong_FromLong(r) : tuple_of({o, fq, fk, fv});
  });
}

// suffix_backward(fq, fk, fv, s, block_states, dO (B, M, P, H, dv), decays, flags) -> (dQ, dK, dV (B, M, P, H, d), dS, d_block_states)
PyObject* suffix_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 8, [&]() -> PyObject* {
    const at::Tensor fq = tensor(a[0]), fk = tensor(a[1]), fv = tensor(a[2]), s = maybe(a[3]), bs = tensor(a[4]), dO5 = tensor(a[5]);
    NEED(dO5.dim() == 5 && dO5.scalar_type() == fq.scalar_type() && dO5.device() == fq.device());
    const int64_t B = dO5.size(0), M = dO5.size(1), P = fq.size(1), H = fq.size(2), dk = fq.size(3), dv = fv.size(3);
    NEED(B * M == fq.size(0) && dO5.size(2) == P && dO5.size(3) == H && dO5.size(4) == dv);
    const at::Tensor dO = rows_of(dO5);
    NEED(fk.sizes() == fq.sizes() && fv.dim() == 4 && fk.scalar_type() == fq.scalar_type() && fv.scalar_type() == fq.scalar_type() && bs.dim() == 5 &&
         bs.is_contiguous() && bs.device() == fq.device() && in_place(fq) && in_place(fk) && in_place(fv) && (!s.defined() || state_ok(s)));
    const Decays g(a[6], H);
    Place here(fq);
    const at::Tensor dQ = make_like(fq), dK = make_like(fk), dV = make_like(fv), dB = make_like(bs),
                     dS = s.defined() ? make({B, H, dk, dv}, fq, bs.scalar_type()) : at::Tensor();
    const Dims d(fq, P, H, dk, dv, g, 0, integer(a[7]), B);
    const fpb_seq q4 = seq(fq), k4 = seq(fk), v4 = seq(fv), o4 = seq(dO), gq = seq(dQ), gk = seq(dK), gv = seq(dV);
    const fpb_state s0 = state(s), gs = state(dS);
    const int r = unlocked([&] {
      return entry.suffix_bwd(&d.d, (int32_t)M, (int32_t)bs.size(1), &q4, &k4, &v4, &s0, bs.data_ptr(), &o4, &gq, &gk, &gv, &gs,
                              dB.data_ptr(), here.stream);
    });
    if (r) return PyLong_FromLong(r);
    auto rows = [&](const at::Tensor& t) { return t.unflatten(0, {B, M}); };
    return tuple_of({rows(dQ), rows(dK), rows(dV), dS, dB});
  });
}

// rotary(q, k, phasors, conjugate, out_dtype) -> (q', k')
PyObject* rotary(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 5, [&]() -> PyObject* {
    const at::Tensor q = tensor(a[0]), k = tensor(a[1]), ph = tensor(a[2]);
    NEED(q.dim() == 4 && k.sizes() == q.sizes() && real(q.scalar_type()) && k.scalar_type() == q.scalar_type() && k.device() == q.device());
    const int64_t B = q.size(0), T = q.size(1), H = q.size(2), d = q.size(3);
    NEED(d % 8 == 0 && ph.scalar_type() == at::kFloat && ph.is_contiguous() && ph.dim() == 4 && (ph.size(0) == 1 || ph.size(0) == B) &&
         ph.size(1) == T && ph.size(2) == d / 2 && ph.size(3) == 2 && ph.device() == q.device() && (uintptr_t)ph.data_ptr() % 16 == 0);
    NEED(THPDtype_Check(a[4]));
    const at::ScalarType odt = reinterpret_cast<THPDtype*>(a[4])->scalar_type;
    NEED(real(odt) && in_place(q) && in_place(k) && aligned(q, 16) && aligned(k, 16));
    Place here(q);
    const at::Tensor q2 = make({B, T, H, d}, q, odt), k2 = make({B, T, H, d}, q, odt);
    const fpb_seq qi = seq(q), ki = seq(k), qo = seq(q2), ko = seq(k2);
    const int r = unlocked([&] {
      return entry.rotary((int32_t)B, (int32_t)T, (int32_t)H, (int32_t)d, code(q.scalar_type()), code(odt), a[3] == Py_True ? 1 : 0,
                          (const float*)ph.data_ptr(), ph.size(0) == 1 ? 0 : T * (d / 2), &qi, &ki, &qo, &ko, here.stream);
    });
    return r ? PyLong_FromLong(r) : tuple_of({q2, k2});
  });
}

void check_gate(const at::Tensor& o, const at::Tensor& z) {
  NEED(o.dim() == 4 && z.sizes() == o.sizes() && real(o.scalar_type()) && z.scalar_type() == o.scalar_type() && z.device() == o.device());
  const int64_t nb = o.scalar_type() == at::kFloat ? 8 : 4;
  NEED(in_place(o) && in_place(z) && aligned(o, nb) && aligned(z, nb));
}
// gate_forward(o, z, eps, swish) -> (y,)
PyObject* gate_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 4, [&]() -> PyObject* {
    const at::Tensor o = tensor(a[0]), z = tensor(a[1]);
    check_gate(o, z);
    NEED(PyFloat_Check(a[2]));
    Place here(o);
    const at::Tensor y = make(o.sizes(), o, o.scalar_type());
    const fpb_seq so = seq(o), sz = seq(z), sy = seq(y);
    const int r = unlocked([&] {
      return entry.gate_fwd((int32_t)o.size(0), (int32_t)o.size(1), (int32_t)o.size(2), (int32_t)o.size(3), code(o.scalar_type()),
                            (float)PyFloat_AS_DOUBLE(a[2]), a[3] == Py_True ? 1 : 0, &so, &sz, &sy, here.stream);
    });
    return r ? PyLong_FromLong(r) : tuple_of({y});
  });
}
// gate_backward(o, z, dy, eps, swish) -> (d_o, d_z)
PyObject* gate_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 5, [&]() -> PyObject* {
    const at::Tensor o = tensor(a[0]), z = tensor(a[1]), dy = tensor(a[2]);
    check_gate(o, z);
    check_gate(o, dy);
    NEED(PyFloat_Check(a[3]));
    Place here(o);
    const at::Tensor d_o = make(o.sizes(), o, o.scalar_type()), d_z = make(o.sizes(), o, o.scalar_type());
    const fpb_seq so = seq(o), sz = seq(z), sy = seq(dy), go = seq(d_o), gz = seq(d_z);
    const int r = unlocked([&] {
      return entry.gate_bwd((int32_t)o.size(0), (int32_t)o.size(1), (int32_t)o.size(2), (int32_t)o.size(3), code(o.scalar_type()),
                            (float)PyFloat_AS_DOUBLE(a[3]), a[4] == Py_True ? 1 : 0, &so, &sz, &sy, &go, &gz, here.stream);
    });
    return r ? PyLong_FromLong(r) : tuple_of({d_o, d_z});
  });
}

const float* param(const at::Tensor& t, int64_t d, const at::Tensor& like) {
  if (!t.defined()) return nullptr;
  NEED(t.scalar_type() == at::kFloat && t.is_contiguous() && t.dim() == 1 && t.size(0) == d && t.device() == like.device() &&
       (uintptr_t)t.data_ptr() % 16 == 0);
  return (const float*)t.data_ptr();
}
void check_norm(const at::Tensor& x) {
  NEED(x.dim() >= 1 && real(x.scalar_type()) && x.is_contiguous() && (uintptr_t)x.data_ptr() % 16 == 0);
  const int64_t vec = 16 / x.element_size(), d = x.size(-1);
  NEED(d % vec == 0 && d <= 128 * vec);
}
// norm_forward(x, weight, bias, eps) -> (y,)
PyObject* norm_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 4, [&]() -> PyObject* {
    const at::Tensor x = tensor(a[0]), w = maybe(a[1]), b = maybe(a[2]);
    check_norm(x);
    NEED(PyFloat_Check(a[3]));
    const int64_t d = x.size(-1), rows = x.numel() / d;
    const float *pw = param(w, d, x), *pb = param(b, d, x);
    Place here(x);
    const at::Tensor y = make(x.sizes(), x, x.scalar_type());
    const int r = unlocked([&] {
      return entry.norm_fwd(rows, (int32_t)d, code(x.scalar_type()), (float)PyFloat_AS_DOUBLE(a[3]), x.data_ptr(), d, pw, pb, y.data_ptr(), d,
                            here.stream);
    });
    return r ? PyLong_FromLong(r) : tuple_of({y});
  });
}
// norm_backward(x, weight, dy, eps, need_w, need_b) -> (dx, dw, db), the last two fp32
PyObject* norm_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 6, [&]() -> PyObject* {
    const at::Tensor x = tensor(a[0]), w = maybe(a[1]), dy = tensor(a[2]);
    check_norm(x);
    check_norm(dy);
    NEED(PyFloat_Check(a[3]) && dy.numel() == x.numel() && dy.size(-1) == x.size(-1) && dy.scalar_type() == x.scalar_type() && dy.device() == x.device());
    const int64_t d = x.size(-1), rows = x.numel() / d;
    const float* pw = param(w, d, x);
    Place here(x);
    const at::Tensor dx = make(dy.sizes(), x, x.scalar_type());
    const at::Tensor dw = a[4] == Py_True ? make({d}, x, at::kFloat) : at::Tensor(), db = a[5] == Py_True ? make({d}, x, at::kFloat) : at::Tensor();
    const int r = unlocked([&] {
      return entry.norm_bwd(rows, (int32_t)d, code(x.scalar_type()), (float)PyFloat_AS_DOUBLE(a[3]), x.data_ptr(), d, pw, dy.data_ptr(), d,
                            dx.data_ptr(), dw.defined() ? (float*)dw.data_ptr() : nullptr, db.defined() ? (float*)db.data_ptr() : nullptr, here.stream);
    });
    return r ? PyLong_FromLong(r) : tuple_of({dx, dw, db});
  });
}

// column_sums(g (..., n), a or None) -> (sums (n), d_a or None): all contiguous bf16
PyObject* column_sums(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 2, [&]() -> PyObject* {
    const at::Tensor g = tensor(a[0]), act = maybe(a[1]);
    NEED(g.scalar_type() == at::kBFloat16 && g.dim() >= 1 && g.is_contiguous() && g.size(-1) % 64 == 0 && (uintptr_t)g.data_ptr() % 16 == 0);
    if (act.defined())
      NEED(act.scalar_type() == at::kBFloat16 && act.is_contiguous() && act.sizes() == g.sizes() && act.device() == g.device() &&
           (uintptr_t)act.data_ptr() % 16 == 0);
    const int64_t cols = g.size(-1), rows = g.numel() / cols;
    NEED(cols <= FPB_COLUMN_SUMS_SCRATCH / 4);
    Place here(g);
    const at::Tensor scratch = make({FPB_COLUMN_SUMS_SCRATCH}, g, at::kByte);
    const at::Tensor sums = make({cols}, g, at::kBFloat16), d_a = act.defined() ? make(g.sizes(), g, at::kBFloat16) : at::Tensor();
    const int r = unlocked([&] {
      return entry.column_sums(rows, cols, g.data_ptr(), cols, act.defined() ? act.data_ptr() : nullptr, d_a.defined() ? d_a.data_ptr() : nullptr,
                               scratch.data_ptr(), sums.data_ptr(), here.stream);
    });
    return r ? PyLong_FromLong(r) : tuple_of({sums, d_a});
  });
}

// address(t, dtype, align, device_index, n0, n1) -> address of a contiguous parameter of that shape (n1 = 0: one dimension), or None
PyObject* address(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 6, [&]() -> PyObject* {
    const at::Tensor t = tensor(a[0]);
    NEED(THPDtype_Check(a[1]) && t.scalar_type() == reinterpret_cast<THPDtype*>(a[1])->scalar_type && t.device().index() == integer(a[3]));
    const int64_t n0 = integer(a[4]), n1 = integer(a[5]);
    NEED(t.dim() == (n1 ? 2 : 1) && t.size(0) == n0 && (!n1 || t.size(1) == n1) && t.is_contiguous());
    const uintptr_t p = (uintptr_t)t.data_ptr();
    NEED(p % (uintptr_t)integer(a[2]) == 0);
    return PyLong_FromUnsignedLongLong(p);
  });
}

// wanted(ctx) -> per tensor input of the autograd Function whose backward runs, whether this backward uses its gradient:
// an input that requires none, or that autograd.grad(..., inputs) leaves out, does not (needs_input_grad tells the first only)
PyObject* wanted(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 1 || !THPFunction_Check(a[0])) Py_RETURN_NONE;
  const auto node = reinterpret_cast<THPFunction*>(a[0])->cdata.lock();
  if (!node) Py_RETURN_NONE;
  const Py_ssize_t outputs = (Py_ssize_t)node->num_outputs();
  PyObject* r = PyTuple_New(outputs);
  if (!r) return nullptr;
  for (Py_ssize_t i = 0; i < outputs; ++i) PyTuple_SET_ITEM(r, i, PyBool_FromLong(node->task_should_compute_output((size_t)i)));
  return r;
}

// bind(addresses): the C ABI's entry points in the order of `Entry`
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != ENTRIES) { PyErr_SetString(PyExc_TypeError, "wrong number of entry points"); return nullptr; }
  void* p[ENTRIES];
  for (int i = 0; i < ENTRIES; ++i) {
    p[i] = PyLong_AsVoidPtr(a[i]);
    if (!p[i]) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null entry point"); return nullptr; }
  }
  memcpy(&entry, p, sizeof(entry));
  Py_RETURN_NONE;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(step), FAST(forward), FAST(backward), FAST(suffix_forward), FAST(suffix_backward), FAST(rotary), FAST(gate_forward),
                         FAST(gate_backward), FAST(norm_forward), FAST(norm_backward), FAST(column_sums), FAST(address), FAST(wanted), FAST(bind), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "fpb_fast_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_fpb_fast_calls(void) { return PyModule_Create(&module); }
