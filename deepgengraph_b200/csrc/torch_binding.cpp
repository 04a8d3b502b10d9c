// Host path of the public operators: one CPython call from argument checks to kernel launch.
//
// A call on a short problem is bound by the host, not by the GPU: through ctypes the checks, the output allocation and the
// stream look-up cost 8 us (bandwidth ops) to 19 us (attention) of Python per call, where the kernels take 3 to 10 us.  The
// functions here take the same arguments, allocate outputs and scratch from torch's caching allocator and enter the C ABI.
//
// Every function handles the regular case only -- plain CUDA tensors on the current device that satisfy the operator's
// contract -- and returns None otherwise, after which the Python operator runs its own checks and raises the error it
// documents (or switches devices, or dispatches a tensor subclass).  A non-zero status of the library also returns None.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>

#include "../../include/b200attn.h"

namespace {

using at::Tensor;

// ---------------------------------------------------------------- arguments
const Tensor* tensor_arg(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;   // subclasses (fake tensors, ...) take the Python path
  const Tensor& t = THPVariable_Unpack(o);
  return t.defined() && t.is_cuda() && t.has_storage() ? &t : nullptr;
}

bool float_arg(PyObject* o, double* v) {
  if (PyFloat_CheckExact(o)) {
    *v = PyFloat_AS_DOUBLE(o);
    return true;
  }
  if (!PyLong_CheckExact(o)) return false;
  *v = PyLong_AsDouble(o);
  if (*v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

bool int_arg(PyObject* o, int* v) {
  if (!PyLong_Check(o)) return false;
  int overflow = 0;
  const long x = PyLong_AsLongAndOverflow(o, &overflow);
  if (overflow != 0 || x < INT32_MIN || x > INT32_MAX) return false;
  *v = (int)x;
  return true;
}

bool bool_arg(PyObject* o, bool* v) {
  if (!PyBool_Check(o)) return false;
  *v = o == Py_True;
  return true;
}

// softmax scale: None or a non-positive number selects 1 / sqrt(head_dim); the library refuses a NaN
bool scale_arg(PyObject* o, int64_t head_dim, float* v) {
  double s = 0.0;
  if (o != Py_None && (!float_arg(o, &s) || std::isnan(s))) return false;
  *v = (float)(s > 0.0 ? s : 1.0 / std::sqrt((double)head_dim));
  return true;
}

int dtype_code(at::ScalarType t) {
  return t == at::kHalf ? B200_F16 : t == at::kBFloat16 ? B200_BF16 : t == at::kFloat ? B200_F32 : -1;
}

// the device all tensors are on, if it is the current one; -1 otherwise
int common_device(std::initializer_list<const Tensor*> ts) {
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return -1;
  int dev = -1;
  for (const Tensor* t : ts) {
    if (t == nullptr) return -1;
    const int d = t->device().index();
    if (dev >= 0 && d != dev) return -1;
    dev = d;
  }
  return dev >= 0 && dev == (int)c10::cuda::current_device() ? dev : -1;
}

void* stream_of(int dev) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(); }

Tensor empty(at::IntArrayRef sizes, at::ScalarType type, int dev) {
  return Tensor(at::detail::empty_cuda(sizes, type, c10::Device(c10::kCUDA, (c10::DeviceIndex)dev), std::nullopt));
}

// Runs `call` (a C-ABI entry point, which may block while the launch queue is full) without the interpreter lock.
template <class F>
int without_gil(F call) {
  PyThreadState* state = PyEval_SaveThread();
  const int rc = call();
  PyEval_RestoreThread(state);
  return rc;
}

PyObject* tuple_of(std::initializer_list<Tensor> ts) {
  PyObject* out = PyTuple_New((Py_ssize_t)ts.size());
  if (out == nullptr) return nullptr;
  Py_ssize_t i = 0;
  for (const Tensor& t : ts) PyTuple_SET_ITEM(out, i++, THPVariable_Wrap(t));
  return out;
}

// Exceptions of the allocator (out of memory) become Python exceptions of the type torch itself raises: the Python path
// is taken, whose own allocation then fails with it.
template <class F>
PyObject* guarded(F body) {
  try {
    return body();
  } catch (const std::exception&) {
    if (PyErr_Occurred()) PyErr_Clear();
    Py_RETURN_NONE;
  }
}

// ---------------------------------------------------------------- attention
struct Qkv {
  const Tensor *q, *k, *v;
  int dev, dtype;
  int64_t B, Sq, Skv, H, Hk, D;
  bool contiguous;
};

// [B, S, H, D] view whose heads are packed inside (possibly wider) token rows
bool row_strided(const Tensor& t) {
  const auto sz = t.sizes();
  const auto st = t.strides();
  return st[3] == 1 && st[2] == sz[3] && st[1] >= sz[2] * sz[3] && st[1] % 8 == 0 &&
         (sz[0] == 1 || (st[0] >= sz[1] * st[1] && st[0] % 8 == 0));
}

bool parse_qkv(PyObject* const* args, bool allow_strided, Qkv* p) {
  p->q = tensor_arg(args[0]);
  p->k = tensor_arg(args[1]);
  p->v = tensor_arg(args[2]);
  p->dev = common_device({p->q, p->k, p->v});
  if (p->dev < 0) return false;
  const Tensor &q = *p->q, &k = *p->k, &v = *p->v;
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4) return false;
  const auto type = q.scalar_type();
  if ((type != at::kHalf && type != at::kBFloat16) || k.scalar_type() != type || v.scalar_type() != type) return false;
  p->dtype = dtype_code(type);
  const auto qs = q.sizes(), ks = k.sizes();
  p->B = qs[0], p->Sq = qs[1], p->H = qs[2], p->D = qs[3], p->Skv = ks[1], p->Hk = ks[2];
  if (v.sizes() != ks || ks[0] != p->B || ks[3] != p->D || p->Hk <= 0 || p->H % p->Hk != 0) return false;
  if (p->B <= 0 || p->Sq <= 0 || p->Skv <= 0 || p->B > INT32_MAX || p->Sq > INT32_MAX || p->Skv > INT32_MAX) return false;
  p->contiguous = q.is_contiguous() && k.is_contiguous() && v.is_contiguous();
  return p->contiguous || (allow_strided && row_strided(q) && row_strided(k) && row_strided(v));
}

void strides_of(const Tensor& t, int64_t* token, int64_t* batch) {
  *token = t.stride(1);
  *batch = t.size(0) > 1 ? t.stride(0) : t.size(1) * t.stride(1);
}

// attn_fwd(q, k, v, causal, window, softcap, scale, want_lse) -> out | (out, lse) | None
PyObject* attn_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Qkv p;
    bool causal, want_lse;
    int window;
    double softcap;
    float scale;
    if (n != 8 || !parse_qkv(args, true, &p) || !bool_arg(args[3], &causal) || !int_arg(args[4], &window) ||
        !float_arg(args[5], &softcap) || !scale_arg(args[6], p.D, &scale) || !bool_arg(args[7], &want_lse))
      Py_RETURN_NONE;
    Tensor out = empty({p.B, p.Sq, p.H, p.D}, p.q->scalar_type(), p.dev), lse;
    if (want_lse) lse = empty({p.B, p.H, p.Sq}, at::kFloat, p.dev);
    float* lse_ptr = want_lse ? static_cast<float*>(lse.data_ptr()) : nullptr;
    const void *q = p.q->data_ptr(), *k = p.k->data_ptr(), *v = p.v->data_ptr();
    void *o = out.data_ptr(), *stream = stream_of(p.dev);
    int64_t qt, qb, kt, kb, vt, vb;
    strides_of(*p.q, &qt, &qb);
    strides_of(*p.k, &kt, &kb);
    strides_of(*p.v, &vt, &vb);
    const int rc = without_gil([&] {
      if (p.contiguous)
        return b200_attn_fwd(q, k, v, o, lse_ptr, (int)p.B, (int)p.Sq, (int)p.Skv, (int)p.H, (int)p.Hk, (int)p.D, p.dtype,
                             causal, window, (float)softcap, scale, stream);
      return b200_attn_fwd_strided(q, k, v, o, lse_ptr, (int)p.B, (int)p.Sq, (int)p.Skv, (int)p.H, (int)p.Hk, (int)p.D,
                                   p.dtype, qt, qb, kt, kb, vt, vb, causal, window, (float)softcap, scale, stream);
    });
    if (rc != B200_OK) Py_RETURN_NONE;
    return want_lse ? tuple_of({out, lse}) : THPVariable_Wrap(out);
  });
}

struct Workspace {
  Tensor buffer;
  void* ptr;
  int64_t bytes;
};
Workspace score_workspace(const Qkv& p) {
  Workspace w;
  w.bytes = b200_attn_score_workspace_bytes((int)p.B, (int)p.Sq, (int)p.Skv, (int)p.H);
  w.buffer = empty({w.bytes}, at::kByte, p.dev);
  w.ptr = w.buffer.data_ptr();
  return w;
}

// attn_score(q, k, v, want_sq, causal, window, softcap, scale) -> (out, colsum[, colsum_sq]) | None
PyObject* attn_score(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Qkv p;
    bool want_sq, causal;
    int window;
    double softcap;
    float scale;
    if (n != 8 || !parse_qkv(args, false, &p) || !bool_arg(args[3], &want_sq) || !bool_arg(args[4], &causal) ||
        !int_arg(args[5], &window) || !float_arg(args[6], &softcap) || !scale_arg(args[7], p.D, &scale))
      Py_RETURN_NONE;
    Tensor out = empty(p.q->sizes(), p.q->scalar_type(), p.dev), score = empty({p.B, p.Hk, p.Skv}, at::kFloat, p.dev), sq;
    if (want_sq) sq = empty({p.B, p.Hk, p.Skv}, at::kFloat, p.dev);
    const Workspace ws = score_workspace(p);
    const void *q = p.q->data_ptr(), *k = p.k->data_ptr(), *v = p.v->data_ptr();
    float *s1 = static_cast<float*>(score.data_ptr()), *s2 = want_sq ? static_cast<float*>(sq.data_ptr()) : nullptr;
    void *o = out.data_ptr(), *stream = stream_of(p.dev);
    const int rc = without_gil([&] {
      return b200_attn_score_gqa(q, k, v, o, s1, s2, nullptr, ws.ptr, ws.bytes, (int)p.B, (int)p.Sq, (int)p.Skv, (int)p.H,
                                 (int)p.Hk, (int)p.D, p.dtype, causal, window, (float)softcap, scale, stream);
    });
    if (rc != B200_OK) Py_RETURN_NONE;
    return want_sq ? tuple_of({out, score, sq}) : tuple_of({out, score});
  });
}

// attn_snapkv(q, k, v, kernel_size, causal, scale) -> (out, pooled) | None
PyObject* attn_snapkv(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Qkv p;
    int kernel;
    bool causal;
    float scale;
    if (n != 6 || !parse_qkv(args, false, &p) || !int_arg(args[3], &kernel) || !bool_arg(args[4], &causal) ||
        !scale_arg(args[5], p.D, &scale))
      Py_RETURN_NONE;
    Tensor out = empty(p.q->sizes(), p.q->scalar_type(), p.dev), score = empty({p.B, p.Hk, p.Skv}, at::kFloat, p.dev);
    Tensor pooled = empty({p.B, p.Hk, p.Skv}, at::kFloat, p.dev);
    const Workspace ws = score_workspace(p);
    const void *q = p.q->data_ptr(), *k = p.k->data_ptr(), *v = p.v->data_ptr();
    float *s1 = static_cast<float*>(score.data_ptr()), *s2 = static_cast<float*>(pooled.data_ptr());
    void *o = out.data_ptr(), *stream = stream_of(p.dev);
    const int rc = without_gil([&] {
      const int st = b200_attn_score_gqa(q, k, v, o, s1, nullptr, nullptr, ws.ptr, ws.bytes, (int)p.B, (int)p.Sq,
                                         (int)p.Skv, (int)p.H, (int)p.Hk, (int)p.D, p.dtype, causal, -1, 0.f, scale, stream);
      return st != B200_OK ? st : b200_avg_pool1d_f32(s1, s2, p.B * p.Hk, (int)p.Skv, kernel, stream);
    });
    if (rc != B200_OK) Py_RETURN_NONE;
    return tuple_of({out, pooled});
  });
}

// attn_corm(q, k, v, causal, scale) -> (out, bool flags) | None
PyObject* attn_corm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Qkv p;
    bool causal;
    float scale;
    if (n != 5 || !parse_qkv(args, false, &p) || !bool_arg(args[3], &causal) || !scale_arg(args[4], p.D, &scale))
      Py_RETURN_NONE;
    Tensor out = empty(p.q->sizes(), p.q->scalar_type(), p.dev), score = empty({p.B, p.Hk, p.Skv}, at::kFloat, p.dev);
    Tensor flags = empty({p.B, p.Hk, p.Skv}, at::kBool, p.dev);
    const Workspace ws = score_workspace(p);
    const void *q = p.q->data_ptr(), *k = p.k->data_ptr(), *v = p.v->data_ptr();
    float* s1 = static_cast<float*>(score.data_ptr());
    uint8_t* f = static_cast<uint8_t*>(flags.data_ptr());
    void *o = out.data_ptr(), *stream = stream_of(p.dev);
    const int rc = without_gil([&] {
      return b200_attn_score_gqa(q, k, v, o, s1, nullptr, f, ws.ptr, ws.bytes, (int)p.B, (int)p.Sq, (int)p.Skv, (int)p.H,
                                 (int)p.Hk, (int)p.D, p.dtype, causal, 0, 0.f, scale, stream);
    });
    if (rc != B200_OK) Py_RETURN_NONE;
    return tuple_of({out, flags});
  });
}

// attn_kf(q, k, v, exp_rand | None, seed, tau, causal, scale) -> (out, kf_score) | None
PyObject* attn_kf(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Qkv p;
    bool causal;
    double tau;
    float scale;
    if (n != 8 || !parse_qkv(args, false, &p) || !PyLong_Check(args[4]) || !float_arg(args[5], &tau) ||
        !bool_arg(args[6], &causal) || !scale_arg(args[7], p.D, &scale))
      Py_RETURN_NONE;
    const float* noise = nullptr;
    if (args[3] != Py_None) {
      const Tensor* e = tensor_arg(args[3]);
      if (common_device({p.q, e}) < 0 || e->scalar_type() != at::kFloat || !e->is_contiguous() ||
          e->sizes() != at::IntArrayRef({p.B, p.H, p.Sq, p.Skv}))
        Py_RETURN_NONE;
      noise = static_cast<const float*>(e->data_ptr());
    }
    const uint64_t seed = PyLong_AsUnsignedLongLongMask(args[4]);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    Tensor out = empty(p.q->sizes(), p.q->scalar_type(), p.dev), score = empty({p.B, p.Hk, p.Skv}, at::kFloat, p.dev);
    const Workspace ws = score_workspace(p);
    const void *q = p.q->data_ptr(), *k = p.k->data_ptr(), *v = p.v->data_ptr();
    float* s1 = static_cast<float*>(score.data_ptr());
    void *o = out.data_ptr(), *stream = stream_of(p.dev);
    const int rc = without_gil([&] {
      if (noise != nullptr)
        return b200_attn_kf_score_gqa(q, k, v, noise, o, s1, ws.ptr, ws.bytes, (int)p.B, (int)p.Sq, (int)p.Skv, (int)p.H,
                                      (int)p.Hk, (int)p.D, p.dtype, causal, (float)tau, scale, stream);
      return b200_attn_kf_score_seeded(q, k, v, seed, o, s1, ws.ptr, ws.bytes, (int)p.B, (int)p.Sq, (int)p.Skv, (int)p.H,
                                       (int)p.Hk, (int)p.D, p.dtype, causal, (float)tau, scale, stream);
    });
    if (rc != B200_OK) Py_RETURN_NONE;
    return tuple_of({out, score});
  });
}

// ---------------------------------------------------------------- eviction
// kv_evict(score, score_sq | None, k, v, q_len, budget, recent, return_indices) -> kv_cache | (kv_cache, indices) | None
PyObject* kv_evict(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 8) Py_RETURN_NONE;
    const bool roco = args[1] != Py_None;
    const Tensor *s = tensor_arg(args[0]), *s2 = roco ? tensor_arg(args[1]) : s, *k = tensor_arg(args[2]),
                 *v = tensor_arg(args[3]);
    int q_len, budget, recent;
    bool want_idx;
    const int dev = common_device({s, s2, k, v});
    if (dev < 0 || !int_arg(args[4], &q_len) || !int_arg(args[5], &budget) || !int_arg(args[6], &recent) ||
        !bool_arg(args[7], &want_idx))
      Py_RETURN_NONE;
    if (s->dim() != 3 || s->scalar_type() != at::kFloat || !s->is_contiguous() || s2->scalar_type() != at::kFloat ||
        !s2->is_contiguous() || s2->sizes() != s->sizes())
      Py_RETURN_NONE;
    if (k->dim() != 4 || v->sizes() != k->sizes() || k->scalar_type() != v->scalar_type() || !k->is_contiguous() ||
        !v->is_contiguous() || dtype_code(k->scalar_type()) < 0)
      Py_RETURN_NONE;
    const int64_t B = k->size(0), S = k->size(1), H = k->size(2), D = k->size(3), keep = (int64_t)budget + recent;
    if (s->sizes() != at::IntArrayRef({B, H, S}) || budget < 0 || recent < 0 || keep <= 0 || keep > S || B <= 0 || H <= 0 ||
        S > INT32_MAX || B > INT32_MAX)
      Py_RETURN_NONE;
    Tensor cache = empty({B, 2, keep, H, D}, k->scalar_type(), dev), idx;
    if (want_idx) idx = empty({B, H, keep}, at::kInt, dev);
    int32_t* ip = want_idx ? static_cast<int32_t*>(idx.data_ptr()) : nullptr;
    const float *sp = static_cast<const float*>(s->data_ptr()), *sp2 = static_cast<const float*>(s2->data_ptr());
    const void *kp = k->data_ptr(), *vp = v->data_ptr();
    void *cp = cache.data_ptr(), *stream = stream_of(dev);
    const int type = dtype_code(k->scalar_type());
    const int rc = without_gil([&] {
      if (roco)
        return b200_kv_evict_roco(sp, sp2, kp, vp, cp, ip, (int)B, (int)S, (int)H, (int)D, q_len, budget, recent, type,
                                  stream);
      return b200_kv_evict_topk(sp, kp, vp, cp, ip, (int)B, (int)S, (int)H, (int)D, budget, type, stream);
    });
    if (rc != B200_OK) Py_RETURN_NONE;
    return want_idx ? tuple_of({cache, idx}) : THPVariable_Wrap(cache);
  });
}

// ---------------------------------------------------------------- bandwidth ops
// These write into tensors of the caller and return True when the kernel was launched, None otherwise.

// norm(out | None, input, residual | None, weight, epsilon): rms_norm, or fused_add_rms_norm when residual is given
PyObject* norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 5) Py_RETURN_NONE;
    const bool add = args[2] != Py_None;
    const Tensor *x = tensor_arg(args[1]), *other = tensor_arg(add ? args[2] : args[0]), *w = tensor_arg(args[3]);
    double eps;
    const int dev = common_device({x, other, w});
    if (dev < 0 || !float_arg(args[4], &eps) || x->dim() < 1) Py_RETURN_NONE;
    const int64_t hidden = x->size(-1);
    const auto type = x->scalar_type();
    const int code = dtype_code(type);
    if (code < 0 || other->scalar_type() != type || w->scalar_type() != type || other->sizes() != x->sizes() ||
        w->numel() != hidden || hidden <= 0 || hidden > INT32_MAX || !x->is_contiguous() || !other->is_contiguous() ||
        !w->is_contiguous())
      Py_RETURN_NONE;
    const int64_t tokens = x->numel() / hidden;
    void *xp = x->data_ptr(), *op = other->data_ptr(), *stream = stream_of(dev);
    const void* wp = w->data_ptr();
    const int rc = without_gil([&] {
      return add ? b200_fused_add_rms_norm(xp, op, wp, (float)eps, tokens, (int)hidden, code, stream)
                 : b200_rms_norm(op, xp, wp, (float)eps, tokens, (int)hidden, code, stream);
    });
    if (rc != B200_OK) Py_RETURN_NONE;
    Py_RETURN_TRUE;
  });
}

// act_and_mul(out, input, gelu)
PyObject* act_and_mul(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    bool gelu;
    if (n != 3 || !bool_arg(args[2], &gelu)) Py_RETURN_NONE;
    const Tensor *out = tensor_arg(args[0]), *in = tensor_arg(args[1]);
    const int dev = common_device({out, in});
    if (dev < 0 || in->dim() < 1 || out->dim() != in->dim()) Py_RETURN_NONE;
    const int64_t two_d = in->size(-1), d = two_d / 2;
    const int code = dtype_code(in->scalar_type());
    if (code < 0 || out->scalar_type() != in->scalar_type() || two_d != 2 * d || d <= 0 || d > INT32_MAX ||
        out->size(-1) != d || out->sizes().slice(0, out->dim() - 1) != in->sizes().slice(0, in->dim() - 1) ||
        !out->is_contiguous() || !in->is_contiguous())
      Py_RETURN_NONE;
    const int64_t tokens = in->numel() / two_d;
    void *op = out->data_ptr(), *stream = stream_of(dev);
    const void* ip = in->data_ptr();
    const int rc = without_gil([&] {
      return gelu ? b200_gelu_tanh_and_mul(op, ip, tokens, (int)d, code, stream)
                  : b200_silu_and_mul(op, ip, tokens, (int)d, code, stream);
    });
    if (rc != B200_OK) Py_RETURN_NONE;
    Py_RETURN_TRUE;
  });
}

// uniformly strided rows [tokens, width]: the token stride, or -1
int64_t uniform_row_stride(const Tensor& t) {
  const int64_t nd = t.dim();
  int64_t stride = t.stride(nd - 2), span = t.size(nd - 2) * stride;
  for (int64_t i = nd - 3; i >= 0; --i) {   // leading dimensions continue the same progression
    if (t.size(i) != 1 && t.stride(i) != span) return -1;
    span *= t.size(i);
  }
  return stride;
}

// rotary(positions, query, key, head_size, theta)
PyObject* rotary(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    int head;
    double theta;
    if (n != 5 || !int_arg(args[3], &head) || !float_arg(args[4], &theta) || head <= 0) Py_RETURN_NONE;
    const Tensor *pos = tensor_arg(args[0]), *q = tensor_arg(args[1]), *k = tensor_arg(args[2]);
    const int dev = common_device({pos, q, k});
    if (dev < 0 || pos->scalar_type() != at::kInt || !pos->is_contiguous() || q->scalar_type() != k->scalar_type())
      Py_RETURN_NONE;
    const int code = dtype_code(q->scalar_type());
    if (code < 0 || q->dim() < 2 || k->dim() < 2 || q->stride(-1) != 1 || k->stride(-1) != 1) Py_RETURN_NONE;
    const int64_t qw = q->size(-1), kw = k->size(-1);
    if (qw <= 0 || kw <= 0 || qw % head != 0 || kw % head != 0) Py_RETURN_NONE;
    const int64_t tokens = q->numel() / qw;
    if (tokens <= 0 || k->numel() / kw != tokens || pos->numel() != tokens) Py_RETURN_NONE;
    const int64_t qs = uniform_row_stride(*q), ks = uniform_row_stride(*k);
    if (qs < qw || ks < kw) Py_RETURN_NONE;
    const int32_t* pp = static_cast<const int32_t*>(pos->data_ptr());
    void *qp = q->data_ptr(), *kp = k->data_ptr(), *stream = stream_of(dev);
    const int rc = without_gil([&] {
      return b200_rotary_embedding_online(pp, qp, kp, tokens, (int)(qw / head), (int)(kw / head), head, qs, ks, (float)theta,
                                          code, stream);
    });
    if (rc != B200_OK) Py_RETURN_NONE;
    Py_RETURN_TRUE;
  });
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {FAST(attn_fwd), FAST(attn_score), FAST(attn_snapkv), FAST(attn_corm), FAST(attn_kf),
                          FAST(kv_evict), FAST(norm), FAST(act_and_mul), FAST(rotary), {nullptr, nullptr, 0, nullptr}};
#undef FAST
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "b200torch", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_b200torch() { return PyModule_Create(&kModule); }
