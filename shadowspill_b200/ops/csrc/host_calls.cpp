// The hot entry points of ops/functional.py and ops/attention.py in native code: from tensors to the C launchers of
// libss_kernels.so without a Python statement in between. A launch costs about 2.5 us there; reading its operands'
// pointers, sizes and strides, allocating the result and converting a dozen arguments in Python took 6 to 9 us more,
// which bounds models whose kernels are shorter than that.
//
// Every function answers NotImplemented for operands that it does not take as they are, a CPU tensor, another type, a
// stride or an alignment, a wrapped tensor: the caller's Python then decides what becomes of them and words the error.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>

#include "launchers.h"

namespace {

constexpr int kDevices = 64;
int* g_status[kDevices];                 // the devices' status words, set by _lib.status_ptr

struct Refused {};                       // NotImplemented

// Allocations and launches may wait for the GPU, which may wait for another thread.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};
at::Tensor empty(at::IntArrayRef sizes, const at::TensorOptions& options) {
  NoGil free;
  return at::empty(sizes, options);
}

// Kernels enqueued by each launcher's successful calls, which _lib adds to those it counts itself.
enum Entry { GEMM, GEMM2, RESIDUAL, SWIGLU, SWIGLU_BWD, NORM_FWD, NORM_BWD, ROPE, ATTN_FWD, ATTN_BWD, ENTRIES };
const char* const kNames[ENTRIES] = {"ss_gemm_bf16", "ss_gemm2_bf16", "ss_gemm2_residual_bf16", "ss_gemm2_swiglu_bf16",
                                     "ss_gemm2_swiglu_bwd_bf16", "ss_rmsnorm_fwd", "ss_rmsnorm_bwd", "ss_rope",
                                     "ss_attn_fwd", "ss_attn_bwd"};
long long g_launched[ENTRIES];           // under the GIL

struct Failed { const char* what; int rc; };

template <class F, class... A>
void launch(Entry e, F* entry, A... args) {
  int rc;
  {
    NoGil free;
    rc = entry(args...);
  }
  if (rc) throw Failed{kNames[e], rc};
  g_launched[e] += e == ATTN_BWD ? 3 : 1;        // delta, dQ, dK and dV (as _lib counts them)
}

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) throw Refused();
  return THPVariable_Unpack(o);
}
bool none(PyObject* o) { return o == Py_None; }
long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); throw Refused(); }
  return v;
}
double number(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); throw Refused(); }
  return v;
}
void want(bool ok) { if (!ok) throw Refused(); }

// A call's device and where its kernels go. The launchers bind the device of their operands to the thread; where that
// is not the current one already, the Python path keeps its way of doing it.
struct Call {
  int* status;
  void* stream;
  at::TensorOptions bf16, f32;
  explicit Call(const at::Tensor& t) {
    want(t.is_cuda());
    const int dev = t.get_device();
    const auto s = c10::cuda::getCurrentCUDAStream();
    want(dev >= 0 && dev < kDevices && s.device_index() == dev && g_status[dev] != nullptr);
    status = g_status[dev];
    stream = s.stream();
    bf16 = t.options().dtype(at::kBFloat16).requires_grad(false);
    f32 = t.options().dtype(at::kFloat).requires_grad(false);
  }
};
// 2-D bf16 with rows that TMA and 16-byte accesses can take, as functional._plain_rows
void plain_rows(const at::Tensor& t) {
  want(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.stride(1) == 1 && t.stride(0) % 8 == 0 &&
       t.size(1) % 8 == 0 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0);
}
void contiguous(const at::Tensor& t, at::ScalarType type) { want(t.is_cuda() && t.scalar_type() == type && t.is_contiguous()); }

PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

template <class F>
PyObject* guarded(Py_ssize_t given, Py_ssize_t expected, F body) {
  if (given != expected) return PyErr_Format(PyExc_TypeError, "%zd arguments, %zd expected", given, expected);
  try {
    return body();
  } catch (const Refused&) {
    Py_RETURN_NOTIMPLEMENTED;
  } catch (const Failed& e) {
    return PyErr_Format(PyExc_RuntimeError, "%s failed with code %d", e.what, e.rc);
  } catch (...) {                          // of torch: out of memory and the like, as its own calls raise them
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

// gemm(a, b, a_mn, b_mn, out or None, accumulate, alpha)
PyObject* gemm(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 7, [&]() -> PyObject* {
    const at::Tensor &a = tensor(v[0]), &b = tensor(v[1]);
    const int a_mn = v[2] == Py_True, b_mn = v[3] == Py_True;
    plain_rows(a);
    plain_rows(b);
    const Call c(a);
    const int64_t M = a.size(a_mn), K = a.size(!a_mn), N = b.size(b_mn);
    want(b.size(!b_mn) == K && N % 8 == 0 && b.get_device() == a.get_device());
    const int accumulate = v[5] == Py_True;
    at::Tensor made;
    const at::Tensor* out = &made;
    if (none(v[4])) {
      want(!accumulate);
      made = empty({M, N}, c.bf16);
    } else {
      out = &tensor(v[4]);
      want(out->is_cuda() && out->get_device() == a.get_device() && out->dim() == 2 && out->size(0) == M &&
           out->size(1) == N && out->stride(1) == 1 && (reinterpret_cast<uintptr_t>(out->data_ptr()) & 15) == 0);
    }
    const int f32 = out->scalar_type() == at::kFloat;
    want((f32 || out->scalar_type() == at::kBFloat16) && out->stride(0) % (f32 ? 4 : 8) == 0);
    const float alpha = static_cast<float>(number(v[6]));
    if (M >= 256 && N >= 128)
      launch(GEMM2, ss_gemm2_bf16, a.data_ptr(), b.data_ptr(), out->data_ptr(), M, N, K, a.stride(0), b.stride(0),
             out->stride(0), a_mn, b_mn, f32, accumulate, alpha, 0, c.status, c.stream);
    else
      launch(GEMM, ss_gemm_bf16, a.data_ptr(), b.data_ptr(), out->data_ptr(), M, N, K, a.stride(0), b.stride(0),
             out->stride(0), a_mn, b_mn, f32, accumulate, alpha, 0, 0, c.status, c.stream);
    if (none(v[4])) return wrap(std::move(made));
    Py_INCREF(v[4]);
    return v[4];
  });
}

// linear_residual(x, w, residual, out or None)
PyObject* linear_residual(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 4, [&]() -> PyObject* {
    const at::Tensor &x = tensor(v[0]), &w = tensor(v[1]), &res = tensor(v[2]);
    plain_rows(x); plain_rows(w); plain_rows(res);
    const Call c(x);
    const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
    want(K > 0 && w.size(1) == K && res.size(0) == M && res.size(1) == N);    // no launch without a product: no sum either
    at::Tensor made;
    const at::Tensor* out = &made;
    if (none(v[3])) made = empty({M, N}, c.bf16);
    else { out = &tensor(v[3]); plain_rows(*out); want(out->size(0) == M && out->size(1) == N); }
    launch(RESIDUAL, ss_gemm2_residual_bf16, x.data_ptr(), w.data_ptr(), res.data_ptr(), out->data_ptr(), M, N, K,
                                          x.stride(0), w.stride(0), res.stride(0), out->stride(0), c.status, c.stream);
    if (none(v[3])) return wrap(std::move(made));
    Py_INCREF(v[3]);
    return v[3];
  });
}

// swiglu_linear(x, w13, gu or None, out or None, keep_gu) -> (gu or None, h)
PyObject* swiglu_linear(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 5, [&]() -> PyObject* {
    const at::Tensor &x = tensor(v[0]), &w = tensor(v[1]);
    plain_rows(x); plain_rows(w);
    const Call c(x);
    const int64_t T = x.size(0), F2 = w.size(0), K = x.size(1);
    want(w.size(1) == K && F2 % 16 == 0);
    at::Tensor gu, h;
    if (!none(v[2])) { gu = tensor(v[2]); plain_rows(gu); want(gu.size(0) == T && gu.size(1) == F2); }
    else if (v[4] == Py_True) gu = empty({T, F2}, c.bf16);
    if (!none(v[3])) { h = tensor(v[3]); plain_rows(h); want(h.size(0) == T && h.size(1) == F2 / 2); }
    else h = empty({T, F2 / 2}, c.bf16);
    launch(SWIGLU, ss_gemm2_swiglu_bf16, x.data_ptr(), w.data_ptr(), gu.defined() ? gu.data_ptr() : nullptr, h.data_ptr(),
                                        T, F2 / 2, K, x.stride(0), w.stride(0), gu.defined() ? gu.stride(0) : 0,
                                        h.stride(0), c.status, c.stream);
    PyObject* kept = gu.defined() ? wrap(std::move(gu)) : Py_NewRef(Py_None);
    return Py_BuildValue("(NN)", kept, wrap(std::move(h)));
  });
}

// swiglu_linear_dgrad(dy, w2, gu)
PyObject* swiglu_linear_dgrad(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 3, [&]() -> PyObject* {
    const at::Tensor &dy = tensor(v[0]), &w = tensor(v[1]), &gu = tensor(v[2]);
    plain_rows(dy); plain_rows(w); plain_rows(gu);
    const Call c(dy);
    const int64_t T = dy.size(0), F = w.size(1), K = dy.size(1);
    want(w.size(0) == K && gu.size(0) == T && gu.size(1) == 2 * F);
    at::Tensor dgu = empty({T, 2 * F}, c.bf16);
    launch(SWIGLU_BWD, ss_gemm2_swiglu_bwd_bf16, dy.data_ptr(), w.data_ptr(), gu.data_ptr(), dgu.data_ptr(), T, F, K,
                                            dy.stride(0), w.stride(0), gu.stride(0), dgu.stride(0), c.status, c.stream);
    return wrap(std::move(dgu));
  });
}

// rmsnorm_fwd(x, w, eps, zero_centered, delta or None, out or None, rstd or None) -> (y, rstd)
PyObject* rmsnorm_fwd(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 7, [&]() -> PyObject* {
    const at::Tensor &x = tensor(v[0]), &w = tensor(v[1]);
    contiguous(x, at::kBFloat16); contiguous(w, at::kBFloat16);
    want(x.dim() == 2 && w.numel() == x.size(1));
    const Call c(x);
    at::Tensor y, rs;
    const void* delta = nullptr;
    if (!none(v[4])) { const at::Tensor& d = tensor(v[4]); contiguous(d, at::kBFloat16); want(d.numel() == x.numel()); delta = d.data_ptr(); }
    if (!none(v[5])) { y = tensor(v[5]); contiguous(y, at::kBFloat16); want(y.numel() == x.numel()); }
    else y = empty({x.size(0), x.size(1)}, c.bf16);
    if (!none(v[6])) { rs = tensor(v[6]); contiguous(rs, at::kFloat); want(rs.numel() == x.size(0)); }
    else rs = empty({x.size(0)}, c.f32);
    launch(NORM_FWD, ss_rmsnorm_fwd, x.data_ptr(), delta, w.data_ptr(), y.data_ptr(), static_cast<float*>(rs.data_ptr()),
                                  x.size(0), x.size(1), static_cast<float>(number(v[2])), v[3] == Py_True, c.status,
                                  c.stream);
    return Py_BuildValue("(NN)", wrap(std::move(y)), wrap(std::move(rs)));
  });
}

// rmsnorm_bwd(x, w, gy, rstd, dw or None, zero_centered, dx or None, accumulate) -> dx
PyObject* rmsnorm_bwd(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 8, [&]() -> PyObject* {
    const at::Tensor &x = tensor(v[0]), &w = tensor(v[1]), &gy = tensor(v[2]), &rs = tensor(v[3]);
    contiguous(x, at::kBFloat16); contiguous(w, at::kBFloat16); contiguous(gy, at::kBFloat16); contiguous(rs, at::kFloat);
    want(x.dim() == 2 && w.numel() == x.size(1) && gy.numel() == x.numel() && rs.numel() == x.size(0));
    const Call c(x);
    float* dw = nullptr;
    if (!none(v[4])) { const at::Tensor& d = tensor(v[4]); contiguous(d, at::kFloat); want(d.numel() == x.size(1)); dw = static_cast<float*>(d.data_ptr()); }
    const int accumulate = v[7] == Py_True;
    at::Tensor dx;
    if (!none(v[6])) { dx = tensor(v[6]); contiguous(dx, at::kBFloat16); want(dx.numel() == x.numel()); }
    else { want(!accumulate); dx = empty({x.size(0), x.size(1)}, c.bf16); }
    launch(NORM_BWD, ss_rmsnorm_bwd, x.data_ptr(), w.data_ptr(), gy.data_ptr(), static_cast<const float*>(rs.data_ptr()),
                                  dx.data_ptr(), dw, x.size(0), x.size(1), v[5] == Py_True, accumulate, c.status, c.stream);
    return wrap(std::move(dx));
  });
}

// rope_(buf, positions, col0, heads, dh, rot, theta, inverse) -> buf
PyObject* rope(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 8, [&]() -> PyObject* {
    const at::Tensor &buf = tensor(v[0]), &pos = tensor(v[1]);
    want(buf.is_cuda() && buf.scalar_type() == at::kBFloat16 && buf.dim() == 2 && buf.stride(1) == 1);
    contiguous(pos, at::kInt);
    want(pos.numel() == buf.size(0));
    const Call c(buf);
    launch(ROPE, ss_rope, buf.data_ptr(), static_cast<const int*>(pos.data_ptr()), buf.size(0), buf.stride(0),
                           integer(v[2]), integer(v[3]), integer(v[4]), integer(v[5]), static_cast<float>(number(v[6])),
                           v[7] == Py_True, c.stream);
    Py_INCREF(v[0]);
    return v[0];
  });
}

// [T, heads, dh] with adjacent heads; the row pitch
int64_t rows3(const at::Tensor& t, int64_t T, int64_t heads, int64_t dh) {
  want(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 3 && t.size(0) == T && t.size(1) == heads &&
       t.size(2) == dh && t.stride(2) == 1 && t.stride(1) == dh);
  return t.stride(0);
}
float attention_scale(PyObject* o, int64_t dh) {
  return static_cast<float>(none(o) ? 1.0 / std::sqrt(static_cast<double>(dh)) : number(o));
}

// attention_fwd(q, k, v, cu_seqlens, scale or None, out or None, lse or None) -> (out, lse)
PyObject* attention_fwd(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 7, [&]() -> PyObject* {
    const at::Tensor &q = tensor(v[0]), &k = tensor(v[1]), &vv = tensor(v[2]), &cu = tensor(v[3]);
    want(q.dim() == 3 && k.dim() == 3);
    const int64_t T = q.size(0), H = q.size(1), dh = q.size(2), Hk = k.size(1);
    want(Hk > 0);
    const int64_t ldq = rows3(q, T, H, dh), ldk = rows3(k, T, Hk, dh), ldv = rows3(vv, T, Hk, dh);
    contiguous(cu, at::kInt);
    const Call c(q);
    at::Tensor out, lse;
    if (!none(v[5])) out = tensor(v[5]);
    else out = empty({T, H, dh}, c.bf16);
    const int64_t ldo = rows3(out, T, H, dh);
    if (!none(v[6])) { lse = tensor(v[6]); contiguous(lse, at::kFloat); want(lse.numel() == H * T); }
    else lse = empty({H, T}, c.f32);
    launch(ATTN_FWD, ss_attn_fwd, q.data_ptr(), k.data_ptr(), vv.data_ptr(), out.data_ptr(), static_cast<float*>(lse.data_ptr()),
                               static_cast<const int*>(cu.data_ptr()), cu.numel() - 1, T, H, Hk, dh, ldq, ldk, ldv, ldo,
                               attention_scale(v[4], dh), c.status, c.stream);
    return Py_BuildValue("(NN)", wrap(std::move(out)), wrap(std::move(lse)));
  });
}

// attention_bwd(q, k, v, out, lse, dout, cu_seqlens, scale or None, dq, dk, dv (or None each)) -> (dq, dk, dv)
PyObject* attention_bwd(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 11, [&]() -> PyObject* {
    const at::Tensor &q = tensor(v[0]), &k = tensor(v[1]), &vv = tensor(v[2]), &out = tensor(v[3]), &lse = tensor(v[4]),
                     &dout = tensor(v[5]), &cu = tensor(v[6]);
    want(q.dim() == 3 && k.dim() == 3);
    const int64_t T = q.size(0), H = q.size(1), dh = q.size(2), Hk = k.size(1);
    want(Hk > 0);
    const int64_t ldq = rows3(q, T, H, dh), ldk = rows3(k, T, Hk, dh), ldv = rows3(vv, T, Hk, dh),
                  ldo = rows3(dout, T, H, dh);
    contiguous(out, at::kBFloat16);
    contiguous(lse, at::kFloat);
    contiguous(cu, at::kInt);
    want(out.numel() == T * H * dh && lse.numel() == H * T);
    const Call c(q);
    at::Tensor g[3];
    const int64_t heads[3] = {H, Hk, Hk};
    int64_t ld[3];
    for (int i = 0; i < 3; ++i) {
      if (none(v[8 + i])) g[i] = empty({T, heads[i], dh}, c.bf16);
      else g[i] = tensor(v[8 + i]);
      ld[i] = rows3(g[i], T, heads[i], dh);
    }
    at::Tensor delta = empty({H, T}, c.f32);          // kernel scratch
    launch(ATTN_BWD, ss_attn_bwd_g, q.data_ptr(), k.data_ptr(), vv.data_ptr(), out.data_ptr(),
                                 static_cast<const float*>(lse.data_ptr()), dout.data_ptr(), g[0].data_ptr(),
                                 g[1].data_ptr(), g[2].data_ptr(), static_cast<const int*>(cu.data_ptr()),
                                 static_cast<float*>(delta.data_ptr()), cu.numel() - 1, T, H, Hk, dh, ldq, ldk, ldv, ldo,
                                 ld[0], ld[1], ld[2], attention_scale(v[7], dh), c.status, c.stream);
    return Py_BuildValue("(NNN)", wrap(std::move(g[0])), wrap(std::move(g[1])), wrap(std::move(g[2])));
  });
}

// set_status(device, address)
PyObject* set_status(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded(n, 2, [&]() -> PyObject* {
    const long long dev = integer(v[0]), ptr = integer(v[1]);
    want(dev >= 0 && dev < kDevices);
    g_status[dev] = reinterpret_cast<int*>(ptr);
    Py_RETURN_NONE;
  });
}

// launched() -> {launcher: kernels}
PyObject* launched(PyObject*, PyObject* const*, Py_ssize_t n) {
  return guarded(n, 0, [&]() -> PyObject* {
    PyObject* d = PyDict_New();
    for (int e = 0; d != nullptr && e < ENTRIES; ++e) {
      PyObject* count = PyLong_FromLongLong(g_launched[e]);
      if (count == nullptr || (g_launched[e] && PyDict_SetItemString(d, kNames[e], count))) Py_CLEAR(d);
      Py_XDECREF(count);
    }
    return d;
  });
}

#define SS_CALL(name) {#name, reinterpret_cast<PyCFunction>(name), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {SS_CALL(gemm), SS_CALL(linear_residual), SS_CALL(swiglu_linear), SS_CALL(swiglu_linear_dgrad),
                         SS_CALL(rmsnorm_fwd), SS_CALL(rmsnorm_bwd), SS_CALL(rope), SS_CALL(attention_fwd),
                         SS_CALL(attention_bwd), SS_CALL(set_status), SS_CALL(launched), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_calls", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host_calls() { return PyModule_Create(&module); }
