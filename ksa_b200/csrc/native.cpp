// The ordinary calls of the operators in native code: argument checks, output tensors and launches of one operator in one call
// from Python.  The calls of a decode step or a short prompt are bound by the host (a projection through Python and ctypes took
// 17 to 19 us, of which the launch itself is 4), and so is a training step on short sequences.
//
// Every function takes plain tensors only (dense CUDA tensors of this device without conjugation, wrappers or subclasses) in the
// forms that its kernels take as they are, and returns None for anything else: the Python operator then goes its general way,
// with its own checks, errors and copies.  Nothing is kept between calls.
//
// This file knows torch, the kernel library does not: it calls the library's C entry points like any other user.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <pybind11/pybind11.h>

#include <atomic>
#include <tuple>

extern "C" {
const char* ksa_last_error();
int ksa_gemm_on_pairs(int M, int N, int pair_min_tiles);
int ksa_gemm_narrow_plan(int M, int N, int K, int glu, int pair_min_tiles, int ragged);
int ksa_gemm_tall_plan(int M, int N, int K, int glu, int ragged);
int ksa_gemm_tall_bf16(const void* x, const void* w, void* c, int M, int N, int K, long long ldx, long long ldw, long long ldc, int glu,
                       int columns, int split, void* stream);
int ksa_rmsnorm_bwd_parts(int rows);
int ksa_attn_bwd_num_segments(int lq);
int ksa_gemm_bf16(const void* a, const void* b, void* c, int M, int N, int K, long long lda, long long ldb, long long ldc,
                  int a_mn_major, int b_mn_major, int out_fp32, int accumulate, float alpha, int sm_limit, void* stream);
int ksa_gemm2_bf16(const void* a, const void* b, void* c, int M, int N, int K, long long lda, long long ldb, long long ldc,
                   int a_mn_major, int b_mn_major, int out_fp32, int accumulate, float alpha, void* stream);
int ksa_gemm_narrow_bf16(const void* x, const void* w, void* c, int M, int N, int K, long long ldx, long long ldw, long long ldc,
                         int w_mn_major, int glu, int bt, int split, float alpha, void* stream);
int ksa_gemm2_swiglu_bf16(const void* a, const void* b, void* gu, void* h, int M, int F, int K, long long lda, long long ldb,
                          long long ld_gu, long long ld_h, void* stream);
int ksa_gemv_bf16(const void* a, const void* b, void* c, int M, int N, int K, long long lda, long long ldb, long long ldc,
                  void* stream);
int ksa_gemv_swiglu_bf16(const void* a, const void* b, void* c, int M, int N, int K, long long lda, long long ldb, long long ldc,
                         void* stream);
int ksa_gemv_norm_bf16(const void* x, const void* delta, const void* norm_w, void* res_out, const void* b, void* c, int M, int N,
                       int K, long long ldx, long long ld_delta, long long ld_res, long long ldb, long long ldc, float eps,
                       int delta_rows, int glu, void* stream);
int ksa_rmsnorm_fwd(const void* x, const void* delta, const void* w, void* res, void* y, void* rstd, int rows, int D, float eps,
                    int delta_rows, void* stream);
int ksa_rmsnorm_bwd(const void* dy, const void* x, const void* w, const void* rstd, const void* dres, void* dx, void* partial,
                    void* dw, int accumulate, int rows, int D, void* stream);
int ksa_qknorm_rope_fwd(const void* qkv, void* out, const void* q_w, const void* k_w, const void* pos, void* rstd,
                        long long in_stride, long long out_stride, int T, int Hq, int Hkv, int D, float theta, float eps,
                        int interleaved, int copy_v, void* stream);
int ksa_qknorm_rope_bwd(const void* qkv, const void* d_out, void* d_qkv, const void* q_w, const void* k_w, const void* pos,
                        const void* rstd, void* dqw, void* dkw, long long in_stride, long long dout_stride, int T, int Hq, int Hkv,
                        int D, float theta, float eps, int interleaved, int copy_v, void* stream);
int ksa_swiglu_fwd(const void* gu, void* out, long long rows, int F, void* stream);
int ksa_swiglu_bwd(const void* gu, const void* dout, void* dgu, long long rows, int F, void* stream);
int ksa_attn_fwd(const void* q, const void* k, const void* v, const void* ks, const void* vs, void* o, void* lse, int B, int Hq,
                 int Hkv, int HD, int Lq, int Lk, int Ns, long long q_rs, long long q_bs, long long k_rs, long long k_bs,
                 long long v_rs, long long v_bs, long long ks_rs, long long ks_bs, long long vs_rs, long long vs_bs, long long o_rs,
                 long long o_bs, int q_off, int k_off, int s_off, int chunk, int n_sum, int window, int tok_window, float scale,
                 const void* q_doc_start, const void* k_doc_end, void* stream);
int ksa_set_launch_beside(int on);
int ksa_set_dependent_launch(int mode);
int ksa_summary_attn_fwd(const void* q, const void* k, const void* v, const void* ks, const void* vs, void* o, void* lse, int B,
                         int Hq, int Hkv, int D, int Nq, int seq_len, long long q_rs, long long q_bs, long long k_rs,
                         long long k_bs, long long v_rs, long long v_bs, long long ks_rs, long long ks_bs, long long vs_rs,
                         long long vs_bs, long long o_rs, long long o_bs, int chunk, int n_sum, int chunk0, int k_off, int s_off,
                         float scale, void* stream);
int ksa_attn_bwd_fused(const void* q, const void* k, const void* v, const void* ks, const void* vs, const void* o, const void* dout,
                       const void* lse, void* stats, void* dq32, void* dq, void* dk, void* dv, void* dks, void* dvs, int B, int Hq,
                       int Hkv, int HD, int Lq, int Lk, int Ns, long long q_rs, long long q_bs, long long k_rs, long long k_bs,
                       long long v_rs, long long v_bs, long long ks_rs, long long ks_bs, long long vs_rs, long long vs_bs,
                       long long o_rs, long long o_bs, long long dq_rs, long long dq_bs, long long dk_rs, long long dk_bs,
                       long long dv_rs, long long dv_bs, long long dks_rs, long long dks_bs, long long dvs_rs, long long dvs_bs,
                       int q_off, int k_off, int s_off, int chunk, int n_sum, int window, int tok_window, float scale,
                       void* part_k, void* part_v, const void* q_doc_start, const void* k_doc_end, void* stream);
int ksa_summary_attn_bwd(const void* q, const void* k, const void* v, const void* ks, const void* vs, const void* o,
                         const void* dout, const void* lse, void* dq, void* dk, void* dv, void* dks, void* dvs, int B, int Hq,
                         int Hkv, int D, int Nq, int seq_len, long long q_rs, long long q_bs, long long k_rs, long long k_bs,
                         long long v_rs, long long v_bs, long long ks_rs, long long ks_bs, long long vs_rs, long long vs_bs,
                         long long o_rs, long long o_bs, long long dq_rs, long long dq_bs, long long dk_rs, long long dk_bs,
                         long long dv_rs, long long dv_bs, long long dks_rs, long long dks_bs, long long dvs_rs, long long dvs_bs,
                         int chunk, int n_sum, int chunk0, int k_off, int s_off, float scale, const void* part_k,
                         const void* part_v, int n_keys, void* stream);
}

namespace {

using at::Tensor;
std::atomic<long long> g_launches{0};

void check(const char* name, int rc, int kernels = 1) {
  if (rc != 0) throw std::runtime_error(std::string(name) + " failed (" + std::to_string(rc) + "): " + ksa_last_error());
  g_launches.fetch_add(kernels, std::memory_order_relaxed);
}
#define LAUNCH(entry, ...) check(#entry, entry(__VA_ARGS__))

// The arguments of one call.  `plain` turns false at the first one that is not of the ordinary kind.
struct Args {
  PyObject* const* v;
  Py_ssize_t n, at = 0;
  bool plain = true;
  c10::DeviceIndex device = -1;      // of the first tensor; it has to be the current one

  Args(PyObject* const* v, Py_ssize_t n) : v(v), n(n) {}

  PyObject* next() {
    if (at >= n) { plain = false; return Py_None; }
    return v[at++];
  }
  bool dense(const Tensor& t) {
    static const uint64_t allowed = (c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
                                     c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) |
                                     c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA)).raw_repr();
    if (!t.defined() || (t.key_set().raw_repr() & ~allowed) != 0 || !t.device().is_cuda() || !t.has_storage()) return false;
    if (device < 0) {
      device = c10::cuda::current_device();
      if (device < 0) return false;
    }
    return t.device().index() == device && t.numel() > 0 && t.const_data_ptr() != nullptr;
  }
  // a tensor of the given type; `optional`: None gives nullptr
  const Tensor* tensor(at::ScalarType type = at::kBFloat16, bool optional = false) {
    PyObject* o = next();
    if (optional && o == Py_None) return nullptr;
    if (!THPVariable_CheckExact(o)) { plain = false; return nullptr; }
    const Tensor& t = THPVariable_Unpack(o);
    if (!dense(t) || t.scalar_type() != type) { plain = false; return nullptr; }
    return &t;
  }
  long long integer() {
    PyObject* o = next();
    if (!PyLong_Check(o)) { plain = false; return 0; }       // bool is one too
    const long long x = PyLong_AsLongLong(o);
    if (x == -1 && PyErr_Occurred()) { PyErr_Clear(); plain = false; }
    if (x > INT_MAX || x < INT_MIN) plain = false;           // the entry points take sizes as int
    return x;
  }
  float real() {
    PyObject* o = next();
    const double x = PyFloat_Check(o) || PyLong_Check(o) ? PyFloat_AsDouble(o) : (plain = false, 0.0);
    if (PyErr_Occurred()) { PyErr_Clear(); plain = false; }
    return (float)x;
  }
  bool ok() { return plain && at == n; }
  void* stream() const { return c10::cuda::getCurrentCUDAStream(device).stream(); }
  Tensor empty(at::IntArrayRef sizes, at::ScalarType type = at::kBFloat16) const {
    return at::empty(sizes, at::TensorOptions().dtype(type).device(c10::Device(c10::kCUDA, device)));
  }
};

bool rows2d(const Tensor* t) { return t->dim() == 2 && t->stride(1) == 1 && t->stride(0) > 0; }      // rows with any pitch
bool packed2d(const Tensor* t) { return t->dim() == 2 && t->is_contiguous(); }
bool vector(const Tensor* t, long long n) { return t->dim() == 1 && t->size(0) == n && t->is_contiguous(); }
bool fits(long long x) { return x > 0 && x <= INT_MAX; }
const char* at_row(const Tensor& t, long long row) {
  return static_cast<const char*>(t.const_data_ptr()) + row * t.stride(0) * (long long)t.element_size();
}
char* at_row_mut(const Tensor& t, long long row) {
  return static_cast<char*>(t.mutable_data_ptr()) + row * t.stride(0) * (long long)t.element_size();
}
PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* wrap(const Tensor& a, const Tensor& b) { return Py_BuildValue("(NN)", wrap(a), wrap(b)); }
PyObject* none() { Py_RETURN_NONE; }

// While it lives, launches may run beside the kernel before them: csrc/host.h (launch_beside) says when that is sound.
struct Beside {
  explicit Beside(bool on) : before(ksa_set_launch_beside(on)) {}
  ~Beside() { ksa_set_launch_beside(before); }
  Beside(const Beside&) = delete;
  int before;
};

// While it lives, products of a thread that launches dependently read their weights early.
struct EarlyWeights {
  explicit EarlyWeights(bool on) : before(on ? ksa_set_dependent_launch(1) : 0), set(on) {
    if (set && before != 0) ksa_set_dependent_launch(before);       // ordinary launches stay ordinary
  }
  ~EarlyWeights() { if (set) ksa_set_dependent_launch(before); }
  EarlyWeights(const EarlyWeights&) = delete;
  int before;
  bool set;
};

// The kernel for C[M, N] = op(A) op(B) (+ C): the rules of `gemm` in ops/__init__.py, which explains them.
struct Product {
  const void* a;
  const void* b;
  void* c;
  long long M, N, K, lda, ldb, ldc;
  int a_mn, b_mn, fp32, accumulate;
};
void gemm(const Product& p, int pair_min, void* st) {
  const int M = (int)p.M, N = (int)p.N, K = (int)p.K;
  const bool bf16_out = !p.fp32 && !p.accumulate;
  if (M <= 16 && !p.a_mn && !p.b_mn && bf16_out && K % 8 == 0) {
    LAUNCH(ksa_gemv_bf16, p.a, p.b, p.c, M, N, K, p.lda, p.ldb, p.ldc, st);
    return;
  }
  if (!p.a_mn && !p.b_mn && bf16_out && (reinterpret_cast<uintptr_t>(p.c) & 15) == 0 && p.ldc % 8 == 0) {
    const int plan = ksa_gemm_tall_plan(M, N, K, 0, p.lda % 64 != 0 || p.ldb % 64 != 0);
    if (plan != 0) {
      LAUNCH(ksa_gemm_tall_bf16, p.a, p.b, p.c, M, N, K, p.lda, p.ldb, p.ldc, 0, plan / 16, plan % 16, st);
      return;
    }
  }
  if (!p.a_mn && bf16_out) {
    const int plan = ksa_gemm_narrow_plan(M, N, K, 0, pair_min, (p.lda % 64 != 0) + 2 * (p.ldb % 64 != 0));
    if (plan != 0) {
      LAUNCH(ksa_gemm_narrow_bf16, p.a, p.b, p.c, M, N, K, p.lda, p.ldb, p.ldc, p.b_mn, 0, plan / 16, plan % 16, 1.f, st);
      return;
    }
  }
  if (ksa_gemm_on_pairs(M, N, pair_min))
    LAUNCH(ksa_gemm2_bf16, p.a, p.b, p.c, M, N, K, p.lda, p.ldb, p.ldc, p.a_mn, p.b_mn, p.fp32, p.accumulate, 1.f, st);
  else
    LAUNCH(ksa_gemm_bf16, p.a, p.b, p.c, M, N, K, p.lda, p.ldb, p.ldc, p.a_mn, p.b_mn, p.fp32, p.accumulate, 1.f, 0, st);
}
bool sizes_ok(const Product& p) { return fits(p.M) && fits(p.N) && fits(p.K); }

// gemm(a, b, out | None, fp32 output, a_mn, b_mn, accumulate, pair_min) -> out
PyObject* py_gemm(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *x = a.tensor(), *w = a.tensor();
  PyObject* o = a.next();
  const bool fp32 = a.integer() != 0;
  const Tensor* out = nullptr;
  if (o != Py_None) {
    if (!THPVariable_CheckExact(o)) return none();
    out = &THPVariable_Unpack(o);
    if (!a.dense(*out) || out->scalar_type() != (fp32 ? at::kFloat : at::kBFloat16)) return none();
  }
  const int a_mn = a.integer() != 0, b_mn = a.integer() != 0, acc = a.integer() != 0, pair_min = (int)a.integer();
  if (!a.ok() || !rows2d(x) || !rows2d(w) || (acc && !out)) return none();
  Product p{x->const_data_ptr(), w->const_data_ptr(), nullptr, x->size(a_mn), w->size(b_mn), x->size(!a_mn), x->stride(0),
            w->stride(0), 0, a_mn, b_mn, fp32, acc};
  if (p.K != w->size(!b_mn) || !sizes_ok(p)) return none();
  if (out && !(rows2d(out) && out->size(0) == p.M && out->size(1) == p.N)) return none();
  Tensor made;
  {
    pybind11::gil_scoped_release no_gil;
    if (!out) made = a.empty({p.M, p.N}, fp32 ? at::kFloat : at::kBFloat16);
    const Tensor& c = out ? *out : made;
    p.c = c.mutable_data_ptr();
    p.ldc = c.stride(0);
    gemm(p, pair_min, a.stream());
  }
  if (out) { Py_INCREF(o); return o; }
  return wrap(made);
  END_HANDLE_TH_ERRORS
}

// linear(x, w, pair_min, weights_ready) -> y [..., N], for any x with contiguous rows.  weights_ready: no kernel that may still run when
// the one before this product has begun its work writes w (csrc/host.h, kLaunchEarlyWeights)
PyObject* py_linear(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *x = a.tensor(), *w = a.tensor();
  const int pair_min = (int)a.integer();
  const bool ready = a.integer() != 0;
  if (!a.ok() || !rows2d(w) || !(rows2d(x) || (x->dim() > 0 && x->is_contiguous())) || x->size(-1) != w->size(1)) return none();
  if (c10::GradMode::is_enabled() && (x->requires_grad() || w->requires_grad())) return none();
  const long long K = w->size(1), M = x->numel() / K;
  Product p{x->const_data_ptr(), w->const_data_ptr(), nullptr, M, w->size(0), K, x->dim() == 2 ? x->stride(0) : K, w->stride(0),
            w->size(0), 0, 0, 0, 0};
  if (!sizes_ok(p)) return none();
  Tensor y;
  {
    pybind11::gil_scoped_release no_gil;
    auto sizes = x->sizes().vec();
    sizes.back() = p.N;
    y = a.empty(sizes);
    p.c = y.mutable_data_ptr();
    const EarlyWeights early(ready);
    gemm(p, pair_min, a.stream());
  }
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

// linear_dw(dy, x, lo, hi, out | None, accumulate, pair_min, beside) -> dy[lo:hi]^T x[lo:hi], into an fp32 buffer or as bf16.
// beside: the caller launched another product of the same tensors just before (csrc/host.h, launch_beside)
PyObject* py_linear_dw(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *dy = a.tensor(), *x = a.tensor();
  const long long lo = a.integer(), hi = a.integer();
  const Tensor* out = a.tensor(at::kFloat, true);
  const int acc = a.integer() != 0, pair_min = (int)a.integer();
  const bool on = a.integer() != 0;
  if (!a.ok() || !rows2d(dy) || !rows2d(x) || dy->size(0) != x->size(0) || lo < 0 || hi <= lo || hi > x->size(0)) return none();
  Product p{at_row(*dy, lo), at_row(*x, lo), nullptr, dy->size(1), x->size(1), hi - lo, dy->stride(0), x->stride(0), 0, 1, 1,
            out != nullptr, out != nullptr && acc};
  if (!sizes_ok(p) || (out && !(rows2d(out) && out->size(0) == p.M && out->size(1) == p.N))) return none();
  Tensor made;
  {
    pybind11::gil_scoped_release no_gil;
    if (!out) made = a.empty({p.M, p.N});
    const Tensor& c = out ? *out : made;
    p.c = c.mutable_data_ptr();
    p.ldc = c.stride(0);
    const Beside beside(on && out);      // memory allocated here might be what the kernel before has just let go
    gemm(p, pair_min, a.stream());
  }
  return wrap(out ? *out : made);
  END_HANDLE_TH_ERRORS
}

// dual_linear(x, w_a, w_b, n_a, b_mn, pair_min): rows [:n_a] of x times w_a, the others times w_b.  b_mn: the weights as they lie,
// [K, N] (the gradient of x from that of y)
PyObject* py_dual_linear(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *x = a.tensor(), *wa = a.tensor(), *wb = a.tensor();
  const long long n_a = a.integer();
  const int b_mn = a.integer() != 0, pair_min = (int)a.integer();
  if (!a.ok() || !packed2d(x) || !rows2d(wa) || !rows2d(wb) || wa->sizes() != wb->sizes() || n_a < 0 || n_a > x->size(0)) return none();
  const long long R = x->size(0), N = wa->size(b_mn), K = wa->size(!b_mn);
  if (K != x->size(1) || !fits(R) || !fits(N) || !fits(K)) return none();
  Tensor y;
  {
    pybind11::gil_scoped_release no_gil;
    y = a.empty({R, N});
    void* st = a.stream();
    if (n_a > 0)
      gemm({x->const_data_ptr(), wa->const_data_ptr(), y.mutable_data_ptr(), n_a, N, K, K, wa->stride(0), N, 0, b_mn, 0, 0}, pair_min, st);
    const Beside beside(n_a > 16);     // at most 16 text rows take a product that lets its successors start before it waits
    if (R > n_a)
      gemm({at_row(*x, n_a), wb->const_data_ptr(), at_row_mut(y, n_a), R - n_a, N, K, K, wb->stride(0), N, 0, b_mn, 0, 0}, pair_min, st);
  }
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

// rms_norm(x, delta | None, w, eps) -> (x + delta, norm, 1 / rms), or (norm, 1 / rms) without delta
PyObject* py_rms_norm(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *x = a.tensor(), *d = a.tensor(at::kBFloat16, true), *w = a.tensor();
  const float eps = a.real();
  if (!a.ok() || !packed2d(x) || !vector(w, x->size(1)) || !fits(x->size(0)) || !fits(x->size(1))) return none();
  if (d && !(packed2d(d) && d->size(1) == x->size(1) && d->size(0) <= x->size(0))) return none();
  const int rows = (int)x->size(0), D = (int)x->size(1);
  Tensor res, y, rstd;
  {
    pybind11::gil_scoped_release no_gil;
    y = a.empty({rows, D});
    if (d) res = a.empty({rows, D});
    rstd = a.empty({rows}, at::kFloat);
    LAUNCH(ksa_rmsnorm_fwd, x->const_data_ptr(), d ? d->const_data_ptr() : nullptr, w->const_data_ptr(),
           d ? res.mutable_data_ptr() : nullptr, y.mutable_data_ptr(), rstd.mutable_data_ptr(), rows, D, eps, d ? (int)d->size(0) : 0,
           a.stream());
  }
  if (!d) return wrap(y, rstd);
  return Py_BuildValue("(NNN)", wrap(res), wrap(y), wrap(rstd));
  END_HANDLE_TH_ERRORS
}

// rms_norm_bwd(dy, x, w, rstd, dres | None, dw (fp32), accumulate) -> dx
PyObject* py_rms_norm_bwd(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *dy = a.tensor(), *x = a.tensor(), *w = a.tensor(), *rstd = a.tensor(at::kFloat), *dres = a.tensor(at::kBFloat16, true),
               *dw = a.tensor(at::kFloat);
  const int acc = a.integer() != 0;
  if (!a.ok() || !packed2d(x) || !packed2d(dy) || dy->sizes() != x->sizes() || (dres && !(packed2d(dres) && dres->sizes() == x->sizes())))
    return none();
  if (!fits(x->size(0)) || !fits(x->size(1)) || !vector(w, x->size(1)) || !vector(dw, x->size(1)) || !vector(rstd, x->size(0))) return none();
  const int rows = (int)x->size(0), D = (int)x->size(1);
  Tensor dx;
  {
    pybind11::gil_scoped_release no_gil;
    dx = a.empty({rows, D});
    Tensor partial = a.empty({ksa_rmsnorm_bwd_parts(rows), D}, at::kFloat);
    check("ksa_rmsnorm_bwd",
          ksa_rmsnorm_bwd(dy->const_data_ptr(), x->const_data_ptr(), w->const_data_ptr(), rstd->const_data_ptr(),
                          dres ? dres->const_data_ptr() : nullptr, dx.mutable_data_ptr(), partial.mutable_data_ptr(),
                          dw->mutable_data_ptr(), acc, rows, D, a.stream()), 2);
  }
  return wrap(dx);
  END_HANDLE_TH_ERRORS
}

// qk_norm_rope(qkv, q_w | None, k_w | None, pos (int32), Hq, Hkv, D, theta, eps, interleaved) -> (out, rstd)
PyObject* py_qk_norm_rope(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *qkv = a.tensor(), *qw = a.tensor(at::kBFloat16, true), *kw = a.tensor(at::kBFloat16, true), *pos = a.tensor(at::kInt);
  const long long Hq = a.integer(), Hkv = a.integer(), D = a.integer();
  const float theta = a.real(), eps = a.real();
  const int inter = a.integer() != 0;
  if (!a.ok() || Hq <= 0 || Hkv <= 0 || D <= 0 || !rows2d(qkv) || qkv->size(1) != (Hq + 2 * Hkv) * D || !fits(qkv->size(0)) ||
      !vector(pos, qkv->size(0)) || (qw && !vector(qw, D)) || (kw && !vector(kw, D)))
    return none();
  const int T = (int)qkv->size(0);
  Tensor out, rstd;
  {
    pybind11::gil_scoped_release no_gil;
    out = a.empty({T, qkv->size(1)});
    rstd = a.empty({T, Hq + Hkv}, at::kFloat);
    LAUNCH(ksa_qknorm_rope_fwd, qkv->const_data_ptr(), out.mutable_data_ptr(), qw ? qw->const_data_ptr() : nullptr,
           kw ? kw->const_data_ptr() : nullptr, pos->const_data_ptr(), rstd.mutable_data_ptr(), qkv->stride(0), out.stride(0), T, (int)Hq,
           (int)Hkv, (int)D, theta, eps, inter, 1, a.stream());
  }
  return wrap(out, rstd);
  END_HANDLE_TH_ERRORS
}

// qk_norm_rope_bwd(qkv, d_out, q_w | None, k_w | None, pos, rstd, dq_w (fp32) | None, dk_w | None, Hq, Hkv, D, theta, eps, interleaved)
// -> d_qkv; the weight gradients are added to dq_w and dk_w
PyObject* py_qk_norm_rope_bwd(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *qkv = a.tensor(), *g = a.tensor(), *qw = a.tensor(at::kBFloat16, true), *kw = a.tensor(at::kBFloat16, true),
               *pos = a.tensor(at::kInt), *rstd = a.tensor(at::kFloat), *dqw = a.tensor(at::kFloat, true), *dkw = a.tensor(at::kFloat, true);
  const long long Hq = a.integer(), Hkv = a.integer(), D = a.integer();
  const float theta = a.real(), eps = a.real();
  const int inter = a.integer() != 0;
  if (!a.ok() || Hq <= 0 || Hkv <= 0 || D <= 0 || !packed2d(qkv) || qkv->size(1) != (Hq + 2 * Hkv) * D || !fits(qkv->size(0)) ||
      !packed2d(g) || g->sizes() != qkv->sizes() || !vector(pos, qkv->size(0)) || !packed2d(rstd) || rstd->size(0) != qkv->size(0) ||
      rstd->size(1) != Hq + Hkv || (qw && !vector(qw, D)) || (kw && !vector(kw, D)) || (dqw && !vector(dqw, D)) || (dkw && !vector(dkw, D)))
    return none();
  const int T = (int)qkv->size(0);
  Tensor d;
  {
    pybind11::gil_scoped_release no_gil;
    d = a.empty(qkv->sizes());
    LAUNCH(ksa_qknorm_rope_bwd, qkv->const_data_ptr(), g->const_data_ptr(), d.mutable_data_ptr(), qw ? qw->const_data_ptr() : nullptr,
           kw ? kw->const_data_ptr() : nullptr, pos->const_data_ptr(), rstd->const_data_ptr(), dqw ? dqw->mutable_data_ptr() : nullptr,
           dkw ? dkw->mutable_data_ptr() : nullptr, qkv->stride(0), g->stride(0), T, (int)Hq, (int)Hkv, (int)D, theta, eps, inter, 1,
           a.stream());
  }
  return wrap(d);
  END_HANDLE_TH_ERRORS
}

// swiglu(gate | up rows) -> rows of half the width
PyObject* py_swiglu(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor* gu = a.tensor();
  if (!a.ok() || gu->dim() < 1 || !gu->is_contiguous() || gu->size(-1) % 2 != 0 || !fits(gu->size(-1))) return none();
  const long long F = gu->size(-1) / 2, rows = gu->numel() / (2 * F);
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    auto sizes = gu->sizes().vec();
    sizes.back() = F;
    out = a.empty(sizes);
    LAUNCH(ksa_swiglu_fwd, gu->const_data_ptr(), out.mutable_data_ptr(), rows, (int)F, a.stream());
  }
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// swiglu_bwd(gate | up rows, dout rows) -> d(gate | up)
PyObject* py_swiglu_bwd(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *gu = a.tensor(), *g = a.tensor();
  if (!a.ok() || !packed2d(gu) || !packed2d(g) || gu->size(0) != g->size(0) || gu->size(1) != 2 * g->size(1) || !fits(gu->size(1))) return none();
  Tensor d;
  {
    pybind11::gil_scoped_release no_gil;
    d = a.empty(gu->sizes());
    LAUNCH(ksa_swiglu_bwd, gu->const_data_ptr(), g->const_data_ptr(), d.mutable_data_ptr(), gu->size(0), (int)g->size(1), a.stream());
  }
  return wrap(d);
  END_HANDLE_TH_ERRORS
}

// linear_swiglu(x, w13, pair_min) -> silu(gate) * up where one kernel does it (no gradients wanted), else None
PyObject* py_linear_swiglu(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *x = a.tensor(), *w = a.tensor();
  const int pair_min = (int)a.integer();
  if (!a.ok() || !rows2d(x) || !rows2d(w) || x->size(1) != w->size(1) || w->size(0) % 2 != 0 || !fits(x->size(0)) || !fits(w->size(0)) ||
      !fits(x->size(1)) || x->size(1) % 8 != 0 || x->stride(0) % 8 != 0 || w->stride(0) % 8 != 0)
    return none();
  if (c10::GradMode::is_enabled() && (x->requires_grad() || w->requires_grad())) return none();
  const int M = (int)x->size(0), N = (int)w->size(0), K = (int)x->size(1);
  int plan = 0, tall = 0;
  if (M > 16) {
    tall = ksa_gemm_tall_plan(M, N / 2, K, 1, x->stride(0) % 64 != 0 || w->stride(0) % 64 != 0);
    if (tall == 0 && N % 16 == 0) plan = ksa_gemm_narrow_plan(M, N, K, 1, pair_min, (x->stride(0) % 64 != 0) + 2 * (w->stride(0) % 64 != 0));
    if (plan == 0 && tall == 0) return none();
  }
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = a.empty({M, N / 2});
    if (M <= 16)
      LAUNCH(ksa_gemv_swiglu_bf16, x->const_data_ptr(), w->const_data_ptr(), out.mutable_data_ptr(), M, N, K, x->stride(0), w->stride(0),
             out.stride(0), a.stream());
    else if (tall != 0)
      LAUNCH(ksa_gemm_tall_bf16, x->const_data_ptr(), w->const_data_ptr(), out.mutable_data_ptr(), M, N / 2, K, x->stride(0), w->stride(0),
             out.stride(0), 1, tall / 16, 1, a.stream());
    else
      LAUNCH(ksa_gemm_narrow_bf16, x->const_data_ptr(), w->const_data_ptr(), out.mutable_data_ptr(), M, N, K, x->stride(0), w->stride(0),
             out.stride(0), 0, 1, plan / 16, plan % 16, 1.f, a.stream());
  }
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// gemm_swiglu(x, w13, pair_min) -> (silu(gate) * up, gate | up) from one launch of the CTA-pair kernel where that serves the
// product, else None (333 x 19456 x 2560 45.7 us on pairs; on single CTAs with the activation behind 44.4)
PyObject* py_gemm_swiglu(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *x = a.tensor(), *w = a.tensor();
  const int pair_min = (int)a.integer();
  if (!a.ok() || !rows2d(x) || !rows2d(w) || x->size(1) != w->size(1) || w->size(0) % 128 != 0 || !fits(x->size(0)) || !fits(w->size(0)) ||
      !fits(x->size(1)) || x->stride(0) % 8 != 0 || w->stride(0) % 8 != 0 || x->size(0) <= 16)
    return none();
  const int M = (int)x->size(0), F = (int)(w->size(0) / 2), K = (int)x->size(1);
  if (!ksa_gemm_on_pairs(M, 2 * F, pair_min) ||
      ksa_gemm_narrow_plan(M, 2 * F, K, 2, pair_min, (x->stride(0) % 64 != 0) + 2 * (w->stride(0) % 64 != 0)) != 0)
    return none();
  Tensor h, gu;
  {
    pybind11::gil_scoped_release no_gil;
    h = a.empty({M, F});
    gu = a.empty({M, 2LL * F});
    LAUNCH(ksa_gemm2_swiglu_bf16, x->const_data_ptr(), w->const_data_ptr(), gu.mutable_data_ptr(), h.mutable_data_ptr(), M, F, K, x->stride(0),
           w->stride(0), 2LL * F, F, a.stream());
  }
  return wrap(h, gu);
  END_HANDLE_TH_ERRORS
}

// norm_linear(x, delta | None, norm_w, eps, w, glu) -> (x + delta, product of the normalised rows), at most four rows, no gradients
PyObject* py_norm_linear(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  PyObject* px = n > 0 ? v[0] : Py_None;
  const Tensor *x = a.tensor(), *d = a.tensor(at::kBFloat16, true), *nw = a.tensor();
  const float eps = a.real();
  const Tensor* w = a.tensor();
  const int glu = a.integer() != 0;
  if (!a.ok() || !rows2d(x) || !rows2d(w) || x->size(0) > 4 || x->numel() > 81920 || x->size(1) != w->size(1) || !vector(nw, x->size(1)) || !fits(w->size(0)) ||
      !fits(x->size(1)) || x->size(1) % 8 != 0 || x->stride(0) % 8 != 0 || w->stride(0) % 8 != 0 || (glu && w->size(0) % 2 != 0))
    return none();
  if (d && !(rows2d(d) && d->size(1) == x->size(1) && d->size(0) <= x->size(0) && d->stride(0) % 8 == 0)) return none();
  if (c10::GradMode::is_enabled() && (x->requires_grad() || w->requires_grad())) return none();
  const int M = (int)x->size(0), K = (int)x->size(1), N = (int)w->size(0);
  Tensor res, out;
  {
    pybind11::gil_scoped_release no_gil;
    if (d) res = a.empty({M, K});
    out = a.empty({M, glu ? N / 2 : N});
    LAUNCH(ksa_gemv_norm_bf16, x->const_data_ptr(), d ? d->const_data_ptr() : nullptr, nw->const_data_ptr(),
           d ? res.mutable_data_ptr() : nullptr, w->const_data_ptr(), out.mutable_data_ptr(), M, N, K, x->stride(0), d ? d->stride(0) : K,
           d ? res.stride(0) : x->stride(0), w->stride(0), out.stride(0), eps, d ? (int)d->size(0) : 0, glu, a.stream());
  }
  if (d) return wrap(res, out);
  Py_INCREF(px);
  return Py_BuildValue("(NN)", px, wrap(out));
  END_HANDLE_TH_ERRORS
}

// Column blocks of packed rows [B*L text rows | B*Ns summary rows], each q heads | k heads | v heads.
struct PackedShape {
  long long B, L, Ns, Hq, Hkv, D, chunk, n_sum, window, tok_window;
  float scale;
  void read(Args& a) {
    B = a.integer(); L = a.integer(); Ns = a.integer(); Hq = a.integer(); Hkv = a.integer(); D = a.integer(); chunk = a.integer();
    n_sum = a.integer(); window = a.integer(); tok_window = a.integer(); scale = a.real();
  }
  bool ok(const Tensor* qkv) const {
    return B > 0 && L > 0 && Ns >= 0 && Hq > 0 && Hkv > 0 && D > 0 && chunk > 0 && rows2d(qkv) && qkv->size(0) == B * (L + Ns) &&
           qkv->size(1) == (Hq + 2 * Hkv) * D;
  }
  long long q_cols() const { return Hq * D; }
  const void* block(const Tensor& t, long long row, long long col) const {
    return static_cast<const char*>(t.const_data_ptr()) + (row * t.stride(0) + col) * 2;
  }
  void* block_mut(Tensor& t, long long row, long long col) const {
    return static_cast<char*>(t.mutable_data_ptr()) + (row * t.stride(0) + col) * 2;
  }
};

// attention(qkv, B, L, Ns, Hq, Hkv, D, chunk, n_sum, window, tok_window, scale) -> (out, lse, summary lse | None)
PyObject* py_attention(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor* x = a.tensor();
  PackedShape s;
  s.read(a);
  if (!a.ok() || !s.ok(x)) return none();
  const int B = (int)s.B, L = (int)s.L, Ns = (int)s.Ns, Hq = (int)s.Hq, Hkv = (int)s.Hkv, D = (int)s.D;
  const long long rs = x->stride(0), text = s.B * s.L, kc = s.q_cols(), vc = kc + s.Hkv * s.D, os = s.q_cols();
  Tensor out, lse, lse_s;
  {
    pybind11::gil_scoped_release no_gil;
    out = a.empty({x->size(0), os});
    lse = a.empty({B, Hq, L}, at::kFloat);
    if (Ns) lse_s = a.empty({B, Hq, Ns}, at::kFloat);      // ahead of the launches: no memory of a kernel that may still run
    const void *k = s.block(*x, 0, kc), *vv = s.block(*x, 0, vc);
    const void *ks = Ns ? s.block(*x, text, kc) : nullptr, *vs = Ns ? s.block(*x, text, vc) : nullptr;
    LAUNCH(ksa_attn_fwd, x->const_data_ptr(), k, vv, ks, vs, out.mutable_data_ptr(), lse.mutable_data_ptr(), B, Hq, Hkv, D, L, L, Ns, rs,
           L * rs, rs, L * rs, rs, L * rs, rs, Ns * rs, rs, Ns * rs, os, L * os, 0, 0, 0, (int)s.chunk, s.n_sum > 1 ? (int)s.n_sum : 1,
           (int)s.window, (int)s.tok_window, s.scale, nullptr, nullptr, a.stream());
    if (Ns) {
      const Beside beside(true);
      LAUNCH(ksa_summary_attn_fwd, s.block(*x, text, 0), k, vv, ks, vs, s.block_mut(out, text, 0), lse_s.mutable_data_ptr(), B, Hq, Hkv,
             D, Ns, L, rs, Ns * rs, rs, L * rs, rs, L * rs, rs, Ns * rs, rs, Ns * rs, os, Ns * os, (int)s.chunk, (int)s.n_sum, 0, 0, 0,
             s.scale, a.stream());
    }
  }
  return Py_BuildValue("(NNN)", wrap(out), wrap(lse), Ns ? wrap(lse_s) : none());
  END_HANDLE_TH_ERRORS
}

// attention_bwd(qkv, out, lse, summary lse | None, dout, B, .., scale) -> dqkv, by the fused kernel (head dim 128)
PyObject* py_attention_bwd(PyObject*, PyObject* const* v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a(v, n);
  const Tensor *x = a.tensor(), *o = a.tensor(), *lse = a.tensor(at::kFloat), *lse_s = a.tensor(at::kFloat, true), *g = a.tensor();
  PackedShape s;
  s.read(a);
  if (!a.ok() || !s.ok(x) || s.D != 128 || !packed2d(o) || !packed2d(g) || o->size(0) != x->size(0) || o->size(1) != s.q_cols() ||
      g->sizes() != o->sizes() || !lse->is_contiguous() || lse->numel() != s.B * s.Hq * s.L || (s.Ns > 0) != (lse_s != nullptr))
    return none();
  if (lse_s && !(lse_s->is_contiguous() && lse_s->numel() == s.B * s.Hq * s.Ns)) return none();
  if (reinterpret_cast<uintptr_t>(o->const_data_ptr()) % 16 != 0) return none();      // a saved-tensor hook gives any address
  const int B = (int)s.B, L = (int)s.L, Ns = (int)s.Ns, Hq = (int)s.Hq, Hkv = (int)s.Hkv, D = (int)s.D;
  const long long rs = x->stride(0), text = s.B * s.L, kc = s.q_cols(), vc = kc + s.Hkv * s.D, os = s.q_cols();
  Tensor d;
  {
    pybind11::gil_scoped_release no_gil;
    d = a.empty(x->sizes());
    const long long ds = d.stride(0);
    Tensor stats = a.empty({2, B, Hq, (L + 127) / 128 * 128}, at::kFloat), dq32 = a.empty({B, L, Hq, D}, at::kFloat), part_k, part_v;
    if (Ns && ksa_attn_bwd_num_segments(L) > 1) {
      part_k = a.empty({B, Ns, Hkv, D}, at::kFloat).zero_();
      part_v = a.empty({B, Ns, Hkv, D}, at::kFloat).zero_();
    }
    void *pk = part_k.defined() ? part_k.mutable_data_ptr() : nullptr, *pv = part_v.defined() ? part_v.mutable_data_ptr() : nullptr;
    const void *k = s.block(*x, 0, kc), *vv = s.block(*x, 0, vc);
    const void *ks = Ns ? s.block(*x, text, kc) : nullptr, *vs = Ns ? s.block(*x, text, vc) : nullptr;
    void *dk = s.block_mut(d, 0, kc), *dv = s.block_mut(d, 0, vc);
    void *dks = Ns ? s.block_mut(d, text, kc) : nullptr, *dvs = Ns ? s.block_mut(d, text, vc) : nullptr;
    check("ksa_attn_bwd_fused",
          ksa_attn_bwd_fused(x->const_data_ptr(), k, vv, ks, vs, o->const_data_ptr(), g->const_data_ptr(), lse->const_data_ptr(),
                             stats.mutable_data_ptr(), dq32.mutable_data_ptr(), d.mutable_data_ptr(), dk, dv, dks, dvs, B, Hq, Hkv, D, L,
                             L, Ns, rs, L * rs, rs, L * rs, rs, L * rs, rs, Ns * rs, rs, Ns * rs, os, L * os, ds, L * ds, ds, L * ds, ds,
                             L * ds, ds, Ns * ds, ds, Ns * ds, 0, 0, 0, (int)s.chunk, s.n_sum > 1 ? (int)s.n_sum : 1, (int)s.window,
                             (int)s.tok_window, s.scale, pk, pv, nullptr, nullptr, a.stream()), 3);
    if (Ns)
      LAUNCH(ksa_summary_attn_bwd, s.block(*x, text, 0), k, vv, ks, vs, s.block(*o, text, 0), s.block(*g, text, 0), lse_s->const_data_ptr(),
             s.block_mut(d, text, 0), dk, dv, dks, dvs, B, Hq, Hkv, D, Ns, L, rs, Ns * rs, rs, L * rs, rs, L * rs, rs, Ns * rs, rs, Ns * rs,
             os, Ns * os, ds, Ns * ds, ds, L * ds, ds, L * ds, ds, Ns * ds, ds, Ns * ds, (int)s.chunk, (int)s.n_sum, 0, 0, 0, s.scale, pk,
             pv, Ns, a.stream());
  }
  return wrap(d);
  END_HANDLE_TH_ERRORS
}

PyObject* py_launches(PyObject*, PyObject* const*, Py_ssize_t) { return PyLong_FromLongLong(g_launches.load()); }

#define FN(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FN(gemm), FN(linear), FN(linear_dw), FN(dual_linear), FN(rms_norm), FN(rms_norm_bwd), FN(qk_norm_rope),
                           FN(qk_norm_rope_bwd), FN(swiglu), FN(swiglu_bwd), FN(linear_swiglu), FN(gemm_swiglu), FN(norm_linear), FN(attention),
                           FN(attention_bwd), FN(launches), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "ksa_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_ksa_native() { return PyModule_Create(&g_module); }
