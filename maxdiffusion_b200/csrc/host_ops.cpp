// Host side of the ops that are launched hundreds of times per model call, as a CPython extension: shape checks, output
// allocation, launch shape and the call of the C entry point, without ctypes (which converts 20 to 30 arguments per launch
// one by one). Same kernels, same results and the same current stream as the Python wrappers in `ops/kernels.py` and
// `ops/conv.py`, which take every call: a function here returns NotImplemented for every input that it does not handle
// (another layout, dtype or device), and the caller goes on with the Python wrapper, which then also raises what there is to
// raise. `linear_group` and `geglu_linear` have no wrapper of their own: without them the caller runs one product per matrix,
// and the product and GEGLU as two kernels.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>
#include <unordered_map>
#include <vector>

extern "C" {
int mdb_gemm_bf16(const void*, const void*, void*, const void*, const void*, const void*, int, int, int, long long, long long,
                  long long, long long, long long, int, int, int, int, int, float, int, int, int, void*, void*);
int mdb_gemm_geglu(const void*, const void*, void*, const void*, int, int, int, long long, long long, long long, void*);
int mdb_gemm_group(const void*, const void* const*, int, void*, int, int, int, long long, long long, long long, int, int, void*);
int mdb_flash_fwd(const void*, const void* const*, const void* const*, void*, float*, int, int, int, int, const int*, long long,
                  long long, long long, long long, long long, long long, long long, long long, long long, long long, long long,
                  long long, float, const unsigned int*, unsigned int, const void*, void*);
int mdb_flash_fwd_d64(const void*, const void* const*, const void* const*, void*, float*, int, int, int, int, const int*,
                      long long, long long, long long, long long, long long, long long, long long, long long, long long,
                      long long, long long, long long, float, const unsigned int*, unsigned int, const void*, void*);
int mdb_flash_fwd_narrow(const void*, const void* const*, const void* const*, void*, float*, int, int, int, int, const int*,
                         long long, long long, long long, long long, long long, long long, long long, long long, long long,
                         long long, long long, long long, float, int, void*);
int mdb_ln_fwd(const void*, void*, const void*, const void*, const float*, const float*, long long, int, int, int, float, float*,
               float*, int, void*);
int mdb_geglu_fwd(const void*, void*, long long, int, void*);
int mdb_rms_rope_fwd(const void*, long long, void*, long long, long long, const void*, int, const float*, const float*, int, int,
                     int, int, float, float*, int, void*);
int mdb_gn_cl_sums(const void*, const void*, const float*, const float*, float*, int, int, int, int, void*);
// Weak: over a kernel library without it the norm takes the three launches, whose entry points have kept their arguments. An entry
// point whose arguments change gets another name, so that an object of one kind never calls a library of another.
__attribute__((weak)) int mdb_gn_cl_group(const void*, void*, int, int, int, int, int, float, const void*, const void*, int, const void*, long long, int, void*);
int mdb_gn_cl_fold_fwd(const float*, int, int, int, int, float, float, const void*, const void*, int, float*, float*, float*,
                       float*, void*);
int mdb_gn_cl_apply(const void*, const void*, void*, const float*, const float*, const float*, const float*, const float*, int,
                    int, int, int, void*);
int mdb_conv_igemm(const void*, const void*, const void*, void*, const void*, const void*, const long long*, const long long*,
                   const long long*, const long long*, const int*, const int*, int, int, long long, int, const int*, const int*,
                   int, int, const long long*, const long long*, int, int, int, int, void*, int, void*);
}

// Read from the file before it is loaded (`build.host_ops_built_for`).
extern "C" __attribute__((used)) const char mdb_host_ops_built_for[] = "mdb_host_ops built for " MDB_BUILT_FOR ";";

namespace {

using at::Tensor;

long long g_launches = 0;        // these three and g_plans: under the GIL
PyObject* g_error = nullptr;     // ops._lib.KernelError
PyObject* g_plan = nullptr;      // ops.kernels.gemm_plan

constexpr int kCtasTarget = 148 * 4;
constexpr int kGnGroupElsewhere = 3705;

PyObject* not_implemented() { Py_RETURN_NOTIMPLEMENTED; }

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Other Python threads run while this object lives: around the allocations and the entry points, which may wait for the GPU
// (a full launch queue, the allocator). Nothing of Python's is touched meanwhile, nor what the lock guards above; a tensor
// that Python holds is not copied. The destructor takes the lock back, also when an exception passes.
class WithoutGil {
 public:
  WithoutGil() : state_(PyEval_SaveThread()) {}
  ~WithoutGil() { PyEval_RestoreThread(state_); }
  WithoutGil(const WithoutGil&) = delete;

 private:
  PyThreadState* state_;
};

template <typename F>
int unlocked(F&& f) {
  const WithoutGil lock;
  return f();
}

// nullptr and a Python error when the launch was refused
PyObject* done(int rc, const char* what, const Tensor& out, int launches = 1) {
  if (rc != 0) {
    PyErr_Format(g_error ? g_error : PyExc_RuntimeError, "%s failed with code %d", what, rc);
    return nullptr;
  }
  g_launches += launches;
  return THPVariable_Wrap(out);
}

// A tensor argument or None; false: neither.
bool opt_tensor(PyObject* o, const Tensor*& t) {
  t = nullptr;
  if (o == Py_None) return true;
  if (!THPVariable_Check(o)) return false;
  t = &THPVariable_Unpack(o);
  return true;
}

bool bf16(const Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kBFloat16; }
bool f32(const Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kFloat; }
const void* data(const Tensor* t) { return t ? t->data_ptr() : nullptr; }
// What the kernels' 16-byte accesses need of a row-major bf16 matrix.
bool aligned16(const Tensor& t, int64_t pitch) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0 && (pitch & 7) == 0; }

// All axes but the last as rows of one pitch. False: not that layout.
bool rows_of(const Tensor& t, int64_t& rows, int64_t& pitch) {
  const int64_t n = t.dim();
  if (n < 2 || t.stride(n - 1) != 1) return false;
  rows = 1;
  pitch = t.size(n - 1);
  bool first = true;
  for (int64_t i = n - 2; i >= 0; --i) {
    const int64_t size = t.size(i);
    if (size == 1) continue;
    if (first) pitch = t.stride(i);
    else if (t.stride(i) != pitch * rows) return false;
    first = false;
    rows *= size;
  }
  return rows > 0;
}

struct PlanKey {
  int64_t m, n, k;
  int flags;
  bool operator==(const PlanKey& o) const { return m == o.m && n == o.n && k == o.k && flags == o.flags; }
};
struct PlanHash {
  size_t operator()(const PlanKey& p) const {
    size_t h = static_cast<size_t>(p.m);
    h = h * 1000003u ^ static_cast<size_t>(p.n);
    h = h * 1000003u ^ static_cast<size_t>(p.k);
    return h * 1000003u ^ static_cast<size_t>(p.flags);
  }
};
struct Plan {
  int ctas, bn, splits;
};
std::unordered_map<PlanKey, Plan, PlanHash> g_plans;

// `ops.kernels.gemm_plan`, remembered by its arguments (a pure function of sizes).
bool gemm_plan(int64_t m, int64_t n, int64_t k, bool b_mn, bool splittable, long tile_n, long ctas, Plan& out) {
  const PlanKey key{m, n, k, static_cast<int>(b_mn) | (splittable ? 2 : 0) | (static_cast<int>(tile_n) << 4) |
                                 (static_cast<int>(ctas) << 16)};
  const auto hit = g_plans.find(key);
  if (hit != g_plans.end()) {
    out = hit->second;
    return true;
  }
  if (g_plan == nullptr) {
    PyErr_SetString(PyExc_RuntimeError, "host_ops.setup() has not been called");
    return false;
  }
  PyObject* r = PyObject_CallFunction(g_plan, "LLLOOill", static_cast<long long>(m), static_cast<long long>(n),
                                      static_cast<long long>(k), b_mn ? Py_True : Py_False, splittable ? Py_True : Py_False, 148,
                                      tile_n, ctas);
  if (r == nullptr) return false;
  const bool ok = PyArg_ParseTuple(r, "iii", &out.ctas, &out.bn, &out.splits) != 0;
  Py_DECREF(r);
  if (!ok) return false;
  if (g_plans.size() >= 4096) g_plans.clear();
  g_plans.emplace(key, out);
  return true;
}

// gemm(a, b, a_mn, b_mn, bias, epi, residual, gate, rows_per_batch, out, out_f32, alpha, split_k, tile_n, ctas)
PyObject* py_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 15 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[1])) return not_implemented();
  const Tensor &A = THPVariable_Unpack(a[0]), &B = THPVariable_Unpack(a[1]);
  const bool a_mn = a[2] == Py_True, b_mn = a[3] == Py_True, out_f32 = a[10] == Py_True;
  const Tensor *bias, *residual, *gate, *given;
  if (!opt_tensor(a[4], bias) || !opt_tensor(a[6], residual) || !opt_tensor(a[7], gate) || !opt_tensor(a[9], given))
    return not_implemented();
  const int epi = static_cast<int>(PyLong_AsLong(a[5])), rows_per_batch = static_cast<int>(PyLong_AsLong(a[8]));
  const double alpha = PyFloat_AsDouble(a[11]);
  const long split_k = PyLong_AsLong(a[12]), tile_n = PyLong_AsLong(a[13]), force_ctas = PyLong_AsLong(a[14]);
  if (PyErr_Occurred()) return nullptr;
  if (!bf16(A) || !bf16(B) || A.dim() != 2 || B.dim() != 2 || A.stride(1) != 1 || B.stride(1) != 1) return not_implemented();
  const int64_t K = a_mn ? A.size(0) : A.size(1), M = a_mn ? A.size(1) : A.size(0);
  const int64_t Kb = b_mn ? B.size(0) : B.size(1), N = b_mn ? B.size(1) : B.size(0);
  if (K != Kb || M <= 0 || N <= 0 || K <= 0 || M > INT_MAX || N > INT_MAX || K > INT_MAX) return not_implemented();
  if (bias && (!bf16(*bias) || !bias->is_contiguous())) return not_implemented();
  if (residual && (!bf16(*residual) || residual->dim() != 2 || residual->stride(1) != 1 || !aligned16(*residual, residual->stride(0))))
    return not_implemented();
  if (gate && (!f32(*gate) || gate->stride(-1) != 1)) return not_implemented();
  if (given && (!given->is_cuda() || given->dim() != 2 || given->size(0) != M || given->size(1) != N || given->stride(1) != 1))
    return not_implemented();
  const bool f32_out = given ? given->scalar_type() == at::kFloat : out_f32;
  if (given && !f32_out && given->scalar_type() != at::kBFloat16) return not_implemented();
  Plan plan;
  if (!gemm_plan(M, N, K, b_mn, split_k == 0, tile_n, force_ctas, plan)) return nullptr;
  if (split_k > 0) plan.splits = (!bias && epi == 0 && !residual && !gate) ? static_cast<int>(split_k) : 1;
  Tensor out;
  if (given) out = *given;
  const int rc = unlocked([&] {
    if (!given) out = at::empty({M, N}, A.options().dtype(f32_out ? at::kFloat : at::kBFloat16));
    Tensor partial;
    if (plan.splits > 1) partial = at::empty({plan.splits, M, N}, A.options().dtype(at::kFloat));
    return mdb_gemm_bf16(A.data_ptr(), B.data_ptr(), out.data_ptr(), data(bias), data(residual), data(gate), static_cast<int>(M),
                         static_cast<int>(N), static_cast<int>(K), A.stride(0), B.stride(0), out.stride(0),
                         residual ? residual->stride(0) : 0, gate && gate->dim() == 2 ? gate->stride(0) : 0, rows_per_batch, a_mn,
                         b_mn, epi, f32_out, static_cast<float>(alpha), plan.ctas, plan.bn, plan.splits,
                         plan.splits > 1 ? partial.data_ptr() : nullptr, stream());
  });
  return done(rc, "mdb_gemm_bf16", out);
  END_HANDLE_TH_ERRORS
}

// linear(x, weight, bias, epi, residual, tile_n, ctas): [..., K] x [N, K]^T -> [..., N]
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[1])) return not_implemented();
  const Tensor &x = THPVariable_Unpack(a[0]), &w = THPVariable_Unpack(a[1]);
  const Tensor *bias, *residual;
  if (!opt_tensor(a[2], bias) || !opt_tensor(a[4], residual)) return not_implemented();
  const int epi = static_cast<int>(PyLong_AsLong(a[3]));
  const long tile_n = PyLong_AsLong(a[5]), force_ctas = PyLong_AsLong(a[6]);
  if (PyErr_Occurred()) return nullptr;
  int64_t M, lda, Mr = 0, ldr = 0;
  if (!bf16(x) || !bf16(w) || w.dim() != 2 || w.stride(1) != 1 || !rows_of(x, M, lda)) return not_implemented();
  const int64_t K = x.size(-1), N = w.size(0);
  if (w.size(1) != K || N <= 0 || K <= 0 || M > INT_MAX || N > INT_MAX || K > INT_MAX) return not_implemented();
  if (bias && (!bf16(*bias) || !bias->is_contiguous() || bias->numel() != N)) return not_implemented();
  if (residual && (!bf16(*residual) || !rows_of(*residual, Mr, ldr) || Mr != M || residual->size(-1) != N || !aligned16(*residual, ldr)))
    return not_implemented();
  std::vector<int64_t> sizes(x.sizes().begin(), x.sizes().end());
  sizes.back() = N;
  Plan plan;
  if (!gemm_plan(M, N, K, false, true, tile_n, force_ctas, plan)) return nullptr;
  Tensor out;
  const int rc = unlocked([&] {
    out = at::empty(sizes, x.options());
    Tensor partial;
    if (plan.splits > 1) partial = at::empty({plan.splits, M, N}, x.options().dtype(at::kFloat));
    return mdb_gemm_bf16(x.data_ptr(), w.data_ptr(), out.data_ptr(), data(bias), data(residual), nullptr, static_cast<int>(M),
                         static_cast<int>(N), static_cast<int>(K), lda, w.stride(0), N, ldr, 0, 0, 0, 0, epi, 0, 1.0f, plan.ctas,
                         plan.bn, plan.splits, plan.splits > 1 ? partial.data_ptr() : nullptr, stream());
  });
  return done(rc, "mdb_gemm_bf16", out);
  END_HANDLE_TH_ERRORS
}

// geglu_linear(x, weight, bias): [..., K] x [2 N, K]^T -> h * gelu(gate) [..., N]
PyObject* py_geglu_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[1])) return not_implemented();
  const Tensor &x = THPVariable_Unpack(a[0]), &w = THPVariable_Unpack(a[1]);
  const Tensor* bias;
  if (!opt_tensor(a[2], bias)) return not_implemented();
  int64_t M, lda;
  if (!bf16(x) || !bf16(w) || w.dim() != 2 || w.stride(1) != 1 || !rows_of(x, M, lda)) return not_implemented();
  const int64_t K = x.size(-1), N = w.size(0) / 2;
  if (M <= 128) return not_implemented();  // the GEMM and the GEGLU kernel are as fast
  if (w.size(1) != K || w.size(0) % 16 || N <= 0 || K <= 0 || M > INT_MAX || N > INT_MAX / 2 || K > INT_MAX) return not_implemented();
  if (bias && (!bf16(*bias) || !bias->is_contiguous() || bias->numel() != 2 * N)) return not_implemented();
  std::vector<int64_t> sizes(x.sizes().begin(), x.sizes().end());
  sizes.back() = N;
  Tensor out;
  const int rc = unlocked([&] {
    out = at::empty(sizes, x.options());
    return mdb_gemm_geglu(x.data_ptr(), w.data_ptr(), out.data_ptr(), data(bias), static_cast<int>(M), static_cast<int>(N),
                          static_cast<int>(K), lda, w.stride(0), N, stream());
  });
  return done(rc, "mdb_gemm_geglu", out);
  END_HANDLE_TH_ERRORS
}

// linear_group(x, w0, w1[, w2]): [..., K] x each [N, K]^T, side by side -> [..., n * N]
PyObject* py_linear_group(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int mats = static_cast<int>(n) - 1;
  if (mats < 1 || mats > 3) return not_implemented();
  for (Py_ssize_t i = 0; i < n; ++i)
    if (!THPVariable_Check(a[i])) return not_implemented();
  const Tensor &x = THPVariable_Unpack(a[0]), &w = THPVariable_Unpack(a[1]);
  int64_t M, lda;
  if (!bf16(x) || !rows_of(x, M, lda)) return not_implemented();
  const void* ws[3] = {nullptr, nullptr, nullptr};
  for (int i = 0; i < mats; ++i) {
    const Tensor& t = THPVariable_Unpack(a[1 + i]);
    if (!bf16(t) || t.dim() != 2 || t.sizes() != w.sizes() || t.stride(0) != w.stride(0) || t.stride(1) != 1) return not_implemented();
    ws[i] = t.data_ptr();
  }
  const int64_t K = x.size(-1), N = w.size(0);
  if (w.size(1) != K || (N & 7) || N <= 0 || K <= 0 || M > INT_MAX || N > INT_MAX / 3 || K > INT_MAX) return not_implemented();
  std::vector<int64_t> sizes(x.sizes().begin(), x.sizes().end());
  sizes.back() = mats * N;
  Plan plan;
  if (!gemm_plan(M, mats * N, K, false, false, 0, 0, plan)) return nullptr;
  Tensor out;
  const int rc = unlocked([&] {
    out = at::empty(sizes, x.options());
    return mdb_gemm_group(x.data_ptr(), ws, mats, out.data_ptr(), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), lda,
                          w.stride(0), mats * N, plan.ctas, plan.bn, stream());
  });
  return done(rc, "mdb_gemm_group", out);
  END_HANDLE_TH_ERRORS
}

// attention(q, k, v, scale, out): [B,S,H,D] without a log-sum-exp; D a multiple of 8 up to 128. `out` may be None or a view
// whose rows of D are dense (a part of a wider buffer).
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[1]) || !THPVariable_Check(a[2])) return not_implemented();
  const Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]);
  const double scale = PyFloat_AsDouble(a[3]);
  const Tensor* dst = nullptr;
  if (!opt_tensor(a[4], dst)) return not_implemented();
  if (PyErr_Occurred()) return nullptr;
  const Tensor* ts[3] = {&q, &k, &v};
  for (const Tensor* t : ts) {
    if (!bf16(*t) || t->dim() != 4 || t->stride(3) != 1 || t->numel() == 0) return not_implemented();
    if (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15) return not_implemented();
    for (int i = 0; i < 3; ++i)  // a broadcast dimension of a narrow head is copied, as by the padded path
      if ((t->stride(i) & 7) || (t->stride(i) == 0 && t->size(i) > 1 && t->size(3) != 64 && t->size(3) != 128)) return not_implemented();
  }
  if (dst) {
    if (!bf16(*dst) || dst->sizes() != q.sizes() || dst->stride(3) != 1 || (reinterpret_cast<uintptr_t>(dst->data_ptr()) & 15))
      return not_implemented();
    for (int i = 0; i < 3; ++i)
      if (dst->stride(i) & 7) return not_implemented();
  }
  const int64_t B = q.size(0), S = q.size(1), H = q.size(2), D = q.size(3);
  if (D > 128 || (D & 7) || k.size(0) != B || v.size(0) != B || k.size(2) != H || v.size(2) != H || k.size(3) != D ||
      v.size(3) != D || k.size(1) != v.size(1) || k.size(1) > INT_MAX || S > INT_MAX)
    return not_implemented();
  const void *kp = k.data_ptr(), *vp = v.data_ptr();
  const int len = static_cast<int>(k.size(1)), b = static_cast<int>(B), h = static_cast<int>(H), s = static_cast<int>(S);
  Tensor out;
  const int rc = unlocked([&] {
    out = dst ? *dst : at::empty({B, S, H, D}, q.options());
    if (D == 128 || D == 64) {
      return (D == 128 ? mdb_flash_fwd : mdb_flash_fwd_d64)(
          q.data_ptr(), &kp, &vp, out.data_ptr(), nullptr, b, h, s, 1, &len, q.stride(0), q.stride(1), q.stride(2), k.stride(0),
          k.stride(1), k.stride(2), v.stride(0), v.stride(1), v.stride(2), out.stride(0), out.stride(1), out.stride(2),
          static_cast<float>(scale), nullptr, 0, nullptr, stream());
    }
    return mdb_flash_fwd_narrow(q.data_ptr(), &kp, &vp, out.data_ptr(), nullptr, b, h, s, 1, &len, q.stride(0), q.stride(1),
                                q.stride(2), k.stride(0), k.stride(1), k.stride(2), v.stride(0), v.stride(1), v.stride(2),
                                out.stride(0), out.stride(1), out.stride(2), static_cast<float>(scale), static_cast<int>(D),
                                stream());
  });
  return done(rc, "mdb_flash_fwd", out);
  END_HANDLE_TH_ERRORS
}

int ctas_per_batch(int64_t batches, int64_t rows) {
  const int64_t c = kCtasTarget / (batches > 1 ? batches : 1);
  return static_cast<int>(std::max<int64_t>(1, std::min(rows, c)));
}

// layer_norm(x, gamma, beta, scale, shift, eps): x [B,S,C] contiguous
PyObject* py_layer_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !THPVariable_Check(a[0])) return not_implemented();
  const Tensor& x = THPVariable_Unpack(a[0]);
  const Tensor *gamma, *beta, *scale, *shift;
  if (!opt_tensor(a[1], gamma) || !opt_tensor(a[2], beta) || !opt_tensor(a[3], scale) || !opt_tensor(a[4], shift))
    return not_implemented();
  const double eps = PyFloat_AsDouble(a[5]);
  if (PyErr_Occurred()) return nullptr;
  if (!bf16(x) || x.dim() != 3 || !x.is_contiguous() || x.numel() == 0) return not_implemented();
  const int64_t B = x.size(0), S = x.size(1), C = x.size(2);
  for (const Tensor* p : {gamma, beta})
    if (p && (!bf16(*p) || !p->is_contiguous() || p->numel() != C)) return not_implemented();
  if ((scale == nullptr) != (shift == nullptr)) return not_implemented();
  if (scale) {
    for (const Tensor* p : {scale, shift})
      if (!f32(*p) || p->dim() != 2 || p->size(0) != B || p->size(1) != C || p->stride(1) != 1) return not_implemented();
    if (scale->stride(0) != shift->stride(0)) return not_implemented();
  }
  Tensor y;
  const int rc = unlocked([&] {
    y = at::empty_like(x);
    return mdb_ln_fwd(x.data_ptr(), y.data_ptr(), data(gamma), data(beta), static_cast<const float*>(data(scale)),
                      static_cast<const float*>(data(shift)), scale ? scale->stride(0) : 0, static_cast<int>(B), static_cast<int>(S),
                      static_cast<int>(C), static_cast<float>(eps), nullptr, nullptr, ctas_per_batch(B, S), stream());
  });
  return done(rc, "mdb_ln_fwd", y);
  END_HANDLE_TH_ERRORS
}

// geglu(u): [..., 2 inner] contiguous -> [..., inner]
PyObject* py_geglu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 1 || !THPVariable_Check(a[0])) return not_implemented();
  const Tensor& u = THPVariable_Unpack(a[0]);
  if (!bf16(u) || u.dim() < 1 || !u.is_contiguous() || u.numel() == 0 || u.size(-1) % 16) return not_implemented();
  std::vector<int64_t> sizes(u.sizes().begin(), u.sizes().end());
  const int64_t inner = sizes.back() / 2;
  sizes.back() = inner;
  Tensor y;
  const int rc = unlocked([&] {
    y = at::empty(sizes, u.options());
    return mdb_geglu_fwd(u.data_ptr(), y.data_ptr(), u.numel() / (2 * inner), static_cast<int>(inner), stream());
  });
  return done(rc, "mdb_geglu_fwd", y);
  END_HANDLE_TH_ERRORS
}

// rms_rope(x, w, cos, sin, heads, per_head, eps): [B,S,C] -> [B,S,H,D]
PyObject* py_rms_rope(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7 || !THPVariable_Check(a[0])) return not_implemented();
  const Tensor& x = THPVariable_Unpack(a[0]);
  const Tensor *w, *cs, *sn;
  if (!opt_tensor(a[1], w) || !opt_tensor(a[2], cs) || !opt_tensor(a[3], sn)) return not_implemented();
  const int64_t heads = PyLong_AsLong(a[4]);
  const bool per_head = a[5] == Py_True;
  const double eps = PyFloat_AsDouble(a[6]);
  if (PyErr_Occurred()) return nullptr;
  if (!bf16(x) || x.dim() != 3 || x.stride(2) != 1 || x.numel() == 0) return not_implemented();
  const int64_t B = x.size(0), S = x.size(1), C = x.size(2);
  if (x.stride(0) != S * x.stride(1) || heads <= 0 || C % heads) return not_implemented();
  if (w && (!bf16(*w) || !w->is_contiguous())) return not_implemented();
  if ((cs == nullptr) != (sn == nullptr)) return not_implemented();
  if (cs) {
    for (const Tensor* p : {cs, sn})
      if (!f32(*p) || p->dim() != 2 || p->size(0) != S || p->size(1) != 64 || !p->is_contiguous()) return not_implemented();
  }
  Tensor y;
  const int rc = unlocked([&] {
    y = at::empty({B, S, heads, C / heads}, x.options());
    return mdb_rms_rope_fwd(x.data_ptr(), x.stride(1), y.data_ptr(), C, S * C, data(w), per_head, static_cast<const float*>(data(cs)),
                            static_cast<const float*>(data(sn)), static_cast<int>(B), static_cast<int>(S), static_cast<int>(C),
                            static_cast<int>(per_head ? 128 : C), static_cast<float>(eps), nullptr, ctas_per_batch(B, S), stream());
  });
  return done(rc, "mdb_rms_rope_fwd", y);
  END_HANDLE_TH_ERRORS
}

// group_norm_cl(x, groups, gamma, beta, eps, act): x [N,C,H,W] in channels-last memory
PyObject* py_group_norm_cl(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !THPVariable_Check(a[0])) return not_implemented();
  const Tensor& x = THPVariable_Unpack(a[0]);
  const Tensor *gamma, *beta;
  const int64_t groups = PyLong_AsLong(a[1]);
  if (!opt_tensor(a[2], gamma) || !opt_tensor(a[3], beta)) return not_implemented();
  const double eps = PyFloat_AsDouble(a[4]);
  const bool act = a[5] == Py_True;
  if (PyErr_Occurred()) return nullptr;
  if (!bf16(x) || x.dim() != 4 || x.numel() == 0 || !x.is_contiguous(at::MemoryFormat::ChannelsLast) ||
      (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15))
    return not_implemented();
  const int64_t N = x.size(0), C = x.size(1), HW = x.size(2) * x.size(3);
  if (groups <= 0 || C % groups || (C & 7) || N > 65535 || HW > INT_MAX) return not_implemented();
  for (const Tensor* p : {gamma, beta})
    if (p && (!bf16(*p) || !p->is_contiguous() || p->numel() != C)) return not_implemented();
  const int splits = static_cast<int>(std::max<int64_t>(1, std::min((kCtasTarget + N - 1) / N, (HW + 15) / 16)));
  const int in = static_cast<int>(N), ic = static_cast<int>(C), ihw = static_cast<int>(HW), ig = static_cast<int>(groups);
  Tensor y;
  if (mdb_gn_cl_group != nullptr) {
    const int rc = unlocked([&] {
      y = at::empty_like(x);
      return mdb_gn_cl_group(x.data_ptr(), y.data_ptr(), in, ihw, ic, ig, splits, static_cast<float>(eps), data(gamma), data(beta),
                             gamma || beta ? 1 : 0, nullptr, 0, act, stream());
    });
    if (rc != kGnGroupElsewhere) return done(rc, "mdb_gn_cl_group", y);
  }
  if (C > 2048) return not_implemented();
  const int rc = unlocked([&] {
    // one buffer: the strips' sums, then a and b [N, C], mean and rstd [N, groups]
    const int64_t sums = N * splits * C * 2;
    const auto f = x.options().dtype(at::kFloat).memory_format(at::MemoryFormat::Contiguous);
    const Tensor work = at::empty({sums + 2 * N * C + 2 * N * groups}, f);
    float* partial = work.data_ptr<float>();
    float *ca = partial + sums, *cb = ca + N * C, *mean = cb + N * C, *rstd = mean + N * groups;
    if (!y.defined()) y = at::empty_like(x);
    void* st = stream();
    int err = mdb_gn_cl_sums(x.data_ptr(), nullptr, nullptr, nullptr, partial, in, ihw, ic, splits, st);
    if (err == 0)
      err = mdb_gn_cl_fold_fwd(partial, in, splits, ic, ig, static_cast<float>(HW * (C / groups)), static_cast<float>(eps),
                               data(gamma), data(beta), gamma || beta ? 1 : 0, ca, cb, mean, rstd, st);
    if (err == 0)
      err = mdb_gn_cl_apply(x.data_ptr(), nullptr, y.data_ptr(), ca, cb, nullptr, nullptr, nullptr, in, ihw, ic, act, st);
    return err;
  });
  return done(rc, "mdb_gn_cl", y, 3);
  END_HANDLE_TH_ERRORS
}

// Integers of a tuple; false (and no Python error) when it is not a tuple of that many.
template <typename T>
bool ints(PyObject* o, T* out, Py_ssize_t n) {
  if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != n) return false;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const long long v = PyLong_AsLongLong(PyTuple_GET_ITEM(o, i));
    if (v == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
    out[i] = static_cast<T>(v);
  }
  return true;
}

// conv(x, x_alt, w, out, bias, residual, dims, strides, alt_dims, alt_strides, box, ext, c_in, n_pad, taps, begin, alt_dim,
//      alt_shift, out_strides, class_off, epi, ctas, max_bn, splits, m_tiles, group): the arguments of `ops.conv._launch`, shapes as
// tuples, taps and begin as the addresses of int arrays. Returns `out`.
PyObject* py_conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 26 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[2]) || !THPVariable_Check(a[3])) return not_implemented();
  const Tensor &x = THPVariable_Unpack(a[0]), &w = THPVariable_Unpack(a[2]), &out = THPVariable_Unpack(a[3]);
  const Tensor *alt, *bias, *residual;
  if (!opt_tensor(a[1], alt) || !opt_tensor(a[4], bias) || !opt_tensor(a[5], residual)) return not_implemented();
  long long dims[5], strides[4], alt_dims[5], alt_strides[4], os[4], class_off[4] = {0, 0, 0, 0};
  int box[3], ext[4];
  const Py_ssize_t classes = PyTuple_Check(a[19]) ? PyTuple_GET_SIZE(a[19]) : 0;
  if (classes < 1 || classes > 4 || !ints(a[6], dims, 5) || !ints(a[7], strides, 4) || !ints(a[8], alt_dims, 5) ||
      !ints(a[9], alt_strides, 4) || !ints(a[10], box, 3) || !ints(a[11], ext, 4) || !ints(a[18], os, 4) ||
      !ints(a[19], class_off, classes))
    return not_implemented();
  const int c_in = static_cast<int>(PyLong_AsLong(a[12])), n_pad = static_cast<int>(PyLong_AsLong(a[13]));
  const int* taps = static_cast<const int*>(PyLong_AsVoidPtr(a[14]));
  const int* begin = static_cast<const int*>(PyLong_AsVoidPtr(a[15]));
  const int alt_dim = static_cast<int>(PyLong_AsLong(a[16])), alt_shift = static_cast<int>(PyLong_AsLong(a[17]));
  const int epi = static_cast<int>(PyLong_AsLong(a[20])), ctas = static_cast<int>(PyLong_AsLong(a[21]));
  const int max_bn = static_cast<int>(PyLong_AsLong(a[22])), splits = static_cast<int>(PyLong_AsLong(a[23]));
  const int64_t m_tiles = PyLong_AsLongLong(a[24]);
  const int group = static_cast<int>(PyLong_AsLong(a[25]));
  if (PyErr_Occurred()) return nullptr;
  const int rc = unlocked([&] {
    Tensor partial;
    if (splits > 1)
      partial = at::empty({splits * static_cast<int64_t>(classes) * m_tiles * 128 * n_pad},
                          out.options().dtype(at::kFloat).memory_format(at::MemoryFormat::Contiguous));
    return mdb_conv_igemm(x.data_ptr(), data(alt), w.data_ptr(), out.data_ptr(), data(bias), data(residual), dims, strides, alt_dims,
                          alt_strides, box, ext, c_in, n_pad, w.size(1), static_cast<int>(classes), begin, taps, alt_dim, alt_shift,
                          os, class_off, epi, ctas, max_bn, splits, splits > 1 ? partial.data_ptr() : nullptr, group, stream());
  });
  return done(rc, "mdb_conv_igemm", out);
  END_HANDLE_TH_ERRORS
}

// setup(KernelError, gemm_plan)
PyObject* py_setup(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "setup(error, plan)");
    return nullptr;
  }
  Py_INCREF(a[0]);
  Py_XSETREF(g_error, a[0]);
  Py_INCREF(a[1]);
  Py_XSETREF(g_plan, a[1]);
  g_plans.clear();
  Py_RETURN_NONE;
}

PyObject* py_launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches); }

#define MDB_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {MDB_FAST(gemm), MDB_FAST(linear), MDB_FAST(geglu_linear), MDB_FAST(linear_group), MDB_FAST(attention), MDB_FAST(layer_norm), MDB_FAST(geglu),
                          MDB_FAST(rms_rope), MDB_FAST(group_norm_cl), MDB_FAST(conv), MDB_FAST(setup),
                          {"launches", py_launches, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_ops() { return PyModule_Create(&kModule); }
