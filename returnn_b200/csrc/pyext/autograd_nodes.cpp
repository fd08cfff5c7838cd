// Autograd nodes of operators that a model calls in every layer: layer norm, linear layer, convolution module, attention with head dim 64, softmax
// cross entropy. They allocate and launch what the Python functions of returnn_b200/ops do (which stay for traced
// programs), without the interpreter: in the backward pass the engine's thread does not wait for the GIL. A layer norm of 6656 x 512, forward and
// backward, is 16 us of kernels; its calls took 122 us. The kernels are those of librb200.so.
//
// Everything a node keeps goes through save_for_backward, so hooks on saved tensors see it; nothing is kept between calls but the launch count.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

extern "C" {
const char* rb200_last_error();
int rb200_layer_norm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, long long rows, int n, float eps, int x_bf16,
                         int w_bf16, int rms, cudaStream_t stream);
int rb200_layer_norm_bwd(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd, void* dx, float* part, float* dgamma,
                         float* dbeta, long long rows, int n, int n_part, int x_bf16, int w_bf16, int rms, cudaStream_t stream);
int rb200_layer_norm_bwd_typed(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd, void* dx, float* work, void* dgamma,
                               void* dbeta, long long rows, int n, int w_bf16, int rms, cudaStream_t stream);
int rb200_gemm_bf16_ex(const void* a, const void* b, void* c, void* c2, const void* bias, int m, int n, int k, int lda, int ldb, int ldc, int a_mn_major,
                       int b_mn_major, int bias_bf16, int act, int out_fp32, int accumulate, float alpha, const void* dact_z, float drop_p,
                       const long long* seed, const long long* offset, unsigned long long drop_site, const void* resid, float res_scale, int split_k,
                       int* status, cudaStream_t stream);
int rb200_act_grad_colsum(const void* z, const void* dy, void* dz, float* db, float* work, int m, int n, int act, cudaStream_t stream);
int rb200_weight_grad_slices(int m, int k, int n);
int rb200_weight_grad_sliced(const void* x, const void* dy, float* part, float* dw, int m, int k, int n, int rows, int* status, cudaStream_t stream);
int rb200_conv_module_fwd(const void* x, const float* filt, const float* bias, const float* gamma, const float* beta, const int* row_batch,
                          const int* row_pos, const int* lens, void* y, void* z, float* part, float* stats, float* running_mean, float* running_var,
                          int n_rows, int n_seqs, int C, int K, int own_stats, float eps, float momentum, cudaStream_t stream);
int rb200_conv_module_bwd(const void* x, const void* y, const void* dz, const float* stats, const float* filt, const float* gamma, const float* beta,
                          const int* row_batch, const int* row_pos, const int* lens, void* ds, float* part, int n_tiles, float* sum_ds, float* sum_ds_yh,
                          void* dx, float* dfilt, float* dbias, int n_rows, int n_seqs, int C, int K, cudaStream_t stream);
int rb200_flash_fwd(const void* q, const void* k, const void* v, void* o, float* o32, float* lse, void* keep, const int* k_lens, const int* g, float scale,
                    float p_drop, const long long* seed, const long long* offset, int* status, cudaStream_t stream);
int rb200_flash_bwd_one_kernel(int tq, int tk);
int rb200_flash_bwd(const void* q, const void* k, const void* v, const float* o32, const void* d_o, void* dq, void* dk, void* dv, float* lse, float* delta,
                    void* keep, const int* k_lens, const int* g, float scale, float p_drop, int* status, cudaStream_t stream);
int rb200_softmax_ce_fwd(const void* logits, const int* targets, float* loss, float* lse, long long rows, int v, float smoothing, int is_bf16, int grad_only,
                         int* amax, cudaStream_t stream);
int rb200_softmax_ce_bwd(const void* logits, const int* targets, const float* lse, const float* dloss, void* dlogits, long long rows, int v, float smoothing,
                         int is_bf16, int grad_only, cudaStream_t stream);
}

namespace {

std::atomic<long long> launches{0};

void count(int n = 1) { launches.fetch_add(n, std::memory_order_relaxed); }
void check(int status, const char* what) {
  TORCH_CHECK(status == 0, what, " failed with status ", status, " ", rb200_last_error());
}
cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
template <typename T = void>
T* ptr(const Tensor& t) {
  return static_cast<T*>(t.data_ptr());
}
template <typename T = void>
T* ptr(const OptTensor& t) {
  return t.has_value() && t->defined() ? static_cast<T*>(t->data_ptr()) : nullptr;
}
bool is_bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }

// A debugger of the kernels (ops/guard.py) may allocate in our place: hook(like, shape, type) with type 0 fp32, 1 bf16, 2 int32, None: not its concern
std::atomic<PyObject*> allocator{nullptr};

Tensor hooked(PyObject* hook, at::IntArrayRef shape, const Tensor& like, at::ScalarType type) {
  const int code = type == at::kFloat ? 0 : type == at::kBFloat16 ? 1 : type == at::kInt ? 2 : -1;
  Tensor res;
  if (code >= 0) {
    const PyGILState_STATE gil = PyGILState_Ensure();
    PyObject* dims = PyTuple_New((Py_ssize_t)shape.size());
    for (size_t i = 0; dims && i < shape.size(); ++i) PyTuple_SET_ITEM(dims, (Py_ssize_t)i, PyLong_FromLongLong(shape[i]));
    PyObject* t = dims ? THPVariable_Wrap(like.detach()) : nullptr;
    PyObject* r = t ? PyObject_CallFunction(hook, "OOi", t, dims, code) : nullptr;
    if (r && THPVariable_Check(r)) res = THPVariable_Unpack(r);
    const bool failed = r == nullptr;
    Py_XDECREF(r);
    Py_XDECREF(t);
    Py_XDECREF(dims);
    if (failed) PyErr_Clear();
    PyGILState_Release(gil);
    TORCH_CHECK(!failed, "the allocation hook failed");
  }
  return res;
}

Tensor fresh(at::IntArrayRef shape, const Tensor& like, at::ScalarType type) {
  if (PyObject* hook = allocator.load(std::memory_order_acquire)) {
    const Tensor t = hooked(hook, shape, like, type);
    if (t.defined()) return t;
  }
  return at::empty(shape, like.options().dtype(type));
}
Tensor fresh_like(const Tensor& t) { return fresh(t.sizes(), t, t.scalar_type()); }  // (contiguous)

// ---- layer norm, RMS norm
struct LayerNorm : Function<LayerNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& gamma, const OptTensor& beta, double eps, bool rms) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t n = x.size(-1);
    const Tensor x2 = x.reshape({-1, n}).contiguous();
    const int64_t rows = x2.size(0);
    const Tensor g = gamma.contiguous();
    const Tensor b = beta.has_value() ? beta->contiguous() : Tensor();
    Tensor y = fresh_like(x2);
    Tensor mean = fresh({rows}, x, at::kFloat), rstd = fresh({rows}, x, at::kFloat);
    check(rb200_layer_norm_fwd(ptr(x2), ptr(g), b.defined() ? ptr(b) : nullptr, ptr(y), ptr<float>(mean), ptr<float>(rstd), rows, (int)n, (float)eps, is_bf16(x2),
                               is_bf16(g), rms, stream()),
          "layer_norm_fwd");
    count();
    ctx->save_for_backward({x2, g, mean, rstd});
    ctx->saved_data["has_beta"] = beta.has_value();
    ctx->saved_data["rms"] = rms;
    ctx->saved_data["shape"] = x.sizes().vec();
    return y.reshape(x.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &g = saved[1], &mean = saved[2], &rstd = saved[3];
    const c10::cuda::CUDAGuard guard(x2.device());
    const bool has_beta = ctx->saved_data["has_beta"].toBool(), rms = ctx->saved_data["rms"].toBool();
    const auto shape = ctx->saved_data["shape"].toIntVector();
    const int64_t rows = x2.size(0), n = x2.size(1);
    const Tensor dy = grads[0].reshape({rows, n}).contiguous();
    Tensor dx = fresh_like(x2);
    if (is_bf16(x2) && n <= 512 && rows > 0 && is_bf16(dy) && (is_bf16(g) || g.scalar_type() == at::kFloat)) {
      // one kernel, which also leaves the parameter gradients in the type of the parameters
      Tensor work = fresh({2 * n + 1}, x2, at::kFloat);
      Tensor dgamma = fresh_like(g), dbeta = has_beta ? fresh_like(g) : Tensor();
      check(rb200_layer_norm_bwd_typed(ptr(x2), ptr(dy), ptr(g), ptr<float>(mean), ptr<float>(rstd), ptr(dx), ptr<float>(work), ptr(dgamma),
                                       has_beta ? ptr(dbeta) : nullptr, rows, (int)n, is_bf16(g), rms, stream()),
            "layer_norm_bwd");
      count();
      return {dx.reshape(shape), dgamma, dbeta, Tensor(), Tensor()};
    }
    const int64_t n_part = std::min<int64_t>(296, std::max<int64_t>(1, (rows + 31) / 32));
    Tensor part = fresh({2, n_part, n}, x2, at::kFloat), dgamma = fresh({n}, x2, at::kFloat), dbeta = fresh({n}, x2, at::kFloat);
    check(rb200_layer_norm_bwd(ptr(x2), ptr(dy), ptr(g), ptr<float>(mean), ptr<float>(rstd), ptr(dx), ptr<float>(part), ptr<float>(dgamma), ptr<float>(dbeta), rows,
                               (int)n, (int)n_part, is_bf16(x2), is_bf16(g), rms, stream()),
          "layer_norm_bwd");
    count(2);
    return {dx.reshape(shape), dgamma.to(g.scalar_type()), has_beta ? dbeta.to(g.scalar_type()) : Tensor(), Tensor(), Tensor()};
  }
};

// ---- linear layer
// c [m, n] = a b with the operands' layouts as they are stored (see rb200_gemm_bf16_ex)
void gemm(const Tensor& a, const Tensor& b, const Tensor& c, const Tensor* c2, const OptTensor& bias, int64_t m, int64_t n, int64_t k, bool a_mn, bool b_mn, int act,
          const Tensor& status) {
  const int64_t lda = a.size(0) == 1 ? a.size(1) : a.stride(0), ldb = b.size(0) == 1 ? b.size(1) : b.stride(0);
  check(rb200_gemm_bf16_ex(ptr(a), ptr(b), ptr(c), c2 ? ptr(*c2) : nullptr, ptr(bias), (int)m, (int)n, (int)k, (int)lda, (int)ldb, (int)c.stride(0), a_mn, b_mn,
                           bias.has_value() && is_bf16(*bias), act, c.scalar_type() == at::kFloat, 0, 1.f, nullptr, 0.f, nullptr, nullptr, 0, nullptr, 1.f, 0,
                           ptr<int>(status), stream()),
        "gemm_bf16_ex");
  count();
}

bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }

// gradient before the activation and its column sums (db, if defined), elementwise: shapes that the kernel does not take
Tensor grad_pre_elementwise(const Tensor& dy, const Tensor& z, int act, const Tensor& db) {
  Tensor dz = dy;
  if (act) {
    const Tensor zf = z.to(at::kFloat), d = dy.to(at::kFloat);
    if (act == 1) {
      dz = at::where(zf > 0, dy, at::zeros({}, dy.options()));  // (also where the gradient is not finite)
    } else if (act == 2) {
      const Tensor s = at::sigmoid(zf);
      dz = (d * (s * (1 + zf * (1 - s)))).to(dy.scalar_type());
    } else {
      const Tensor cdf = 0.5 * (1 + at::erf(zf * 0.7071067811865476)), pdf = at::exp(-0.5 * zf * zf) * 0.3989422804014327;
      dz = (d * (cdf + zf * pdf)).to(dy.scalar_type());
    }
  }
  if (db.defined()) db.copy_(dz.to(at::kFloat).sum(0));
  return dz;
}

struct Linear : Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x2, const Tensor& weight, const OptTensor& bias, int64_t act, bool differentiable, const Tensor& status) {
    const c10::cuda::CUDAGuard guard(x2.device());
    const Tensor w = weight.to(at::kBFloat16).contiguous();
    const int64_t m = x2.size(0), k = x2.size(1), n = w.size(1);
    Tensor y = fresh({m, n}, x2, at::kBFloat16), z;
    // (a parameter says that it requires a gradient under no_grad as well; that of the bias alone needs the pre-activation too)
    if (act && differentiable && (x2.requires_grad() || weight.requires_grad() || (bias.has_value() && bias->requires_grad()))) {
      z = fresh({m, n}, x2, at::kBFloat16);
      gemm(x2, w, z, &y, bias, m, n, k, false, true, (int)act, status);
    } else {
      gemm(x2, w, y, nullptr, bias, m, n, k, false, true, (int)act, status);
    }
    ctx->save_for_backward({x2, w, z});
    ctx->saved_data["act"] = act;
    ctx->saved_data["w_dtype"] = weight.scalar_type();
    ctx->saved_data["has_bias"] = bias.has_value();
    if (bias.has_value()) ctx->saved_data["bias_dtype"] = bias->scalar_type();
    ctx->saved_data["status"] = status;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &w = saved[1], &z = saved[2];
    const c10::cuda::CUDAGuard guard(x2.device());
    const Tensor status = ctx->saved_data["status"].toTensor();
    const int act = (int)ctx->saved_data["act"].toInt();
    const bool has_bias = ctx->saved_data["has_bias"].toBool();
    const int64_t m = x2.size(0), k = x2.size(1), n = w.size(1);
    Tensor dy = grads[0].contiguous(), dx, dw, db;
    if (has_bias && ctx->needs_input_grad(2)) db = fresh({n}, dy, at::kFloat);
    if (act || db.defined()) {
      // 16-byte accesses: a gradient that starts off that alignment takes the elementwise form
      if (is_bf16(dy) && n % 8 == 0 && aligned16(dy) && (!z.defined() || aligned16(z))) {
        Tensor dz = act ? fresh_like(dy) : dy, work;
        if (db.defined()) work = fresh({4 * 148 * 64 + n}, dy, at::kFloat);
        check(rb200_act_grad_colsum(act ? ptr(z) : nullptr, ptr(dy), act ? ptr(dz) : nullptr, db.defined() ? ptr<float>(db) : nullptr,
                                    work.defined() ? ptr<float>(work) : nullptr, (int)m, (int)n, act, stream()),
              "act_grad_colsum");
        count(work.defined() ? 2 : 1);
        dy = dz;
      } else {
        dy = grad_pre_elementwise(dy, z, act, db);
      }
    }
    if (ctx->needs_input_grad(0)) {
      // dX[m,k] = dY[m,n] W[k,n]^T: contraction over n, W rows are contiguous in n -> "K-major" B
      dx = fresh({m, k}, x2, at::kBFloat16);
      gemm(dy, w, dx, nullptr, std::nullopt, m, k, n, false, false, 0, status);
    }
    if (ctx->needs_input_grad(1)) {
      // dW[k,n] = X[m,k]^T dY[m,n]: contraction over m, both operands contiguous in their output dim
      const auto w_dtype = ctx->saved_data["w_dtype"].toScalarType();
      if (w_dtype == at::kFloat) {
        dw = fresh({k, n}, x2, at::kFloat);
        const int rows = rb200_weight_grad_slices((int)m, (int)k, (int)n);
        if (rows == 0) {
          gemm(x2, dy, dw, nullptr, std::nullopt, k, n, m, true, true, 0, status);
        } else {
          Tensor part = fresh({(m + rows - 1) / rows, k, n}, x2, at::kFloat);
          check(rb200_weight_grad_sliced(ptr(x2), ptr(dy), ptr<float>(part), ptr<float>(dw), (int)m, (int)k, (int)n, rows, ptr<int>(status), stream()),
                "weight_grad_sliced");
          count(2);
        }
      } else {
        dw = fresh({k, n}, x2, at::kBFloat16);
        gemm(x2, dy, dw, nullptr, std::nullopt, k, n, m, true, true, 0, status);
        dw = dw.to(w_dtype);
      }
    }
    if (db.defined()) db = db.to(ctx->saved_data["bias_dtype"].toScalarType());
    return {dx, dw, db, Tensor(), Tensor(), Tensor()};
  }
};

Tensor linear(const Tensor& x_, const Tensor& weight, OptTensor bias, int64_t act, const Tensor& status) {
  Tensor x = is_bf16(x_) ? x_ : x_.to(at::kBFloat16);
  if (bias.has_value() && !is_bf16(*bias) && bias->scalar_type() != at::kFloat) bias = bias->to(at::kFloat);
  const Tensor x2 = x.reshape({-1, x.size(-1)}).contiguous();
  const Tensor y = Linear::apply(x2, weight, bias, act, at::GradMode::is_enabled(), status);
  if (x.dim() == 2) return y;
  auto shape = x.sizes().vec();
  shape.back() = weight.size(1);
  return y.reshape(shape);
}

// ---- convolution module
struct ConvModule : Function<ConvModule> {
  // batch statistics only: with running statistics the caller takes the Python function
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& filt, const OptTensor& bias, const OptTensor& gamma, const OptTensor& beta,
                        const OptTensor& running_mean, const OptTensor& running_var, const Tensor& row_batch, const Tensor& row_pos, const Tensor& lens, double eps,
                        double momentum) {
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = x_.contiguous();
    const int64_t N = x.size(0), C = x.size(1) / 2, K = filt.size(-1);
    auto f32 = [](const OptTensor& t) { return t.has_value() ? t->to(at::kFloat).contiguous() : Tensor(); };
    const Tensor f = filt.reshape({C, K}).to(at::kFloat).contiguous(), b = f32(bias), g = f32(gamma), be = f32(beta);
    auto p = [](const Tensor& t) { return t.defined() ? ptr<float>(t) : nullptr; };
    Tensor y = fresh({N, C}, x, at::kBFloat16), z = fresh({N, C}, x, at::kBFloat16);
    Tensor part = fresh({(N + 31) / 32 * 2 * C}, x, at::kFloat), stats = fresh({2, C}, x, at::kFloat);  // mean, 1 / deviation
    check(rb200_conv_module_fwd(ptr(x), ptr<float>(f), p(b), p(g), p(be), ptr<int>(row_batch), ptr<int>(row_pos), ptr<int>(lens), ptr(y), ptr(z), ptr<float>(part),
                                ptr<float>(stats), ptr<float>(running_mean), ptr<float>(running_var), (int)N, (int)lens.size(0), (int)C, (int)K, 1, (float)eps,
                                (float)momentum, stream()),
          "conv_module_fwd");
    count(K <= 32 ? 4 : 3);
    ctx->save_for_backward({x, f, y, stats, g, be, row_batch, row_pos, lens});
    auto& d = ctx->saved_data;
    d["fshape"] = filt.sizes().vec();
    d["fdtype"] = filt.scalar_type();
    if (bias.has_value()) d["bdtype"] = bias->scalar_type();
    if (gamma.has_value()) d["gdtype"] = gamma->scalar_type();
    if (beta.has_value()) d["bedtype"] = beta->scalar_type();
    return z;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &f = s[1], &y = s[2], &stats = s[3], &g = s[4], &be = s[5], &row_batch = s[6], &row_pos = s[7], &lens = s[8];
    const c10::cuda::CUDAGuard guard(x.device());
    auto& d = ctx->saved_data;
    const int64_t N = x.size(0), C = x.size(1) / 2, K = f.size(1);
    const Tensor dz = grads[0].contiguous();
    const int64_t tiles = std::min<int64_t>(296, std::max<int64_t>(1, (N + 15) / 16));
    Tensor ds = fresh({N, C}, x, at::kBFloat16);
    // the sums of the two passes, one after the other in the same scratch
    Tensor part = fresh({std::max(tiles * 2 * C, (N + 31) / 32 * C * (K + 1))}, x, at::kFloat);
    Tensor sum_ds = fresh({C}, x, at::kFloat), sum_ds_yh = fresh({C}, x, at::kFloat), dx = fresh_like(x), df = fresh({C, K}, x, at::kFloat);
    const bool has_bias = d.count("bdtype") > 0, has_gamma = d.count("gdtype") > 0, has_beta = d.count("bedtype") > 0;
    Tensor db = has_bias ? fresh({C}, x, at::kFloat) : Tensor();
    auto p = [](const Tensor& t) { return t.defined() ? ptr<float>(t) : nullptr; };
    check(rb200_conv_module_bwd(ptr(x), ptr(y), ptr(dz), ptr<float>(stats), ptr<float>(f), p(g), p(be), ptr<int>(row_batch), ptr<int>(row_pos), ptr<int>(lens),
                                ptr(ds), ptr<float>(part), (int)tiles, ptr<float>(sum_ds), ptr<float>(sum_ds_yh), ptr(dx), ptr<float>(df), p(db), (int)N,
                                (int)lens.size(0), (int)C, (int)K, stream()),
          "conv_module_bwd");
    count(5);
    const Tensor none;
    return {dx, df.reshape(d["fshape"].toIntVector()).to(d["fdtype"].toScalarType()), has_bias ? db.to(d["bdtype"].toScalarType()) : none,
            has_gamma ? sum_ds_yh.to(d["gdtype"].toScalarType()) : none, has_beta ? sum_ds.to(d["bedtype"].toScalarType()) : none,
            none, none, none, none, none, none, none};
  }
};

// ---- attention, head dim 64
// [B, T, H, 64] -> bf16 tensor that the kernels address in place, row pitch, head pitch (see ops/sdpa.py, _rows)
Tensor rows_of(const Tensor& t_, int64_t& row, int64_t& head) {
  Tensor t = is_bf16(t_) ? t_ : t_.to(at::kBFloat16);
  const int64_t B = t.size(0), T = t.size(1), H = t.size(2), D = t.size(3);
  int64_t sb = t.stride(0), st = t.stride(1), sh = t.stride(2);
  bool ok = t.stride(3) == 1 && (T == 1 || st % 8 == 0) && (H == 1 || sh % 8 == 0) && aligned16(t);
  if (ok && T == 1) {
    st = B > 1 ? sb : std::max((H - 1) * sh + D, (int64_t)8);
    ok = st % 8 == 0;
  }
  if (ok && H == 1) sh = D;
  ok = ok && (B == 1 || sb == T * st) && sh >= D && st >= (H - 1) * sh + D;
  if (!ok) {
    t = t.contiguous();
    st = H * D;
    sh = D;
  }
  row = st;
  head = sh;
  return t;
}

// seed [2] int64 (key, counter) where there is dropout
struct Flash : Function<Flash> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& k_lens, bool causal, double scale, double p_drop,
                        const OptTensor& seed, const Tensor& status) {
    const c10::cuda::CUDAGuard guard(q.device());
    const int64_t B = q.size(0), Tq = q.size(1), H = q.size(2), Tk = k.size(1);
    std::vector<int64_t> geom(17, 0);
    const Tensor q2 = rows_of(q, geom[6], geom[7]), k2 = rows_of(k, geom[8], geom[9]), v2 = rows_of(v, geom[10], geom[11]);
    const int64_t Tqp = (Tq + 63) / 64 * 64, Tkp = (Tk + 63) / 64 * 64, words = (Tk + 127) / 128 * 4;
    geom[0] = B; geom[1] = H; geom[2] = Tq; geom[3] = Tk; geom[4] = causal; geom[5] = Tk - Tq;
    geom[14] = Tqp; geom[15] = Tkp; geom[16] = words;
    Tensor o = fresh({B, Tq, H, 64}, q, at::kBFloat16), lse = fresh({B * H * Tq}, q, at::kFloat), o32, keep, off;
    // the backward pass takes row sums of the output: from a copy of its own in 32 bits, so that the caller may change the result in place
    // (the one kernel of short sequences takes them from the probabilities)
    if ((q.requires_grad() || k.requires_grad() || v.requires_grad()) && !rb200_flash_bwd_one_kernel((int)Tq, (int)Tk)) o32 = fresh({B, Tq, H, 64}, q, at::kFloat);
    if (p_drop > 0.) {
      keep = fresh({B * H * Tq * words}, q, at::kInt);
      off = seed->slice(0, 1, 2).clone();
      seed->select(0, 1).add_(B * H * Tqp * Tkp);
    }
    const std::vector<int> g(geom.begin(), geom.end());
    check(rb200_flash_fwd(ptr(q2), ptr(k2), ptr(v2), ptr(o), o32.defined() ? ptr<float>(o32) : nullptr, ptr<float>(lse), keep.defined() ? ptr(keep) : nullptr,
                          ptr<int>(k_lens), g.data(), (float)scale, (float)p_drop, p_drop > 0. ? ptr<long long>(*seed) : nullptr,
                          off.defined() ? ptr<long long>(off) : nullptr, ptr<int>(status), stream()),
          "flash_fwd");
    count();
    ctx->save_for_backward({q2, k2, v2, o32, lse, keep, k_lens.has_value() ? *k_lens : Tensor()});
    auto& d = ctx->saved_data;
    d["geom"] = geom;
    d["scale"] = scale;
    d["p_drop"] = p_drop;
    d["dtype"] = q.scalar_type();
    d["status"] = status;
    return is_bf16(q) ? o : o.to(q.scalar_type());
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &q2 = s[0], &k2 = s[1], &v2 = s[2], &o32 = s[3], &lse = s[4], &keep = s[5], &k_lens = s[6];
    const c10::cuda::CUDAGuard guard(q2.device());
    auto& d = ctx->saved_data;
    auto geom = d["geom"].toIntVector();
    const Tensor d_o = rows_of(grads[0], geom[12], geom[13]), status = d["status"].toTensor();
    const int64_t B = geom[0], H = geom[1], Tq = geom[2], Tk = geom[3];
    Tensor delta = o32.defined() ? fresh_like(lse) : Tensor(), dq = fresh({B, Tq, H, 64}, q2, at::kBFloat16), dk = fresh({B, Tk, H, 64}, q2, at::kBFloat16),
           dv = fresh({B, Tk, H, 64}, q2, at::kBFloat16);
    const std::vector<int> g(geom.begin(), geom.end());
    check(rb200_flash_bwd(ptr(q2), ptr(k2), ptr(v2), o32.defined() ? ptr<float>(o32) : nullptr, ptr(d_o), ptr(dq), ptr(dk), ptr(dv), ptr<float>(lse),
                          delta.defined() ? ptr<float>(delta) : nullptr,
                          keep.defined() ? ptr(keep) : nullptr, k_lens.defined() ? ptr<int>(k_lens) : nullptr, g.data(), (float)d["scale"].toDouble(),
                          (float)d["p_drop"].toDouble(), ptr<int>(status), stream()),
          "flash_bwd");
    count(o32.defined() ? 2 : 1);
    const auto dt = d["dtype"].toScalarType();
    const Tensor none;
    return {dq.to(dt), dk.to(dt), dv.to(dt), none, none, none, none, none, none};
  }
};

// ---- softmax cross entropy (without the arg max)
struct CrossEntropy : Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits_, const Tensor& targets, double smoothing, bool grad_only) {
    const c10::cuda::CUDAGuard guard(logits_.device());
    const Tensor logits = logits_.contiguous(), tgt = targets.to(at::kInt).contiguous();
    const int64_t rows = logits.size(0), v = logits.size(1);
    Tensor loss = fresh({rows}, logits, at::kFloat), lse = fresh({rows}, logits, at::kFloat);
    check(rb200_softmax_ce_fwd(ptr(logits), ptr<int>(tgt), ptr<float>(loss), ptr<float>(lse), rows, (int)v, (float)smoothing, is_bf16(logits), grad_only, nullptr,
                               stream()),
          "softmax_ce_fwd");
    count();
    ctx->save_for_backward({logits, tgt, lse});
    ctx->saved_data["smoothing"] = smoothing;
    ctx->saved_data["grad_only"] = grad_only;
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &logits = s[0], &tgt = s[1], &lse = s[2];
    const c10::cuda::CUDAGuard guard(logits.device());
    Tensor dlogits = fresh_like(logits);
    const Tensor dl = grads[0].to(at::kFloat).contiguous();
    check(rb200_softmax_ce_bwd(ptr(logits), ptr<int>(tgt), ptr<float>(lse), ptr<float>(dl), ptr(dlogits), logits.size(0), (int)logits.size(1),
                               (float)ctx->saved_data["smoothing"].toDouble(), is_bf16(logits), ctx->saved_data["grad_only"].toBool(), stream()),
          "softmax_ce_bwd");
    count();
    return {dlogits, Tensor(), Tensor(), Tensor()};
  }
};

// ---- the Python side: positional arguments, checked for number and type
struct Args {
  PyObject* const* args;
  const Tensor& tensor(int i) const {
    TORCH_CHECK_TYPE(THPVariable_Check(args[i]), "argument ", i, " must be a tensor");
    return THPVariable_Unpack(args[i]);
  }
  OptTensor opt(int i) const { return args[i] == Py_None ? OptTensor() : OptTensor(tensor(i)); }
  double number(int i) const {
    const double v = PyFloat_AsDouble(args[i]);
    if (v == -1. && PyErr_Occurred()) throw python_error();
    return v;
  }
  int64_t integer(int i) const {
    const long long v = PyLong_AsLongLong(args[i]);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
  }
  bool truth(int i) const { return PyObject_IsTrue(args[i]) == 1; }
};

template <int N, typename Call>
PyObject* enter(PyObject* const* args, Py_ssize_t n, Call call) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n == N, "expected ", N, " arguments, got ", (long)n);
  return THPVariable_Wrap(call(Args{args}));
  END_HANDLE_TH_ERRORS
}

PyObject* py_layer_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return enter<5>(args, n, [](Args a) { return LayerNorm::apply(a.tensor(0), a.tensor(1), a.opt(2), a.number(3), a.truth(4)); });
}
PyObject* py_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return enter<5>(args, n, [](Args a) { return linear(a.tensor(0), a.tensor(1), a.opt(2), a.integer(3), a.tensor(4)); });
}
PyObject* py_conv_module(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return enter<12>(args, n, [](Args a) {
    return ConvModule::apply(a.tensor(0), a.tensor(1), a.opt(2), a.opt(3), a.opt(4), a.opt(5), a.opt(6), a.tensor(7), a.tensor(8), a.tensor(9), a.number(10),
                             a.number(11));
  });
}
PyObject* py_flash(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return enter<9>(args, n, [](Args a) {
    return Flash::apply(a.tensor(0), a.tensor(1), a.tensor(2), a.opt(3), a.truth(4), a.number(5), a.number(6), a.opt(7), a.tensor(8));
  });
}
PyObject* py_cross_entropy(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return enter<4>(args, n, [](Args a) { return CrossEntropy::apply(a.tensor(0), a.tensor(1), a.number(2), a.truth(3)); });
}
PyObject* py_set_allocator(PyObject*, PyObject* hook) {  // the caller keeps the hook alive until it is replaced
  allocator.store(hook == Py_None ? nullptr : hook, std::memory_order_release);
  Py_RETURN_NONE;
}
PyObject* py_launches(PyObject*, PyObject*) { return PyLong_FromLongLong(launches.load(std::memory_order_relaxed)); }

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyMethodDef fast(const char* name, const char* doc) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F)), METH_FASTCALL, doc};
}

PyMethodDef methods[] = {
    fast<py_layer_norm>("layer_norm", "(x, gamma, beta, eps, rms) -> y"),
    fast<py_linear>("linear", "(x, weight, bias, act, status) -> y"),
    fast<py_conv_module>("conv_module", "(x, filt, bias, gamma, beta, running_mean, running_var, row_batch, row_pos, lens, eps, momentum) -> z"),
    fast<py_flash>("flash", "(q, k, v, k_lens, causal, scale, p_drop, seed, status) -> o"),
    fast<py_cross_entropy>("cross_entropy", "(logits, targets, smoothing, grad_only) -> loss"),
    {"set_allocator", py_set_allocator, METH_O, "(hook or None): allocate through hook(like, shape, type); for debugging"},
    {"launches", py_launches, METH_NOARGS, "kernels launched by the nodes so far"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_autograd_nodes", "autograd nodes of the native operators", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__autograd_nodes() { return PyModule_Create(&module); }
