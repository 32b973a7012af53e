// The fused ops of the flow API on local tensors, in native code: checks, result allocation, kernel launches and the autograd nodes.
// Small calls were bound by the host (a decoding step of one token spent 350 us in Python for 65 us of kernels); here a call costs one
// Python-to-C transition. Every entry point answers None when a call is not of the plain form it serves (other types, devices and
// layouts, active modes, transforms and tracers, forward-mode tangents, refused arguments); the Python statement of the op
// (framework/fused_ops.py, _C.py, ops/) then runs and raises what there is to raise.
//
// Counterpart in the reference: the functional layer and its autograd nodes in C++ (oneflow/core/functional/impl/nn_functor.cpp,
// oneflow/core/autograd/gradient_funcs/matmul.cpp, layer_norm.cpp, scaled_dot_product_attention.cpp).
#define PY_SSIZE_T_CLEAN
#include <torch/extension.h>

#include <ATen/cuda/EmptyTensor.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <array>
#include <atomic>
#include <optional>

#include "../kernels/ofb_kernels.h"

extern "C" {
int ofb_layer_norm_fwd(const void*, const void*, const void*, void*, float*, float*, int, int, float, void*);
int ofb_layer_norm_bwd_parts(int);
int ofb_layer_norm_bwd_to(const void*, const void*, const void*, const float*, const float*, const void*, void*, void*, void*, float*, int, int,
                          int, int, void*);
int ofb_column_sum(const void*, float*, int, int, void*);
int ofb_column_sum_store(const void*, void*, int, int, int, void*);
int ofb_bias_act_bwd(const void*, const void*, const void*, void*, long long, int, int, void*);
int ofb_xent_stats(const void*, const long long*, float*, int, int, long long, int, void*);
int ofb_xent_grad_scaled(const void*, const long long*, const float*, float*, void*, int, int, long long, int, float, long long, const float*,
                         long long, void*);
int ofb_fmha_fwd_ex(const void*, const void*, const void*, long long, long long, void*, float*, const int*, int, int, int, int, int, int, int,
                    float, float, unsigned long long, unsigned int, void*);
long long ofb_fmha_bwd_scratch_floats(int, int, int, int);
int ofb_fmha_bwd_ex(const void*, const void*, const void*, long long, long long, const void*, const void*, const float*, void*, void*, void*,
                    long long, long long, float*, const int*, int, int, int, int, int, int, int, float, float, unsigned long long, unsigned int,
                    void*);
}

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

std::atomic<long long> g_launches{0};

struct Refused {};   // a kernel entry point refused the call before it launched anything: the Python statement reports it

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

Tensor new_cuda(at::IntArrayRef size, at::ScalarType type, const Tensor& like) {
  return at::detail::empty_cuda(size, type, like.device(), std::nullopt);
}

bool aligned(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) == 0; }

// A dense tensor whose memory kernels may read through its pointer.
bool plain(const Tensor& t, at::ScalarType type) {
  return t.is_cuda() && t.scalar_type() == type && t.layout() == at::kStrided && !t.unsafeGetTensorImpl()->is_python_dispatch();
}
bool plain_bf16(const Tensor& t) { return plain(t, at::kBFloat16); }

// Modes, transforms and tracers see the Python statement of an op.
bool intercepted() {
  return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::PythonTorchFunctionTLS::stack_len() > 0 ||
         c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) ||
         c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Functionalize) || torch::jit::tracer::isTracing();
}

bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }

template <typename... Ts>
bool wants_grad(const Ts&... ts) {
  return at::GradMode::is_enabled() && (... || (ts.defined() && ts.requires_grad()));
}

Tensor dense(const Tensor& t) {
  Tensor c = t.contiguous();
  return aligned(c) ? c : c.clone();
}

// ------------------------------------------------------------------------------------------------ products
struct Product {
  const Tensor *a, *b;
  bool a_km = false, b_kn = false;
  const Tensor *bias = nullptr, *residual = nullptr, *aux_in = nullptr;
  const Tensor *aux_out = nullptr, *out = nullptr;
  int64_t ldr = 0;
  int act = 0;
  bool accumulate = false;
};

// Operands are matrices (or contiguous stacks of rows) of which only the last dimension's size counts: lda is given by the caller.
int run_product(const Product& p, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldb, int64_t ldc, int64_t ld_aux) {
  OfbGemmArgs g;
  std::memset(&g, 0, sizeof(g));
  g.A = p.a->const_data_ptr();
  g.B = p.b->const_data_ptr();
  g.C = p.out->mutable_data_ptr();
  g.bias = p.bias ? p.bias->const_data_ptr() : nullptr;
  g.residual = p.residual ? p.residual->const_data_ptr() : nullptr;
  g.aux_in = p.aux_in ? p.aux_in->const_data_ptr() : nullptr;
  g.aux_out = p.aux_out ? p.aux_out->mutable_data_ptr() : nullptr;
  g.lda = lda; g.ldb = ldb; g.ldc = ldc; g.ldr = p.ldr; g.ld_aux = ld_aux;
  g.M = static_cast<int>(M); g.N = static_cast<int>(N); g.K = static_cast<int>(K);
  g.a_mn_major = p.a_km; g.b_mn_major = p.b_kn;
  g.act = p.act;
  g.out_fp32 = p.out->scalar_type() == at::kFloat;
  g.accumulate = p.accumulate;
  g.alpha = 1.f;
  const int rc = ofb_gemm_bf16(&g, stream());
  if (rc == 0) g_launches.fetch_add(1, std::memory_order_relaxed);
  return rc;
}

void backward_ok(int rc, const char* what) { TORCH_CHECK(rc == 0, what, " failed: ", ofb_last_error()); }

// dx = dy w (times act'(aux)), [rows, K] from [rows, N] and [N, K]
Tensor data_gradient(const Tensor& dy, const Tensor& w, int64_t rows, int64_t N, int64_t K, at::IntArrayRef shape, const Tensor& aux, int act) {
  Tensor dx = new_cuda(shape, at::kBFloat16, dy);
  Product p;
  p.a = &dy; p.b = &w; p.b_kn = true; p.out = &dx;
  if (aux.defined()) { p.aux_in = &aux; p.act = act; }
  backward_ok(run_product(p, rows, K, N, N, w.dim() == 2 ? w.stride(0) : K, K, K), "gemm");
  return dx;
}

// dw = dy^T x, [N, K]
Tensor weight_gradient(const Tensor& dy, const Tensor& x, int64_t rows, int64_t N, int64_t K, at::IntArrayRef shape) {
  Tensor dw = new_cuda(shape, at::kBFloat16, dy);
  Product p;
  p.a = &dy; p.b = &x; p.a_km = p.b_kn = true; p.out = &dw;
  backward_ok(run_product(p, N, K, rows, N, K, K, 0), "gemm");
  return dw;
}

// Which of the two kernels sums the columns: the same line as ops/kernels.py: column_sum.
bool column_sum_one_launch(int64_t rows, int64_t cols, bool bf16) {
  return bf16 ? rows <= 4096 && cols <= 6144 && rows * cols <= (1 << 23) : rows <= 2048 && cols <= 2048;
}

Tensor bias_gradient(const Tensor& dy, int64_t rows, int64_t N, at::IntArrayRef shape) {
  if (column_sum_one_launch(rows, N, true)) {
    Tensor db = new_cuda(shape, at::kBFloat16, dy);
    backward_ok(ofb_column_sum_store(dy.const_data_ptr(), db.mutable_data_ptr(), static_cast<int>(rows), static_cast<int>(N), 1, stream()),
                "column_sum");
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return db;
  }
  Tensor sum = new_cuda(shape, at::kFloat, dy).zero_();
  backward_ok(ofb_column_sum(dy.const_data_ptr(), sum.data_ptr<float>(), static_cast<int>(rows), static_cast<int>(N), stream()), "column_sum");
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return sum.to(at::kBFloat16);
}

// What `linear` needs to know of its operands; ok is false for calls that the Python statement serves.
struct LinearShape {
  bool ok = false;
  int64_t rows = 0, N = 0, K = 0, ldw = 0;
  std::vector<int64_t> out;

  LinearShape(const Tensor& x, const Tensor& w, const Tensor& bias, const Tensor& residual) {
    if (!plain_bf16(x) || !plain_bf16(w) || x.dim() < 1 || x.numel() == 0 || w.numel() == 0 || (w.dim() != 2 && w.dim() != 3)) return;
    K = w.size(-1);
    if (x.size(-1) != K || x.device() != w.device() || K % 8 || w.size(-2) % 8 || !aligned(w)) return;
    if (w.is_contiguous()) ldw = K;
    else if (w.dim() == 2 && w.stride(1) == 1 && w.stride(0) >= K && w.stride(0) % 8 == 0) ldw = w.stride(0);
    else return;
    N = w.numel() / K;
    rows = x.numel() / K;
    if (rows > INT32_MAX || N > INT32_MAX) return;
    out.assign(x.sizes().begin(), x.sizes().end() - 1);
    out.insert(out.end(), w.sizes().begin(), w.sizes().end() - 1);
    if (bias.defined() && (!plain_bf16(bias) || bias.numel() != N || !bias.is_contiguous() || !aligned(bias) || bias.device() != x.device()))
      return;
    if (residual.defined() && (!plain_bf16(residual) || !residual.sizes().equals(out) || !residual.is_contiguous() || !aligned(residual) ||
                               residual.device() != x.device()))
      return;
    ok = !has_tangent(x) && !has_tangent(w) && !has_tangent(bias) && !has_tangent(residual);
  }
};

// y = act(x w^T + bias) + residual; aux receives the pre-activations where wanted. x2: dense rows.
Tensor linear_forward(const Tensor& x2, const Tensor& w, const Tensor& bias, const Tensor& residual, int act, const LinearShape& s, Tensor* aux) {
  Tensor y = new_cuda(s.out, at::kBFloat16, x2);
  Product p;
  p.a = &x2; p.b = &w; p.out = &y; p.act = act;
  if (bias.defined()) p.bias = &bias;
  if (residual.defined()) { p.residual = &residual; p.ldr = s.N; }
  if (aux) {
    *aux = new_cuda(s.out, at::kBFloat16, x2);
    p.aux_out = aux;
  }
  if (run_product(p, s.rows, s.N, s.K, s.K, s.ldw, s.N, s.N)) throw Refused{};
  return y;
}

OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }

// Backward of y = act(x w^T + b) + residual. `act` is 0 where there is none or where the consumer of an `mlp` has applied its gradient;
// `x_aux` are the pre-activations that x itself came from through `x_act` (inside an `mlp`): their gradient goes into the epilogue of the
// data gradient.
struct LinearNode : public Function<LinearNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& bias_, const OptTensor& residual_,
                               int64_t act, const LinearShape& s, bool private_out, const OptTensor& x_aux, int64_t x_act) {
    const Tensor bias = bias_.value_or(Tensor()), residual = residual_.value_or(Tensor());
    Tensor x2 = dense(x), aux;
    Tensor y = linear_forward(x2, w, bias, residual, static_cast<int>(act), s, act ? &aux : nullptr);
    // the pre-activations belong to whoever applies the activation's gradient: this node, or the consumer of a private result
    ctx->save_for_backward({x2, w, act && !private_out ? aux : Tensor(), x_aux.value_or(Tensor())});
    ctx->saved_data["act"] = private_out ? int64_t(0) : act;
    ctx->saved_data["x_act"] = x_act;
    ctx->saved_data["x_shape"] = x.sizes().vec();
    ctx->saved_data["rows"] = s.rows;
    ctx->saved_data["N"] = s.N;
    ctx->saved_data["has_b"] = bias.defined();
    ctx->saved_data["has_r"] = residual.defined();
    if (bias.defined()) ctx->saved_data["b_shape"] = bias.sizes().vec();
    ctx->saved_data["y_shape"] = s.out;
    ctx->set_materialize_grads(false);    // no gradient of zeros for the pre-activations (16384 x 4096: 35 us)
    if (private_out && aux.defined()) {
      ctx->mark_non_differentiable({aux});
      return {y, aux};
    }
    return {y};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &w = saved[1], &aux = saved[2], &x_aux = saved[3];
    const int act = static_cast<int>(ctx->saved_data["act"].toInt());
    const int64_t rows = ctx->saved_data["rows"].toInt(), N = ctx->saved_data["N"].toInt(), K = w.size(-1);
    const auto x_shape = ctx->saved_data["x_shape"].toIntVector();
    variable_list out(9);   // one per argument of forward
    // inputs that are there count as edges, in their order
    const bool has_b = ctx->saved_data["has_b"].toBool(), has_r = ctx->saved_data["has_r"].toBool();
    const bool want_x = ctx->needs_input_grad(0), want_w = ctx->needs_input_grad(1), want_b = has_b && ctx->needs_input_grad(2);
    const Tensor dy = grads[0].defined() ? grads[0] : at::zeros(ctx->saved_data["y_shape"].toIntVector(), x2.options());
    if (has_r && ctx->needs_input_grad(2 + has_b)) out[3] = dy;
    if (!want_x && !want_w && !want_b) return out;
    c10::cuda::CUDAGuard guard(dy.device());
    Tensor d = dense(dy);
    if (act) {
      Tensor pre = new_cuda(d.sizes(), at::kBFloat16, d);
      backward_ok(ofb_bias_act_bwd(aux.const_data_ptr(), nullptr, d.const_data_ptr(), pre.mutable_data_ptr(), d.numel(), static_cast<int>(N), act,
                                   stream()),
                  "bias_act_bwd");
      g_launches.fetch_add(1, std::memory_order_relaxed);
      d = pre;
    }
    if (want_x)
      out[0] = data_gradient(d, w, rows, N, K, x_shape, x_aux, static_cast<int>(ctx->saved_data["x_act"].toInt()));
    if (want_w) out[1] = weight_gradient(d, x2, rows, N, K, w.sizes());
    if (want_b) out[2] = bias_gradient(d, rows, N, ctx->saved_data["b_shape"].toIntVector());
    return out;
  }
};

Tensor linear(const Tensor& x, const Tensor& w, const Tensor& bias, const Tensor& residual, int act) {
  const LinearShape s(x, w, bias, residual);
  if (!s.ok) throw Refused{};
  c10::cuda::CUDAGuard guard(x.device());
  if (wants_grad(x, w, bias, residual)) return LinearNode::apply(x, w, opt(bias), opt(residual), act, s, false, OptTensor(), 0)[0];
  at::AutoDispatchBelowADInplaceOrView below;
  return linear_forward(dense(x), w, bias, residual, act, s, nullptr);
}

Tensor mlp(const Tensor& x, const Tensor& w1, const Tensor& b1, const Tensor& w2, const Tensor& b2, const Tensor& residual, int act) {
  const LinearShape s1(x, w1, b1, Tensor());
  if (!s1.ok || w1.dim() != 2 || w2.dim() != 2 || !plain_bf16(w2) || w2.size(1) != s1.N || s1.N % 8) throw Refused{};
  c10::cuda::CUDAGuard guard(x.device());
  if (!wants_grad(x, w1, b1, w2, b2, residual)) {
    at::AutoDispatchBelowADInplaceOrView below;
    Tensor h = linear_forward(dense(x), w1, b1, Tensor(), act, s1, nullptr);
    const LinearShape s2(h, w2, b2, residual);
    if (!s2.ok) throw Refused{};
    return linear_forward(h, w2, b2, residual, 0, s2, nullptr);
  }
  // Both layers' forms are known before the first one runs: a refusal leaves no work behind
  std::vector<int64_t> h_shape = s1.out;
  {
    std::vector<int64_t> y_shape(h_shape.begin(), h_shape.end() - 1);
    y_shape.push_back(w2.size(0));
    if (w2.size(0) % 8 || !aligned(w2) || !(w2.is_contiguous() || (w2.stride(1) == 1 && w2.stride(0) >= w2.size(1) && w2.stride(0) % 8 == 0)) ||
        (b2.defined() && (!plain_bf16(b2) || b2.numel() != w2.size(0) || !b2.is_contiguous() || !aligned(b2))) ||
        (residual.defined() && (!plain_bf16(residual) || !residual.sizes().equals(y_shape) || !residual.is_contiguous() || !aligned(residual))) ||
        has_tangent(w2) || has_tangent(b2) || has_tangent(residual))
      throw Refused{};
  }
  Tensor h, aux;
  if (wants_grad(x, w1, b1)) {
    auto first = LinearNode::apply(x, w1, opt(b1), OptTensor(), act, s1, act != 0, OptTensor(), 0);
    h = first[0];
    if (act) aux = first[1];
  } else {
    at::AutoDispatchBelowADInplaceOrView below;
    h = linear_forward(dense(x), w1, b1, Tensor(), act, s1, nullptr);
  }
  const LinearShape s2(h, w2, b2, residual);
  if (!s2.ok) throw Refused{};
  return LinearNode::apply(h, w2, opt(b2), opt(residual), 0, s2, false, opt(aux), act)[0];
}

// ------------------------------------------------------------------------------------------------ layer norm
struct LayerNormNode : public Function<LayerNormNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps) {
    const int64_t cols = x.size(-1), rows = x.numel() / cols;
    Tensor x2 = dense(x);
    Tensor y = new_cuda(x.sizes(), at::kBFloat16, x), mean = new_cuda({rows}, at::kFloat, x), rstd = new_cuda({rows}, at::kFloat, x);
    run(x2, gamma, beta, y, mean, rstd, rows, cols, eps);
    ctx->save_for_backward({x2, gamma, mean, rstd});
    return {y};
  }
  static void run(const Tensor& x2, const Tensor& gamma, const Tensor& beta, const Tensor& y, const Tensor& mean, const Tensor& rstd, int64_t rows,
                  int64_t cols, double eps) {
    if (ofb_layer_norm_fwd(x2.const_data_ptr(), gamma.const_data_ptr(), beta.const_data_ptr(), y.mutable_data_ptr(), mean.data_ptr<float>(),
                           rstd.data_ptr<float>(), static_cast<int>(rows), static_cast<int>(cols), static_cast<float>(eps), stream()))
      throw Refused{};
    g_launches.fetch_add(1, std::memory_order_relaxed);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &gamma = saved[1], &mean = saved[2], &rstd = saved[3];
    c10::cuda::CUDAGuard guard(x2.device());
    const int64_t cols = x2.size(-1), rows = x2.numel() / cols;
    Tensor dy = dense(grads[0]);
    Tensor dx = new_cuda(dy.sizes(), at::kBFloat16, x2), dg, db, scratch;
    const bool want = ctx->needs_input_grad(1) || ctx->needs_input_grad(2);
    if (want) {
      dg = new_cuda(gamma.sizes(), at::kBFloat16, x2);
      db = new_cuda(gamma.sizes(), at::kBFloat16, x2);
      scratch = new_cuda({2 * int64_t(ofb_layer_norm_bwd_parts(static_cast<int>(rows))) * cols}, at::kFloat, x2);
    }
    backward_ok(ofb_layer_norm_bwd_to(dy.const_data_ptr(), x2.const_data_ptr(), gamma.const_data_ptr(), mean.data_ptr<float>(),
                                      rstd.data_ptr<float>(), nullptr, dx.mutable_data_ptr(), want ? dg.mutable_data_ptr() : nullptr,
                                      want ? db.mutable_data_ptr() : nullptr, want ? scratch.data_ptr<float>() : nullptr, 0, want ? 1 : 0,
                                      static_cast<int>(rows), static_cast<int>(cols), stream()),
                "layer_norm_bwd");
    g_launches.fetch_add(want ? 2 : 1, std::memory_order_relaxed);
    variable_list out(4);
    if (ctx->needs_input_grad(0)) out[0] = dx;
    if (ctx->needs_input_grad(1)) out[1] = dg;
    if (ctx->needs_input_grad(2)) out[2] = db;
    return out;
  }
};

Tensor layer_norm(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps) {
  if (!plain_bf16(x) || !plain_bf16(gamma) || !plain_bf16(beta) || x.dim() < 1 || x.numel() == 0) throw Refused{};
  const int64_t cols = x.size(-1);
  if (cols % 8 || cols > 32768 || x.numel() / cols > INT32_MAX) throw Refused{};
  for (const Tensor* t : {&gamma, &beta})
    if (t->numel() != cols || t->dim() != 1 || !t->is_contiguous() || !aligned(*t) || t->device() != x.device() || has_tangent(*t)) throw Refused{};
  if (has_tangent(x)) throw Refused{};
  c10::cuda::CUDAGuard guard(x.device());
  if (wants_grad(x, gamma, beta)) return LayerNormNode::apply(x, gamma, beta, eps)[0];
  at::AutoDispatchBelowADInplaceOrView below;
  const int64_t rows = x.numel() / cols;
  Tensor y = new_cuda(x.sizes(), at::kBFloat16, x), stats = new_cuda({2, rows}, at::kFloat, x);
  Tensor x2 = dense(x);
  if (ofb_layer_norm_fwd(x2.const_data_ptr(), gamma.const_data_ptr(), beta.const_data_ptr(), y.mutable_data_ptr(), stats.data_ptr<float>(),
                         stats.data_ptr<float>() + rows, static_cast<int>(rows), static_cast<int>(cols), static_cast<float>(eps), stream()))
    throw Refused{};
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return y;
}

// ------------------------------------------------------------------------------------------------ attention
// A [B, H, S, D] tensor whose memory is rows of tokens with their heads contiguous inside: the kernels' form.
struct Heads {
  bool ok;
  int64_t B, H, S, D, row;
  explicit Heads(const Tensor& t) : B(t.size(0)), H(t.size(1)), S(t.size(2)), D(t.size(3)), row(t.stride(2)) {
    ok = t.stride(3) == 1 && t.stride(1) == D && t.stride(0) == S * t.stride(2) && aligned(t);
  }
};

Tensor token_major(const Tensor& t) { return dense(t.transpose(1, 2)).transpose(1, 2); }   // [B, H, S, D], dense as [B, S, H, D]

Tensor empty_token_major(int64_t B, int64_t H, int64_t S, int64_t D, const Tensor& like) {
  return at::detail::empty_strided_cuda({B, H, S, D}, {S * H * D, D, H * D, 1}, at::kBFloat16, like.device());
}

Tensor sdpa_run(const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale, Tensor* lse_out) {
  const Heads a(q), b(k), c(v);
  Tensor out = empty_token_major(a.B, a.H, a.S, a.D, q), lse = new_cuda({a.B, a.H, a.S}, at::kFloat, q);
  if (ofb_fmha_fwd_ex(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), a.row, b.row, out.mutable_data_ptr(), lse.data_ptr<float>(),
                      nullptr, static_cast<int>(a.B), static_cast<int>(a.S), static_cast<int>(b.S), static_cast<int>(a.H),
                      static_cast<int>(b.H), static_cast<int>(a.D), causal ? 1 : 0, static_cast<float>(scale), 0.f, 0, 0, stream()))
    throw Refused{};
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (lse_out) *lse_out = lse;
  return out;
}

struct SdpaNode : public Function<SdpaNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale) {
    Tensor lse;
    Tensor out = sdpa_run(q, k, v, causal, scale, &lse);
    ctx->save_for_backward({q, k, v, out, lse});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return {out};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2], &out = saved[3], &lse = saved[4];
    c10::cuda::CUDAGuard guard(q.device());
    const Heads a(q), b(k);
    Tensor d = dense(grads[0].transpose(1, 2));
    Tensor dq = empty_token_major(a.B, a.H, a.S, a.D, q), dk = empty_token_major(b.B, b.H, b.S, b.D, q),
           dv = empty_token_major(b.B, b.H, b.S, b.D, q);
    Tensor scratch = new_cuda({ofb_fmha_bwd_scratch_floats(static_cast<int>(a.B), static_cast<int>(a.S), static_cast<int>(a.H),
                                                           static_cast<int>(a.D))},
                              at::kFloat, q);
    backward_ok(ofb_fmha_bwd_ex(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), a.row, b.row, out.const_data_ptr(), d.const_data_ptr(),
                                lse.data_ptr<float>(), dq.mutable_data_ptr(), dk.mutable_data_ptr(), dv.mutable_data_ptr(), a.H * a.D, b.H * b.D,
                                scratch.data_ptr<float>(), nullptr, static_cast<int>(a.B), static_cast<int>(a.S), static_cast<int>(b.S),
                                static_cast<int>(a.H), static_cast<int>(b.H), static_cast<int>(a.D), ctx->saved_data["causal"].toBool() ? 1 : 0,
                                static_cast<float>(ctx->saved_data["scale"].toDouble()), 0.f, 0, 0, stream()),
                "fmha_bwd");
    g_launches.fetch_add(3, std::memory_order_relaxed);
    return {dq, dk, dv, Tensor(), Tensor()};
  }
};

Tensor sdpa(const Tensor& query, const Tensor& key, const Tensor& value, bool causal, double scale) {
  for (const Tensor* t : {&query, &key, &value})
    if (!plain_bf16(*t) || t->dim() != 4 || t->numel() == 0 || has_tangent(*t) || t->device() != query.device()) throw Refused{};
  const int64_t D = query.size(3), H = query.size(1), Hk = key.size(1);
  if ((D != 64 && D != 128) || key.size(3) != D || !key.sizes().equals(value.sizes()) || H % Hk || query.size(0) != key.size(0)) throw Refused{};
  c10::cuda::CUDAGuard guard(query.device());
  Tensor q = query, k = key, v = value;
  const Heads a(q), b(k), c(v);
  if (!a.ok || !b.ok || !c.ok || b.row != c.row) {
    q = token_major(q);
    k = token_major(k);
    v = token_major(v);
    // a single token keeps the strides of its old order when it is "made contiguous": refused here and in Python
    if (!Heads(q).ok || !Heads(k).ok || !Heads(v).ok) throw Refused{};
  }
  if (wants_grad(q, k, v)) return SdpaNode::apply(q, k, v, causal, scale)[0];
  at::AutoDispatchBelowADInplaceOrView below;
  return sdpa_run(q, k, v, causal, scale, nullptr);
}

// Self-attention over a packed projection [tokens, 3, heads * D].
struct PackedAttentionNode : public Function<PackedAttentionNode> {
  static Tensor run(const Tensor& qkv, int64_t seq, int64_t D, bool causal, double scale, Tensor* lse_out) {
    const int64_t T = qkv.size(0), HD = qkv.size(2), B = T / seq, H = HD / D;
    Tensor out = new_cuda({T, HD}, at::kBFloat16, qkv), lse = new_cuda({B, H, seq}, at::kFloat, qkv);
    const auto* p = static_cast<const at::BFloat16*>(qkv.const_data_ptr());
    if (ofb_fmha_fwd_ex(p, p + HD, p + 2 * HD, 3 * HD, 3 * HD, out.mutable_data_ptr(), lse.data_ptr<float>(), nullptr, static_cast<int>(B),
                        static_cast<int>(seq), static_cast<int>(seq), static_cast<int>(H), static_cast<int>(H), static_cast<int>(D), causal ? 1 : 0,
                        static_cast<float>(scale), 0.f, 0, 0, stream()))
      throw Refused{};
    g_launches.fetch_add(1, std::memory_order_relaxed);
    if (lse_out) *lse_out = lse;
    return out;
  }
  static variable_list forward(AutogradContext* ctx, const Tensor& qkv, int64_t seq, int64_t D, bool causal, double scale) {
    Tensor lse;
    Tensor out = run(qkv, seq, D, causal, scale, &lse);
    ctx->save_for_backward({qkv, out, lse});
    ctx->saved_data["seq"] = seq;
    ctx->saved_data["D"] = D;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return {out};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &qkv = saved[0], &out = saved[1], &lse = saved[2];
    c10::cuda::CUDAGuard guard(qkv.device());
    const int64_t seq = ctx->saved_data["seq"].toInt(), D = ctx->saved_data["D"].toInt();
    const int64_t T = qkv.size(0), HD = qkv.size(2), B = T / seq, H = HD / D;
    Tensor d = dense(grads[0]), dqkv = new_cuda(qkv.sizes(), at::kBFloat16, qkv);
    Tensor scratch = new_cuda({ofb_fmha_bwd_scratch_floats(static_cast<int>(B), static_cast<int>(seq), static_cast<int>(H), static_cast<int>(D))},
                              at::kFloat, qkv);
    const auto* p = static_cast<const at::BFloat16*>(qkv.const_data_ptr());
    auto* g = static_cast<at::BFloat16*>(dqkv.mutable_data_ptr());
    backward_ok(ofb_fmha_bwd_ex(p, p + HD, p + 2 * HD, 3 * HD, 3 * HD, out.const_data_ptr(), d.const_data_ptr(), lse.data_ptr<float>(), g, g + HD,
                                g + 2 * HD, 3 * HD, 3 * HD, scratch.data_ptr<float>(), nullptr, static_cast<int>(B), static_cast<int>(seq),
                                static_cast<int>(seq), static_cast<int>(H), static_cast<int>(H), static_cast<int>(D),
                                ctx->saved_data["causal"].toBool() ? 1 : 0, static_cast<float>(ctx->saved_data["scale"].toDouble()), 0.f, 0, 0,
                                stream()),
                "fmha_bwd");
    g_launches.fetch_add(3, std::memory_order_relaxed);
    return {dqkv, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor attention_packed(const Tensor& qkv, int64_t seq, int64_t D, bool causal, double scale) {
  if (!plain_bf16(qkv) || qkv.dim() != 3 || qkv.size(1) != 3 || qkv.numel() == 0 || !qkv.is_contiguous() || !aligned(qkv) || has_tangent(qkv) ||
      (D != 64 && D != 128) || qkv.size(2) % D || seq < 1 || qkv.size(0) % seq || seq > INT32_MAX)
    throw Refused{};
  c10::cuda::CUDAGuard guard(qkv.device());
  if (wants_grad(qkv)) return PackedAttentionNode::apply(qkv, seq, D, causal, scale)[0];
  at::AutoDispatchBelowADInplaceOrView below;
  return PackedAttentionNode::run(qkv, seq, D, causal, scale, nullptr);
}

// ------------------------------------------------------------------------------------------------ cross entropy
struct XentNode : public Function<XentNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& logits, const Tensor& labels) {
    Tensor stats;
    Tensor loss = run(logits, labels, &stats);
    ctx->save_for_backward({logits, labels, stats});
    return {loss};
  }
  static Tensor run(const Tensor& logits, const Tensor& labels, Tensor* stats_out) {
    const int rows = static_cast<int>(logits.size(0)), cols = static_cast<int>(logits.size(1));
    Tensor stats = new_cuda({rows, 3}, at::kFloat, logits), loss = new_cuda({rows}, at::kFloat, logits);
    const auto* lab = reinterpret_cast<const long long*>(labels.const_data_ptr());
    if (ofb_xent_stats(logits.const_data_ptr(), lab, stats.data_ptr<float>(), rows, cols, cols, 0, stream())) throw Refused{};
    if (ofb_xent_grad_scaled(logits.const_data_ptr(), lab, stats.data_ptr<float>(), loss.data_ptr<float>(), nullptr, rows, cols, cols, 0, 1.f, -100,
                             nullptr, 0, stream()))
      throw Refused{};
    g_launches.fetch_add(2, std::memory_order_relaxed);
    *stats_out = stats;
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &logits = saved[0], &labels = saved[1], &stats = saved[2];
    c10::cuda::CUDAGuard guard(logits.device());
    const int rows = static_cast<int>(logits.size(0)), cols = static_cast<int>(logits.size(1));
    Tensor dl = grads[0].to(at::kFloat), loss = new_cuda({rows}, at::kFloat, logits);
    // (softmax - onehot) * dloss over the logits' own storage: they are not needed again
    backward_ok(ofb_xent_grad_scaled(logits.const_data_ptr(), reinterpret_cast<const long long*>(labels.const_data_ptr()), stats.data_ptr<float>(),
                                     loss.data_ptr<float>(), const_cast<void*>(logits.const_data_ptr()), rows, cols, cols, 0, 1.f, -100,
                                     dl.data_ptr<float>(), dl.stride(0), stream()),
                "xent_grad");
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return {logits.detach(), Tensor()};
  }
};

Tensor cross_entropy(const Tensor& logits, const Tensor& labels) {
  if (!plain_bf16(logits) || logits.dim() != 2 || logits.numel() == 0 || !logits.is_contiguous() || !aligned(logits) || logits.size(1) % 8 ||
      has_tangent(logits) || logits.size(0) > INT32_MAX || logits.size(1) > INT32_MAX)
    throw Refused{};
  if (!plain(labels, at::kLong) || labels.numel() != logits.size(0) || !labels.is_contiguous() || labels.device() != logits.device()) throw Refused{};
  c10::cuda::CUDAGuard guard(logits.device());
  if (wants_grad(logits)) return XentNode::apply(logits, labels)[0];
  at::AutoDispatchBelowADInplaceOrView below;
  Tensor stats;
  return XentNode::run(logits, labels, &stats);
}

// ------------------------------------------------------------------------------------------------ single kernels (no autograd)
bool matrix(const Tensor& t) {
  return plain_bf16(t) && t.dim() == 2 && t.stride(1) == 1 && t.stride(0) % 8 == 0 && aligned(t);
}

// ops/gemm.py: gemm with alpha = 1 and the tile left to the dispatch. Returns (out, aux or undefined).
std::pair<Tensor, Tensor> gemm(const Tensor& a, const Tensor& b, bool a_km, bool b_kn, const Tensor& bias, int act, const Tensor& residual,
                               const Tensor& aux_in, bool want_aux, const Tensor& out_given, bool fp32, bool accumulate) {
  if (!matrix(a) || !matrix(b)) throw Refused{};
  const int64_t M = a.size(a_km ? 1 : 0), K = a.size(a_km ? 0 : 1), N = b.size(b_kn ? 1 : 0), Kb = b.size(b_kn ? 0 : 1);
  if (K != Kb || N % 8 || M < 1 || N < 1 || K < 1 || M > INT32_MAX || N > INT32_MAX || K > INT32_MAX) throw Refused{};
  for (const Tensor* t : {&bias, &residual, &aux_in})
    if (t->defined() && (!plain_bf16(*t) || !aligned(*t) || t->device() != a.device())) throw Refused{};
  if (b.device() != a.device() || (bias.defined() && (!bias.is_contiguous() || bias.numel() != N))) throw Refused{};
  for (const Tensor* t : {&residual, &aux_in})
    if (t->defined() && (t->dim() != 2 || t->size(0) != M || t->size(1) != N || t->stride(1) != 1 || t->stride(0) % 8)) throw Refused{};
  Tensor out = out_given;
  if (out.defined()) {
    if (!(plain_bf16(out) || plain(out, at::kFloat)) || out.dim() != 2 || out.size(0) != M || out.size(1) != N || out.stride(1) != 1 ||
        out.device() != a.device() || !aligned(out) || out.stride(0) % 8)
      throw Refused{};
  } else if (accumulate) {
    throw Refused{};
  }
  c10::cuda::CUDAGuard guard(a.device());
  at::AutoDispatchBelowADInplaceOrView below;
  if (!out.defined()) out = new_cuda({M, N}, fp32 ? at::kFloat : at::kBFloat16, a);
  Tensor aux = want_aux ? new_cuda({M, N}, at::kBFloat16, a) : Tensor();
  Product p;
  p.a = &a; p.b = &b; p.a_km = a_km; p.b_kn = b_kn; p.out = &out; p.act = act; p.accumulate = accumulate;
  if (bias.defined()) p.bias = &bias;
  if (residual.defined()) { p.residual = &residual; p.ldr = residual.stride(0); }
  if (aux_in.defined()) p.aux_in = &aux_in;
  if (want_aux) p.aux_out = &aux;
  const int64_t ld_aux = aux_in.defined() ? aux_in.stride(0) : want_aux ? N : 0;
  if (run_product(p, M, N, K, a.stride(0), b.stride(0), out.stride(0), ld_aux)) throw Refused{};
  return {out, aux};
}

bool vector(const Tensor& t, int64_t n, at::ScalarType type, const Tensor& like) {
  return plain(t, type) && t.numel() == n && t.is_contiguous() && aligned(t) && t.device() == like.device();
}
bool dense_rows(const Tensor& t) { return plain_bf16(t) && t.dim() == 2 && t.numel() > 0 && t.is_contiguous() && aligned(t); }

// ops/kernels.py: layer_norm_fwd with both parameters -> y, mean, rstd
std::array<Tensor, 3> layer_norm_fwd(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps) {
  if (!dense_rows(x) || !vector(gamma, x.size(1), at::kBFloat16, x) || !vector(beta, x.size(1), at::kBFloat16, x) || x.size(0) > INT32_MAX ||
      x.size(1) > 32768)
    throw Refused{};
  c10::cuda::CUDAGuard guard(x.device());
  at::AutoDispatchBelowADInplaceOrView below;
  const int64_t rows = x.size(0), cols = x.size(1);
  Tensor y = new_cuda(x.sizes(), at::kBFloat16, x), mean = new_cuda({rows}, at::kFloat, x), rstd = new_cuda({rows}, at::kFloat, x);
  LayerNormNode::run(x, gamma, beta, y, mean, rstd, rows, cols, eps);
  return {y, mean, rstd};
}

// ops/kernels.py: layer_norm_bwd that adds to fp32 dgamma / dbeta -> dx
Tensor layer_norm_bwd_into(const Tensor& dy, const Tensor& x, const Tensor& gamma, const Tensor& mean, const Tensor& rstd, const Tensor& addend,
                           const Tensor& dgamma, const Tensor& dbeta) {
  if (!dense_rows(x) || !dense_rows(dy) || !dy.sizes().equals(x.sizes()) || dy.device() != x.device()) throw Refused{};
  const int64_t rows = x.size(0), cols = x.size(1);
  if (!vector(gamma, cols, at::kBFloat16, x) || !vector(mean, rows, at::kFloat, x) || !vector(rstd, rows, at::kFloat, x) ||
      !vector(dgamma, cols, at::kFloat, x) || !vector(dbeta, cols, at::kFloat, x) || rows > INT32_MAX || cols > 32768)
    throw Refused{};
  if (addend.defined() && (!dense_rows(addend) || !addend.sizes().equals(x.sizes()) || addend.device() != x.device())) throw Refused{};
  c10::cuda::CUDAGuard guard(x.device());
  at::AutoDispatchBelowADInplaceOrView below;
  Tensor dx = new_cuda(x.sizes(), at::kBFloat16, x);
  Tensor scratch = new_cuda({2 * int64_t(ofb_layer_norm_bwd_parts(static_cast<int>(rows))) * cols}, at::kFloat, x);
  if (ofb_layer_norm_bwd_to(dy.const_data_ptr(), x.const_data_ptr(), gamma.const_data_ptr(), mean.data_ptr<float>(), rstd.data_ptr<float>(),
                            addend.defined() ? addend.const_data_ptr() : nullptr, dx.mutable_data_ptr(), dgamma.mutable_data_ptr(),
                            dbeta.mutable_data_ptr(), scratch.data_ptr<float>(), 1, 0, static_cast<int>(rows), static_cast<int>(cols), stream()))
    throw Refused{};
  g_launches.fetch_add(2, std::memory_order_relaxed);
  return dx;
}

// ops/kernels.py: column_sum that adds to an fp32 vector
Tensor column_sum_into(const Tensor& x, const Tensor& out) {
  if (!dense_rows(x) || !vector(out, x.size(1), at::kFloat, x) || x.size(0) > INT32_MAX || x.size(1) > INT32_MAX) throw Refused{};
  c10::cuda::CUDAGuard guard(x.device());
  if (ofb_column_sum(x.const_data_ptr(), out.data_ptr<float>(), static_cast<int>(x.size(0)), static_cast<int>(x.size(1)), stream()))
    throw Refused{};
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return out;
}

// ------------------------------------------------------------------------------------------------ Python
Tensor arg(PyObject* o) {
  if (o == Py_None) return Tensor();
  if (!THPVariable_Check(o)) throw Refused{};
  return THPVariable_Unpack(o);
}
int64_t int_arg(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);   // bools and numpy integers included, as in Python's own index()
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    throw Refused{};
  }
  return v;
}
double float_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    throw Refused{};
  }
  return v;
}
bool bool_arg(PyObject* o) { return PyObject_IsTrue(o) == 1; }

template <int N, typename F>
PyObject* call(PyObject* const* args, Py_ssize_t n, F body) {
  HANDLE_TH_ERRORS
  if (n != N) {
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");
    return nullptr;
  }
  try {
    if (intercepted()) throw Refused{};
    return body(args);
  } catch (const Refused&) {
    Py_RETURN_NONE;
  }
  END_HANDLE_TH_ERRORS
}

template <typename F>
PyObject* without_gil(F f) {
  Tensor out;
  {
    pybind11::gil_scoped_release release;
    out = f();
  }
  return THPVariable_Wrap(std::move(out));
}

PyObject* py_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {   // x, weight, bias, act, residual
  return call<5>(args, n, [](PyObject* const* a) {
    const Tensor x = arg(a[0]), w = arg(a[1]), b = arg(a[2]), r = arg(a[4]);
    const int act = static_cast<int>(int_arg(a[3]));
    return without_gil([&] { return linear(x, w, b, r, act); });
  });
}
PyObject* py_mlp(PyObject*, PyObject* const* args, Py_ssize_t n) {      // x, w1, b1, w2, b2, act, residual
  return call<7>(args, n, [](PyObject* const* a) {
    const Tensor x = arg(a[0]), w1 = arg(a[1]), b1 = arg(a[2]), w2 = arg(a[3]), b2 = arg(a[4]), r = arg(a[6]);
    const int act = static_cast<int>(int_arg(a[5]));
    return without_gil([&] { return mlp(x, w1, b1, w2, b2, r, act); });
  });
}
PyObject* py_layer_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {   // x, weight, bias, eps
  return call<4>(args, n, [](PyObject* const* a) {
    const Tensor x = arg(a[0]), g = arg(a[1]), b = arg(a[2]);
    const double eps = float_arg(a[3]);
    return without_gil([&] { return layer_norm(x, g, b, eps); });
  });
}
PyObject* py_sdpa(PyObject*, PyObject* const* args, Py_ssize_t n) {     // query, key, value, causal, scale
  return call<5>(args, n, [](PyObject* const* a) {
    const Tensor q = arg(a[0]), k = arg(a[1]), v = arg(a[2]);
    const bool causal = bool_arg(a[3]);
    const double scale = float_arg(a[4]);
    return without_gil([&] { return sdpa(q, k, v, causal, scale); });
  });
}
PyObject* py_attention_packed(PyObject*, PyObject* const* args, Py_ssize_t n) {   // qkv, seq_len, head_size, causal, scale
  return call<5>(args, n, [](PyObject* const* a) {
    const Tensor t = arg(a[0]);
    const int64_t seq = int_arg(a[1]), D = int_arg(a[2]);
    const bool causal = bool_arg(a[3]);
    const double scale = float_arg(a[4]);
    return without_gil([&] { return attention_packed(t, seq, D, causal, scale); });
  });
}
PyObject* py_cross_entropy(PyObject*, PyObject* const* args, Py_ssize_t n) {      // logits, labels
  return call<2>(args, n, [](PyObject* const* a) {
    const Tensor x = arg(a[0]), l = arg(a[1]);
    return without_gil([&] { return cross_entropy(x, l); });
  });
}
// a, b, a_km, b_kn, bias, act, residual, aux_in, want_aux, out, out_fp32, accumulate
PyObject* py_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return call<12>(args, n, [](PyObject* const* a) -> PyObject* {
    const Tensor x = arg(a[0]), y = arg(a[1]), bias = arg(a[4]), res = arg(a[6]), aux = arg(a[7]), out = arg(a[9]);
    const bool want_aux = bool_arg(a[8]);
    auto r = gemm(x, y, bool_arg(a[2]), bool_arg(a[3]), bias, static_cast<int>(int_arg(a[5])), res, aux, want_aux, out, bool_arg(a[10]),
                  bool_arg(a[11]));
    PyObject* o;
    if (a[9] != Py_None) {
      Py_INCREF(a[9]);
      o = a[9];
    } else {
      o = THPVariable_Wrap(std::move(r.first));
    }
    if (!want_aux || !o) return o;
    PyObject* h = THPVariable_Wrap(std::move(r.second));
    PyObject* pair = h ? PyTuple_Pack(2, o, h) : nullptr;
    Py_DECREF(o);
    Py_XDECREF(h);
    return pair;
  });
}
PyObject* py_layer_norm_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {   // x, gamma, beta, eps
  return call<4>(args, n, [](PyObject* const* a) -> PyObject* {
    auto r = layer_norm_fwd(arg(a[0]), arg(a[1]), arg(a[2]), float_arg(a[3]));
    PyObject* t = PyTuple_New(3);
    for (int i = 0; t && i < 3; ++i) PyTuple_SET_ITEM(t, i, THPVariable_Wrap(std::move(r[static_cast<size_t>(i)])));
    return t;
  });
}
PyObject* py_layer_norm_bwd_into(PyObject*, PyObject* const* args, Py_ssize_t n) {   // dy, x, gamma, mean, rstd, addend, dgamma, dbeta
  return call<8>(args, n, [](PyObject* const* a) -> PyObject* {
    return THPVariable_Wrap(layer_norm_bwd_into(arg(a[0]), arg(a[1]), arg(a[2]), arg(a[3]), arg(a[4]), arg(a[5]), arg(a[6]), arg(a[7])));
  });
}
PyObject* py_column_sum_into(PyObject*, PyObject* const* args, Py_ssize_t n) {       // x, out
  return call<2>(args, n, [](PyObject* const* a) -> PyObject* {
    column_sum_into(arg(a[0]), arg(a[1]));
    Py_INCREF(a[1]);
    return a[1];
  });
}
PyObject* py_launches(PyObject*, PyObject* const*, Py_ssize_t) { return PyLong_FromLongLong(g_launches.load()); }

#define OFB_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {OFB_METHOD(linear), OFB_METHOD(mlp),  OFB_METHOD(layer_norm), OFB_METHOD(sdpa),          OFB_METHOD(attention_packed),
                         OFB_METHOD(cross_entropy), OFB_METHOD(gemm), OFB_METHOD(layer_norm_fwd), OFB_METHOD(layer_norm_bwd_into),
                         OFB_METHOD(column_sum_into), OFB_METHOD(launches), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "ofb_torch", "Fused ops of the flow API on local CUDA tensors.", -1, methods,
                      nullptr,               nullptr,     nullptr,                                             nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_ofb_torch() { return PyModule_Create(&module); }
