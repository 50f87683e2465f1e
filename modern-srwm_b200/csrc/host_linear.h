// The layers' linear maps and layer normalisation on this library's kernels, with autograd.
#pragma once
#include "host_common.h"

namespace host {

inline bool plain_f32(const Tensor& t) {
  return t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() &&
         reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
}

// C[M, N] = op(A) op(B)^T (+ add); dense row-major operands.
inline Tensor gemm(const Tensor& A, bool ta, const Tensor& B, bool tb, int64_t M, int64_t N, int64_t K, const Tensor& add,
                   at::IntArrayRef shape, bool relu = false) {
  Tensor C = at::empty(shape, A.options());
  srwm_b200_gemm_args a = {};
  a.A = static_cast<const float*>(A.const_data_ptr());
  a.B = static_cast<const float*>(B.const_data_ptr());
  a.C = static_cast<float*>(C.data_ptr());
  a.lda = ta ? M : K;
  a.ldb = tb ? N : K;
  a.ldc = N;
  if (add.defined()) {
    a.add = static_cast<const float*>(add.const_data_ptr());
    a.ldadd = add.dim() == 1 && A.dim() != 1 ? 0 : N;   // a bias: the same row for all
  }
  a.M = M; a.N = N; a.K = K;
  a.trans_a = ta; a.trans_b = tb;
  Tensor scratch;
  if (const size_t need = api().srwm_b200_gemm_scratch_bytes(M, N, K)) {
    scratch = at::empty({(int64_t)(need / 4)}, A.options());
    a.scratch = scratch.data_ptr();
    a.scratch_bytes = need;
  }
  a.relu = relu && api().srwm_b200_gemm_few_rows(M, N, K);
  check(api().srwm_b200_gemm_f32(&a, stream_of(A)), "gemm_f32");
  return relu && !a.relu ? C.relu_() : C;
}

// Whether the user lets fp32 products run at tf32 precision.  Under either of torch's switches: allowTF32CuBLAS(), the
// older one's query, throws once the newer (matmul.fp32_precision) has been set.
inline bool tf32_allowed() {
  return at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL) == at::Float32Precision::TF32;
}

// x [..., K], w [N, K], add undefined, [..., N] or, without gradients, a bias [N]
inline bool linear_args_ok(const Tensor& x, const Tensor& w, const Tensor& add) {
  if (!plain_f32(x) || !plain_f32(w) || x.dim() < 1 || w.dim() != 2 || w.device() != x.device()) return false;
  const int64_t K = w.size(1), N = w.size(0);
  if (x.size(-1) != K || K % 4 || N % 4 || x.numel() == 0 || w.numel() == 0 || x.numel() / K > 8000000) return false;
  if (add.defined()) {
    if (!plain_f32(add) || add.device() != x.device() || add.dim() < 1 || add.size(-1) != N) return false;
    // (the partial sums of a long product are added to a whole matrix)
    if (add.dim() == 1 && x.dim() > 1)
      return !wants_grad({&x, &w, &add}) && api().srwm_b200_gemm_scratch_bytes(x.numel() / K, N, K) == 0 &&
             !tf32_allowed();
    if (add.dim() != x.dim()) return false;
    for (int64_t d = 0; d + 1 < x.dim(); ++d)
      if (add.size(d) != x.size(d)) return false;
  }
  // (at tf32 precision the library's products are the faster ones)
  return !tf32_allowed();
}
inline Tensor linear_forward(const Tensor& x, const Tensor& w, const Tensor& add, bool relu = false) {
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t K = w.size(1), N = w.size(0);
  auto shape = x.sizes().vec();
  shape.back() = N;
  return gemm(x, false, w, false, x.numel() / K, N, K, add, shape, relu);
}

struct Linear : torch::autograd::Function<Linear> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const std::optional<Tensor>& add) {
    ctx->save_for_backward({x, w});
    ctx->saved_data["add"] = add.has_value();
    return {linear_forward(x, w, add.has_value() ? *add : Tensor())};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    c10::cuda::CUDAGuard guard(t[0].device());
    const Tensor x = dense(t[0]), w = dense(t[1]);
    const int64_t K = w.size(1), N = w.size(0), M = x.numel() / K;
    Tensor dx, dw;
    if (at::GradMode::is_enabled()) {   // create_graph: these gradients are to be differentiated again
      if (ctx->needs_input_grad(0)) dx = at::matmul(g[0], w);
      if (ctx->needs_input_grad(1)) dw = at::matmul(g[0].reshape({M, N}).t(), x.reshape({M, K}));
      return {dx, dw, ctx->saved_data["add"].toBool() ? g[0] : Tensor()};
    }
    const Tensor dy = dense(g[0]);
    if (ctx->needs_input_grad(0)) dx = gemm(dy, false, w, true, M, K, N, Tensor(), x.sizes());
    if (ctx->needs_input_grad(1)) dw = gemm(dy, true, x, true, N, K, M, Tensor(), w.sizes());
    return {dx, dw, ctx->saved_data["add"].toBool() ? g[0] : Tensor()};
  }
};

inline Tensor linear(const Tensor& x, const Tensor& w, const Tensor& add) {
  if (!wants_grad({&x, &w, &add})) return linear_forward(x, w, add);
  return Linear::apply(x, w, add.defined() ? std::optional<Tensor>(add) : std::nullopt)[0];
}

inline bool norm_args_ok(const Tensor& x, const Tensor& w, const Tensor& b) {
  if (!plain_f32(x) || !plain_f32(w) || !plain_f32(b) || x.dim() < 1 || w.dim() != 1 || b.dim() != 1) return false;
  const int64_t D = w.size(0);
  return x.size(-1) == D && b.size(0) == D && D % 4 == 0 && D <= 1024 && x.numel() > 0 && w.device() == x.device() &&
         b.device() == x.device();
}
inline Tensor norm_forward(const Tensor& x, const Tensor& w, const Tensor& b, double eps, Tensor* stats) {
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t D = w.size(0), rows = x.numel() / D;
  Tensor y = at::empty_like(x);
  float *mean = nullptr, *rstd = nullptr;
  if (stats) {
    *stats = floats(x, {2 * rows});
    mean = static_cast<float*>(stats->data_ptr());
    rstd = mean + rows;
  }
  check(api().srwm_b200_norm_forward(static_cast<const float*>(x.const_data_ptr()), static_cast<const float*>(w.const_data_ptr()),
                                     static_cast<const float*>(b.const_data_ptr()), static_cast<float*>(y.data_ptr()), mean, rstd,
                                     rows, D, (float)eps, stream_of(x)),
        "norm_forward");
  return y;
}
struct Norm : torch::autograd::Function<Norm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
    Tensor stats;
    Tensor y = norm_forward(x, w, b, eps, &stats);
    ctx->save_for_backward({x, w, b, stats});
    ctx->saved_data["eps"] = eps;
    return {y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    c10::cuda::CUDAGuard guard(t[0].device());
    const Tensor x = dense(t[0]), w = dense(t[1]), stats = dense(t[3]);
    if (at::GradMode::is_enabled()) {   // create_graph
      Tensor mean, rstd;
      {
        at::NoGradGuard no_grad;
        std::tie(std::ignore, mean, rstd) = at::native_layer_norm(x, w.sizes(), w, t[2], ctx->saved_data["eps"].toDouble());
      }
      auto r = at::native_layer_norm_backward(g[0], x, w.sizes(), mean, rstd, w, t[2], {true, true, true});
      return {std::get<0>(r), std::get<1>(r), std::get<2>(r), Tensor()};
    }
    const Tensor dy = dense(g[0]);
    const int64_t D = w.size(0), rows = x.numel() / D;
    Tensor dx = at::empty_like(x), dw = at::empty_like(w), db = at::empty_like(w);
    const int64_t need = api().srwm_b200_norm_scratch_bytes(rows, D);
    Tensor scratch = floats(x, {need / 4});
    auto f = [](const Tensor& v) { return static_cast<float*>(const_cast<void*>(v.const_data_ptr())); };
    check(api().srwm_b200_norm_backward(f(x), f(w), f(dy), f(stats), f(stats) + rows, f(dx), f(dw), f(db), rows, D,
                                        scratch.data_ptr(), need, stream_of(x)),
          "norm_backward");
    return {dx, dw, db, Tensor()};
  }
};
inline Tensor norm(const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
  if (!wants_grad({&x, &w, &b})) return norm_forward(x, w, b, eps, nullptr);
  return Norm::apply(x, w, b, eps)[0];
}

}  // namespace host
