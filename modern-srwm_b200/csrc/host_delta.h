// Delta-rule operator (fast_weight_delta) and the call on packed slow-net rows (delta_layer).
#pragma once
#include "host_srwm.h"

namespace host {

inline bool delta_args_ok(const Tensor& Q, const Tensor& K, const Tensor& V, const Tensor& beta, const Tensor& W) {
  if (!srwm_input_ok(Q)) return false;
  for (const Tensor* t : {&K, &V})
    if (t->device() != Q.device() || t->scalar_type() != Q.scalar_type() || t->sizes() != Q.sizes() || !seq_ok(*t))
      return false;
  const int64_t N = Q.size(0), H = Q.size(1), L = Q.size(2), E = Q.size(3);
  return beta.device() == Q.device() && beta.scalar_type() == Q.scalar_type() && shape_is(beta, N, H, L, 1) &&
         W.device() == Q.device() && shape_is(W, N, H, E, E) && state_ok(W);
}

// v_old and v_insert share one buffer.
inline Tensor delta_forward(const Tensor& Q, const Tensor& K, const Tensor& V, const Tensor& beta, const Tensor& W,
                            Tensor* saved) {
  int64_t N, H, L, E;
  state_dims(Q, N, H, L, E);
  c10::cuda::CUDAGuard guard(Q.device());
  Tensor out = at::empty_like(Q);
  srwm_b200_delta_fwd_args a = {};
  a.N = N; a.H = H; a.L = L; a.E = E; a.M = E;
  a.io_dtype = io_code(Q);
  a.flags = saved ? 0 : SRWM_B200_FLAG_NO_SAVE;
  a.Q = seq(Q); a.K = seq(K); a.V = seq(V); a.beta = seq(beta);
  a.W = state(W);
  a.out = seq(out);
  if (saved) {
    *saved = floats(Q, {2 * N * H * L * E});
    float* p = static_cast<float*>(saved->data_ptr());
    a.v_old = dense_seq(p, H, L, E);
    a.v_insert = dense_seq(p + N * H * L * E, H, L, E);
  }
  check(api().srwm_b200_delta_forward(&a, stream_of(Q)), "delta_forward");
  return out;
}

struct Delta : torch::autograd::Function<Delta> {
  static variable_list forward(AutogradContext* ctx, const Tensor& Q, const Tensor& K, const Tensor& V,
                               const Tensor& beta, const Tensor& W) {
    Tensor saved;
    Tensor out = delta_forward(Q, K, V, beta, W, &saved);
    ctx->save_for_backward({Q, K, V, beta, saved, W});
    ctx->set_materialize_grads(false);
    return {out};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    c10::cuda::CUDAGuard guard(t[0].device());
    const Tensor Q = saved_rows(t[0]), K = saved_rows(t[1]), V = saved_rows(t[2]), saved = dense(t[4]), W = saved_state(t[5]);
    const Tensor& beta = t[3];
    int64_t N, H, L, E;
    state_dims(Q, N, H, L, E);
    const Tensor go = grad_rows(g[0], Q);
    Tensor gQ = at::empty_like(Q), gK = at::empty_like(K), gV = at::empty_like(Q);
    Tensor gB = at::empty({N, H, L, 1}, Q.options());
    srwm_b200_delta_bwd_args a = {};
    a.N = N; a.H = H; a.L = L; a.E = E; a.M = E;
    a.io_dtype = io_code(Q);
    a.Q = seq(Q); a.K = seq(K); a.V = seq(V); a.beta = seq(beta);
    float* p = static_cast<float*>(saved.data_ptr());
    a.v_old = dense_seq(p, H, L, E);
    a.v_insert = dense_seq(p + N * H * L * E, H, L, E);
    a.grad_out = seq(go);
    a.W = state(W);
    a.grad_Q = seq(gQ); a.grad_K = seq(gK); a.grad_V = seq(gV); a.grad_beta = seq(gB);
    check(api().srwm_b200_delta_backward(&a, stream_of(Q)), "delta_backward");
    if (!W.is_same(t[5])) t[5].detach().copy_(W);   // W_0, put back where W_L was
    return {gQ, gK, gV, gB, Tensor()};
  }
};

inline bool packed_args_ok(const Tensor& x, const Tensor& W) {
  if (!x.is_cuda() || x.dim() != 4 || !io_ok(x) || x.numel() == 0 || x.stride(3) != 1) return false;
  const int64_t E = (x.size(3) - 1) / 3;
  return x.size(3) == 3 * E + 1 && head_dim_ok(E) && W.device() == x.device() &&
         shape_is(W, x.size(0), x.size(1), E, E) && state_ok(W);
}

inline Tensor packed_forward(const Tensor& x, const Tensor& W, double eps, bool zero_init, Tensor* saved) {
  const int64_t N = x.size(0), H = x.size(1), L = x.size(2), E = (x.size(3) - 1) / 3;
  c10::cuda::CUDAGuard guard(x.device());
  Tensor out = like(x, E);
  srwm_b200_delta_packed_fwd_args a = {};
  a.N = N; a.H = H; a.L = L; a.E = E;
  a.io_dtype = io_code(x);
  a.flags = (saved ? 0 : SRWM_B200_FLAG_NO_SAVE) | (zero_init ? SRWM_B200_FLAG_ZERO_INIT : 0);
  a.norm_eps = (float)eps;
  a.qkvb = seq(x);
  a.W = state(W);
  a.out = seq(out);
  if (saved) {
    *saved = floats(x, {2 * N * H * L * E});
    float* p = static_cast<float*>(saved->data_ptr());
    a.v_old = dense_seq(p, H, L, E);
    a.v_insert = dense_seq(p + N * H * L * E, H, L, E);
  }
  check(api().srwm_b200_delta_packed_forward(&a, stream_of(x)), "delta_packed_forward");
  return out;
}

struct DeltaLayer : torch::autograd::Function<DeltaLayer> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& W, double eps, bool zero_init) {
    Tensor saved;
    Tensor out = packed_forward(x, W, eps, zero_init, &saved);
    ctx->save_for_backward({x, saved, W});
    ctx->saved_data["eps"] = eps;
    ctx->set_materialize_grads(false);
    return {out};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    c10::cuda::CUDAGuard guard(t[0].device());
    const Tensor x = t[0].stride(3) == 1 ? t[0] : t[0].contiguous(), saved = dense(t[1]), W = saved_state(t[2]);
    const int64_t N = x.size(0), H = x.size(1), L = x.size(2), E = (x.size(3) - 1) / 3;
    Tensor go;
    if (g[0].defined()) {
      go = g[0].scalar_type() == x.scalar_type() ? g[0] : g[0].to(x.scalar_type());
      if (!seq_ok(go)) go = go.contiguous();
    } else {
      go = at::zeros({N, H, L, E}, x.options());
    }
    Tensor gx = at::empty_like(x);
    srwm_b200_delta_packed_bwd_args a = {};
    a.N = N; a.H = H; a.L = L; a.E = E;
    a.io_dtype = io_code(x);
    a.norm_eps = (float)ctx->saved_data["eps"].toDouble();
    a.qkvb = seq(x);
    float* p = static_cast<float*>(saved.data_ptr());
    a.v_old = dense_seq(p, H, L, E);
    a.v_insert = dense_seq(p + N * H * L * E, H, L, E);
    a.grad_out = seq(go);
    a.W = state(W);
    a.grad_qkvb = seq(gx);
    check(api().srwm_b200_delta_packed_backward(&a, stream_of(x)), "delta_packed_backward");
    if (!W.is_same(t[2])) t[2].detach().copy_(W);
    return {gx, Tensor(), Tensor(), Tensor()};
  }
};

}  // namespace host
