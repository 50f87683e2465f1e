// The agents' layers as one call: what SRlayer / FastFFlayer do around the recurrence in
// Python (views, module calls, one call per kernel) took 20 of an actor step's 31 us.
#pragma once
#include "host_delta.h"
#include "host_linear.h"

namespace host {

// h [L, B, H d], weights [1, H, d, .], state four [B, H, d, .], out_w [in, H d] with in == H d
inline bool sr_step_ok(const Tensor& h, const Four& base, const Four& state, const Tensor& out_w) {
  return plain_f32(h) && h.dim() == 3 && h.numel() > 0 && base[0].dim() == 4 && state[0].defined() && out_w.dim() == 2 &&
         h.size(2) == base[0].size(1) * base[0].size(2) && out_w.size(0) == h.size(2);
}
inline Tensor heads(const Tensor& h, int64_t H, int64_t w) {   // [L, B, H w] -> the [B, H, L, w] view
  const int64_t L = h.size(0), B = h.size(1);
  return h.as_strided({B, H, L, w}, {H * w, w, B * H * w, 1});
}
inline Tensor merged(const Tensor& out, const Tensor& h) { return out.as_strided(h.sizes(), h.strides()); }   // and back

// What the recurrence of an unroll has put out, as a node of h and W_y once more: in the backward of SrUnroll under
// create_graph, whose gradient of the projection's weight depends on them through it.
struct SrUnrolled : torch::autograd::Function<SrUnrolled> {
  static variable_list forward(AutogradContext* ctx, const Tensor& h, const Tensor& W_y, const Tensor& s_y, const Tensor& done,
                               const Tensor& saved, const Tensor& m) {
    ctx->save_for_backward({h, saved, W_y, s_y, done});
    return {m.clone()};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    c10::cuda::CUDAGuard guard(t[0].device());
    const Tensor h = dense(t[0]), &W_y = t[2];
    const int64_t H = W_y.size(1), d = W_y.size(2);
    Tensor gW;
    const Tensor gx = SrwmLayer::detached(heads(h, H, d), t[1], heads(dense(g[0]), H, d), W_y, t[3], t[4], true, &gW);
    return {merged(gx, h), batch_sum(gW, W_y.size(0)), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// The learner's unroll with gradients: heads, recurrence, output projection and residual as one node.  As the parts'
// ten nodes (views, their inverses, sums) it took 250 us of host time around 150 us of kernels.
// (done is a tensor: an absent optional would have no edge, and the weight's would not be the tenth.)
struct SrUnroll : torch::autograd::Function<SrUnroll> {
  static variable_list forward(AutogradContext* ctx, const Tensor& h, const Tensor& W_y, const Tensor& W_q, const Tensor& W_k,
                               const Tensor& w_b, const Tensor& s_y, const Tensor& s_q, const Tensor& s_k, const Tensor& s_b,
                               const Tensor& done, const Tensor& out_w) {
    const Four base = {W_y, W_q, W_k, w_b}, shift = {s_y, s_q, s_k, s_b};
    const Tensor x = heads(h, W_y.size(1), W_y.size(2));
    Four so;
    for (int z = 0; z < 4; ++z) so[z] = state_like(x, x.size(0), x.size(1), x.size(3), z < 3 ? x.size(3) : 4);
    Tensor saved;
    const Tensor m = merged(srwm_forward(x, so, &base, &shift, done, true, &saved), h);
    ctx->set_materialize_grads(false);
    ctx->mark_non_differentiable({so[0], so[1], so[2], so[3]});
    for (int z = 0; z < 4; ++z) ctx->saved_data[std::string(1, (char)('0' + z))] = base[z].size(0);
    ctx->save_for_backward({h, saved, W_y, s_y, m, out_w, done});
    return {linear_forward(m, out_w, h), so[0], so[1], so[2], so[3]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    variable_list r(11);
    if (!g[0].defined()) return r;
    const auto t = ctx->get_saved_variables();
    c10::cuda::CUDAGuard guard(t[0].device());
    const Tensor h = dense(t[0]), m = dense(t[4]), out_w = dense(t[5]), &W_y = t[2];
    const bool again = at::GradMode::is_enabled();   // create_graph (the recurrence's own gradients are not differentiated again)
    const Tensor dy = dense(g[0]);
    const int64_t K = out_w.size(1), N = out_w.size(0), M = h.numel() / K;
    if (ctx->needs_input_grad(10)) {
      if (again) {
        const Tensor mm = SrUnrolled::apply(h, W_y, t[3], t[6], t[1], m)[0];
        r[10] = at::matmul(dy.reshape({M, N}).t(), mm.reshape({M, K}));
      } else {
        r[10] = gemm(dy, true, m, true, N, K, M, Tensor(), out_w.sizes());
      }
    }
    std::array<int64_t, 4> base_n;
    std::array<bool, 4> need;
    for (int z = 0; z < 4; ++z) {
      base_n[z] = ctx->saved_data[std::string(1, (char)('0' + z))].toInt();
      need[z] = ctx->needs_input_grad(1 + z);
    }
    if (!ctx->needs_input_grad(0) && !need[0] && !need[1] && !need[2] && !need[3]) return r;
    const int64_t H = W_y.size(1), d = W_y.size(2);
    const Tensor x = heads(h, H, d);
    at::AutoGradMode off(false);
    const Tensor dm = gemm(dy, false, out_w, true, M, K, N, Tensor(), h.sizes());
    Tensor gW;
    const Tensor gx = SrwmLayer::detached(x, t[1], heads(dm, H, d), W_y, t[3], t[6], true, &gW);
    if (ctx->needs_input_grad(0)) {
      at::AutoGradMode on(again);
      r[0] = again ? merged(gx, h) + dy : merged(gx, h).add_(dy);
    }
    const Four slow = detached_slow(gW, base_n, need);
    for (int z = 0; z < 4; ++z) r[1 + z] = slow[z];
    return r;
  }
};

// One SRWM layer step (no gradients) or detached unroll, done undefined or [L, B].  (out, four states), or nothing where
// the parts decline.
inline variable_list sr_step(const Tensor& h, const Four& base, const Four& state, const Tensor& done, const Tensor& out_w) {
  const int64_t H = base[0].size(1), d = base[0].size(2);
  const Tensor x = heads(h.detach(), H, d);
  const Tensor dn = done.defined() && done.dim() == 2 ? done.t() : done;
  if (!layer_args_ok(x, base, state, dn) || !linear_args_ok(h, out_w, h)) return {};
  if (wants_grad({&h, &base[0], &base[1], &base[2], &base[3], &state[0], &state[1], &state[2], &state[3], &out_w}))
    return SrUnroll::apply(h, base[0], base[1], base[2], base[3], state[0], state[1], state[2], state[3], dn, out_w);
  Four so;
  for (int z = 0; z < 4; ++z) so[z] = state_like(x, x.size(0), H, d, z < 3 ? d : 4);
  const Tensor out = srwm_forward(x, so, &base, &state, dn, true, nullptr);
  // the output follows the view's memory order: it is [L, B, H d] as it lies
  return {linear_forward(merged(out, h), out_w, h), so[0], so[1], so[2], so[3]};
}

// x [L, B, in]; the layer norm's weight and bias, the slow net's rows, fast weights W [B, H, d, d] (left final), out_w.
// (out, a copy of the final W unless it started from zero), or nothing
inline variable_list ff_step(const Tensor& x, const Tensor& lw, const Tensor& lb, double ln_eps, const Tensor& slow_w, const Tensor& W,
                      double norm_eps, bool zero_init, const Tensor& out_w) {
  if (!plain_f32(x) || x.dim() != 3 || x.numel() == 0 || W.dim() != 4 || slow_w.dim() != 2 || out_w.dim() != 2 ||
      !norm_args_ok(x, lw, lb) || !linear_args_ok(x, slow_w, Tensor()))
    return {};
  const int64_t H = W.size(1), d = W.size(2), L = x.size(0), B = x.size(1);
  if (slow_w.size(0) != H * (3 * d + 1) || out_w.size(1) != H * d || out_w.size(0) != x.size(2) || W.size(0) != B ||
      W.device() != x.device() ||
      out_w.device() != x.device() || !head_dim_ok(d) || !state_ok(W) || !plain_f32(out_w) || (H * d) % 4 || x.size(2) % 4)
    return {};
  const Tensor rows = linear_forward(norm_forward(x, lw, lb, ln_eps, nullptr), slow_w, Tensor());
  const Tensor view = heads(rows, H, 3 * d + 1);
  if (!packed_args_ok(view, W)) return {};
  const Tensor out = packed_forward(view, W, norm_eps, zero_init, nullptr);   // laid out [L, B, H, d]
  const Tensor y = linear_forward(out.as_strided({L, B, H * d}, {B * H * d, H * d, 1}), out_w, x);
  if (zero_init) return {y, Tensor()};
  Tensor copy;   // the state handed back (a kernel of ours: a library copy takes the host 3 us longer)
  if (W.is_contiguous()) {
    c10::cuda::CUDAGuard guard(W.device());
    copy = state_like(W, B, H, d, d);
    copy_states({W, Tensor(), Tensor(), Tensor()}, {copy, Tensor(), Tensor(), Tensor()});
  } else {
    copy = W.clone();
  }
  return {y, copy};
}

// What follows the recurrence in an agent's block (no gradients): att [.., K0], the residual h [.., D], the projection's weight, the
// norm's weight and bias, weights and biases of the feed-forward part.  Undefined where the one kernel does not apply.
inline Tensor block_tail(const Tensor& att, const Tensor& h, const Tensor& wo, const Tensor& gamma, const Tensor& beta, double eps,
                         const Tensor& w1, const Tensor& b1, const Tensor& w2, const Tensor& b2) {
  if (!linear_args_ok(att, wo, h) || !norm_args_ok(h, gamma, beta) || w1.dim() != 2 || w2.dim() != 2 || !plain_f32(w1) ||
      !plain_f32(w2) || w1.device() != h.device() || w2.device() != h.device())
    return Tensor();
  const int64_t K0 = wo.size(1), D = wo.size(0), F = w1.size(0), N = w2.size(0), rows = h.numel() / D;
  auto bias_ok = [&](const Tensor& b, int64_t n) {
    return !b.defined() || (plain_f32(b) && b.device() == h.device() && b.dim() == 1 && b.size(0) == n);
  };
  if (w1.size(1) != D || w2.size(1) != F || !bias_ok(b1, F) || !bias_ok(b2, N) || rows > 65536 || K0 > 65536 || D > 65536 ||
      F > 65536 || N > 65536 || !api().srwm_b200_block_fits(rows, K0, D, F, N))
    return Tensor();
  c10::cuda::CUDAGuard guard(h.device());
  auto shape = h.sizes().vec();
  shape.back() = N;
  Tensor y = at::empty(shape, h.options());
  auto in = [](const Tensor& t) { return t.defined() ? static_cast<const float*>(t.const_data_ptr()) : nullptr; };
  srwm_b200_block_args a = {};
  a.att = in(att); a.res = in(h); a.wo = in(wo); a.gamma = in(gamma); a.beta = in(beta);
  a.w1 = in(w1); a.b1 = in(b1); a.w2 = in(w2); a.b2 = in(b2);
  a.y = static_cast<float*>(y.data_ptr());
  a.rows = rows; a.K0 = K0; a.D = D; a.F = F; a.N = N;
  a.eps = eps;
  check(api().srwm_b200_block_forward(&a, stream_of(h)), "block_forward");
  return y;
}

}  // namespace host
