// SRWM operators and the layer-level call: raw calls on tensors and their autograd nodes.
#pragma once
#include "host_common.h"

namespace host {

// The seven saved tensors of a forward share one buffer: q, k, y_diff, q_diff, k_diff, beta, beta_diff.
struct Saved {
  srwm_b200_seq q, k, yd, qd, kd, beta, bd;
};
inline Tensor saved_buffer(const Tensor& x, int64_t rows, int64_t E) { return floats(x, {rows * (5 * E + 8)}); }
inline Saved saved_views(const Tensor& buf, int64_t N, int64_t H, int64_t L, int64_t E) {
  float* p = static_cast<float*>(buf.data_ptr());
  const int64_t rows = N * H * L, b = rows * E;
  return {dense_seq(p, H, L, E),         dense_seq(p + b, H, L, E),     dense_seq(p + 2 * b, H, L, E),
          dense_seq(p + 3 * b, H, L, E), dense_seq(p + 4 * b, H, L, E), dense_seq(p + 5 * b, H, L, 4),
          dense_seq(p + 5 * b + rows * 4, H, L, 4)};
}

using Four = std::array<Tensor, 4>;

inline bool srwm_input_ok(const Tensor& x) {
  return x.is_cuda() && x.dim() == 4 && io_ok(x) && head_dim_ok(x.size(3)) && x.numel() > 0 && seq_ok(x);
}

inline void state_dims(const Tensor& x, int64_t& N, int64_t& H, int64_t& L, int64_t& E) {
  N = x.size(0); H = x.size(1); L = x.size(2); E = x.size(3);
}

// Forward; W: final state out (and in, without `base`).  base / shift / done as in the C ABI's extension block.
inline Tensor srwm_forward(const Tensor& x, const Four& W, const Four* base, const Four* shift, const Tensor& done,
                           bool input_softmax, Tensor* saved) {
  int64_t N, H, L, E;
  state_dims(x, N, H, L, E);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor out = at::empty_like(x);
  srwm_b200_srwm_fwd_args a = {};
  a.N = N; a.H = H; a.L = L; a.E = E;
  a.io_dtype = io_code(x);
  a.flags = (saved ? 0 : SRWM_B200_FLAG_NO_SAVE) | (input_softmax ? SRWM_B200_FLAG_INPUT_SOFTMAX : 0);
  a.x = seq(x);
  a.W_y = state(W[0]); a.W_q = state(W[1]); a.W_k = state(W[2]); a.w_b = state(W[3]);
  a.out = seq(out);
  if (saved) {
    *saved = saved_buffer(x, N * H * L, E);
    const Saved s = saved_views(*saved, N, H, L, E);
    a.q = s.q; a.k = s.k; a.beta = s.beta; a.y_diff = s.yd; a.q_diff = s.qd; a.k_diff = s.kd; a.beta_diff = s.bd;
  }
  srwm_b200_srwm_ext e = {};
  if (base) {
    e.base_W_y = state((*base)[0]); e.base_W_q = state((*base)[1]); e.base_W_k = state((*base)[2]);
    e.base_w_b = state((*base)[3]);
    if (shift) {
      e.shift_W_y = state((*shift)[0]); e.shift_W_q = state((*shift)[1]); e.shift_W_k = state((*shift)[2]);
      e.shift_w_b = state((*shift)[3]);
    }
    if (done.defined()) {
      e.done = static_cast<const uint8_t*>(done.const_data_ptr());
      e.done_stride_n = done.stride(0);
      e.done_stride_l = done.stride(1);
    }
  }
  check(api().srwm_b200_srwm_layer_forward(&a, base ? &e : nullptr, stream_of(x)),
        base ? "srwm_layer_forward" : "srwm_forward");
  return out;
}

// dst (dense) = src, zeros where a source is undefined
inline void copy_states(const Four& src, const Four& dst) {
  srwm_b200_state from[4] = {};
  Four keep;
  float* to[4];
  int64_t N = 0, H = 0, E = 0;
  const Tensor* any = nullptr;
  for (int z = 0; z < 4; ++z) {
    to[z] = dst[z].defined() ? static_cast<float*>(dst[z].data_ptr()) : nullptr;
    if (!to[z]) continue;
    any = &dst[z];
    N = any->size(0); H = any->size(1); E = any->size(2);
    if (!src[z].defined()) continue;
    keep[z] = src[z];
    if (!state_ok(keep[z])) keep[z] = at::empty_like(dst[z]).copy_(keep[z]);
    from[z] = state(keep[z]);
  }
  if (any) check(api().srwm_b200_copy_states(from, to, N, H, E, stream_of(*any)), "copy_states");
}

// Backward through time; W: W_L (or the final shift, with `base`), left unchanged.  gout_state: dL/dW_L,
// undefined where there is none.  Returns (grad_x, per-sample dL/dW_0 x 4).
inline std::array<Tensor, 5> srwm_backward(const Tensor& x_, const Tensor& saved_, const Tensor& grad_out, const Four& W_,
                                           const Four* base_, const Four& gout_state, bool input_softmax) {
  c10::cuda::CUDAGuard guard(x_.device());
  const Tensor x = saved_rows(x_), saved = dense(saved_);
  Four W, base;
  for (int z = 0; z < 4; ++z) {
    W[z] = saved_state(W_[z]);
    if (base_) base[z] = saved_state((*base_)[z]);
  }
  int64_t N, H, L, E;
  state_dims(x, N, H, L, E);
  const Tensor go = grad_rows(grad_out, x);
  std::array<Tensor, 5> r;
  r[0] = at::empty_like(x);
  bool any = false;
  for (const Tensor& g : gout_state) any = any || g.defined();
  for (int z = 0; z < 4; ++z) r[1 + z] = state_like(x, N, H, E, z < 3 ? E : 4);
  if (any) copy_states(gout_state, {r[1], r[2], r[3], r[4]});
  srwm_b200_srwm_bwd_args a = {};
  a.N = N; a.H = H; a.L = L; a.E = E;
  a.io_dtype = io_code(x);
  a.flags = (any ? SRWM_B200_FLAG_STATE_GRAD_IN : 0) | (input_softmax ? SRWM_B200_FLAG_INPUT_SOFTMAX : 0);
  const Saved s = saved_views(saved, N, H, L, E);
  a.x = seq(x);
  a.q = s.q; a.k = s.k; a.beta = s.beta; a.y_diff = s.yd; a.q_diff = s.qd; a.k_diff = s.kd; a.beta_diff = s.bd;
  a.grad_out = seq(go);
  a.W_y = state(W[0]); a.W_q = state(W[1]); a.W_k = state(W[2]); a.w_b = state(W[3]);
  a.grad_x = seq(r[0]);
  a.grad_W_y = state(r[1]); a.grad_W_q = state(r[2]); a.grad_W_k = state(r[3]); a.grad_w_b = state(r[4]);
  srwm_b200_srwm_ext e = {};
  if (base_) {
    e.base_W_y = state(base[0]); e.base_W_q = state(base[1]); e.base_W_k = state(base[2]); e.base_w_b = state(base[3]);
  }
  check(api().srwm_b200_srwm_layer_backward(&a, base_ ? &e : nullptr, stream_of(x)),
        base_ ? "srwm_layer_backward" : "srwm_backward");
  return r;
}

// ---- operator form (self_ref_v0 / stateful_self_ref_v0) --------------------------------------
struct SelfRef : torch::autograd::Function<SelfRef> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& W_y, const Tensor& W_q,
                               const Tensor& W_k, const Tensor& w_b, bool stateful) {
    Tensor saved;
    Tensor out = srwm_forward(x, {W_y, W_q, W_k, w_b}, nullptr, nullptr, Tensor(), false, &saved);
    ctx->save_for_backward({x, saved, W_y, W_q, W_k, w_b});
    ctx->set_materialize_grads(false);
    if (stateful) return {out, W_y, W_q, W_k, w_b};
    return {out};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    Four gs;
    for (size_t z = 1; z < g.size(); ++z) gs[z - 1] = g[z];
    auto r = srwm_backward(t[0], t[1], g[0], {t[2], t[3], t[4], t[5]}, nullptr, gs, false);
    return {r[0], r[1], r[2], r[3], r[4], Tensor()};
  }
};

inline bool operator_args_ok(const Tensor& x, const Four& W) {
  if (!srwm_input_ok(x)) return false;
  const int64_t N = x.size(0), H = x.size(1), E = x.size(3);
  for (int z = 0; z < 4; ++z)
    if (W[z].device() != x.device() || !shape_is(W[z], N, H, E, z < 3 ? E : 4) || !state_ok(W[z])) return false;
  return true;
}

// ---- layer-level form (srwm_layer) ------------------------------------------------------------
// Gradients of the slow weights from the per-sample ones: batch sums where a weight is un-repeated
// ([1,H,E,.]), minus the batch sums of the incoming dL/dshift_out (shift_out = W_L - base).
inline Four slow_gradients(const Four& g, const Four& gshift, const std::array<int64_t, 4>& base_n,
                           const std::array<bool, 4>& need) {
  const int64_t N = g[0].size(0), H = g[0].size(1), E = g[0].size(2);
  Four r;
  srwm_b200_state src[4] = {}, sub[4] = {};
  float* dst[4] = {};
  bool launch = false;
  for (int z = 0; z < 4; ++z) {
    if (!need[z]) continue;
    Tensor gs = gshift[z];
    if (gs.defined() && !state_ok(gs)) gs = gs.to(at::kFloat).contiguous();
    if (base_n[z] == N) {   // per-sample weights, or a batch of one
      r[z] = gs.defined() ? g[z] - gs : g[z];
      continue;
    }
    r[z] = state_like(g[z], 1, H, E, g[z].size(3));
    src[z] = state(g[z]);
    if (gs.defined()) sub[z] = state(gs);
    dst[z] = static_cast<float*>(r[z].data_ptr());
    launch = true;
  }
  if (launch) {
    c10::cuda::CUDAGuard guard(g[0].device());
    check(api().srwm_b200_reduce_states(src, sub, dst, N, H, E, stream_of(g[0])), "reduce_states");
  }
  return r;
}

inline Tensor batch_sum(const Tensor& g, int64_t base_n) {   // of one [N,H,E,E] gradient
  if (base_n == g.size(0)) return g;
  Four gs, none;
  gs[0] = g;
  return slow_gradients(gs, none, {base_n, 0, 0, 0}, {true, false, false, false})[0];
}

// Gradients of the slow weights where the state is detached: W_y's, and zeros for the other three, to which the
// detached state passes none.
inline Four detached_slow(const Tensor& gW, const std::array<int64_t, 4>& base_n, const std::array<bool, 4>& need) {
  const int64_t H = gW.size(1), E = gW.size(2);
  Four r, none, same;   // `same`: those of one launch
  if (need[0]) r[0] = batch_sum(gW, base_n[0]);
  int64_t n = 0;
  for (int z = 1; z < 4; ++z) {
    if (!need[z]) continue;
    r[z] = state_like(gW, base_n[z], H, E, z < 3 ? E : 4);
    if (n == 0) n = base_n[z];
    if (base_n[z] == n) same[z] = r[z];
    else r[z].zero_();
  }
  if (n) {
    c10::cuda::CUDAGuard guard(gW.device());
    copy_states(none, same);
  }
  return r;
}

struct SrwmLayer : torch::autograd::Function<SrwmLayer> {
  using Opt = std::optional<Tensor>;
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& W_y, const Tensor& W_q,
                               const Tensor& W_k, const Tensor& w_b, const Opt& s_y, const Opt& s_q, const Opt& s_k,
                               const Opt& s_b, const Opt& done, bool input_softmax, bool detach) {
    const Four base = {W_y, W_q, W_k, w_b};
    const int64_t N = x.size(0), H = x.size(1), E = x.size(3);
    const bool has_shift = s_y.has_value(), has_done = done.has_value();
    Four shift, shift_out;
    if (has_shift) shift = {*s_y, *s_q, *s_k, *s_b};
    for (int z = 0; z < 4; ++z) shift_out[z] = state_like(x, N, H, E, z < 3 ? E : 4);
    Tensor saved;
    Tensor out = srwm_forward(x, shift_out, &base, has_shift ? &shift : nullptr, has_done ? *done : Tensor(),
                              input_softmax, &saved);
    ctx->set_materialize_grads(false);
    ctx->saved_data["softmax"] = input_softmax;
    ctx->saved_data["detach"] = detach;
    ctx->saved_data["shift"] = has_shift;
    ctx->saved_data["done"] = has_done;
    if (detach) {
      variable_list keep = {x, saved, W_y, W_q, W_k, w_b};
      if (has_shift) keep.push_back(shift[0]);
      if (has_done) keep.push_back(*done);
      ctx->save_for_backward(std::move(keep));
      ctx->mark_non_differentiable({shift_out[0], shift_out[1], shift_out[2], shift_out[3]});
    } else {
      ctx->save_for_backward({x, saved, W_y, W_q, W_k, w_b, shift_out[0], shift_out[1], shift_out[2], shift_out[3]});
    }
    return {out, shift_out[0], shift_out[1], shift_out[2], shift_out[3]};
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    const bool softmax = ctx->saved_data["softmax"].toBool(), detach = ctx->saved_data["detach"].toBool();
    const bool has_shift = ctx->saved_data["shift"].toBool(), has_done = ctx->saved_data["done"].toBool();
    const Tensor& x = t[0];
    const Four base = {t[2], t[3], t[4], t[5]};
    variable_list r(12);
    std::array<int64_t, 4> base_n;
    std::array<bool, 4> need;
    for (int z = 0; z < 4; ++z) {
      base_n[z] = base[z].size(0);
      need[z] = ctx->needs_input_grad(1 + z);
    }
    if (detach) {
      const Tensor shift = has_shift ? t[6] : Tensor();
      const Tensor done = has_done ? t[6 + (has_shift ? 1 : 0)] : Tensor();
      Tensor gW;
      r[0] = detached(x, t[1], g[0], base[0], shift, done, softmax, &gW);
      const Four slow = detached_slow(gW, base_n, need);
      for (int z = 0; z < 4; ++z) r[1 + z] = slow[z];
      return r;
    }
    const Four gshift = {g[1], g[2], g[3], g[4]};
    auto b = srwm_backward(x, t[1], g[0], {t[6], t[7], t[8], t[9]}, &base, gshift, softmax);
    r[0] = b[0];
    const Four per_sample = {b[1], b[2], b[3], b[4]};
    const Four slow = slow_gradients(per_sample, gshift, base_n, need);
    for (int z = 0; z < 4; ++z) {
      r[1 + z] = has_shift && slow[z].is_same(per_sample[z]) ? slow[z].clone() : slow[z];
      if (has_shift) r[5 + z] = per_sample[z];
    }
    return r;
  }

  static Tensor detached(const Tensor& x_, const Tensor& saved_, const Tensor& grad_out, const Tensor& base_,
                         const Tensor& shift_, const Tensor& done, bool softmax, Tensor* gW) {
    c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = saved_rows(x_), saved = dense(saved_), base_Wy = saved_state(base_);
    const Tensor shift_Wy = shift_.defined() ? saved_state(shift_) : shift_;
    int64_t N, H, L, E;
    state_dims(x, N, H, L, E);
    const Tensor go = grad_rows(grad_out, x);
    Tensor gx = at::empty_like(x);
    *gW = state_like(x, N, H, E, E);
    const Saved s = saved_views(saved, N, H, L, E);
    srwm_b200_srwm_bwd_detached_args a = {};
    a.N = N; a.H = H; a.L = L; a.E = E;
    a.io_dtype = io_code(x);
    a.flags = softmax ? SRWM_B200_FLAG_INPUT_SOFTMAX : 0;
    a.x = seq(x);
    a.k = s.k; a.beta = s.beta; a.y_diff = s.yd;
    a.grad_out = seq(go);
    a.base_W_y = state(base_Wy);
    if (shift_Wy.defined()) a.shift_W_y = state(shift_Wy);
    if (done.defined()) {
      a.done = static_cast<const uint8_t*>(done.const_data_ptr());
      a.done_stride_n = done.stride(0);
      a.done_stride_l = done.stride(1);
    }
    a.grad_x = seq(gx);
    a.grad_W_y = state(*gW);
    check(api().srwm_b200_srwm_backward_detached(&a, stream_of(x)), "srwm_backward_detached");
    return gx;
  }
};

// shift: four tensors or four undefined ones; done: undefined, or bytes / bools [N, L]
inline bool layer_args_ok(const Tensor& x, const Four& base, const Four& shift, const Tensor& done) {
  if (!srwm_input_ok(x)) return false;
  const int64_t N = x.size(0), H = x.size(1), E = x.size(3);
  for (int z = 0; z < 4; ++z) {
    const int64_t w = z < 3 ? E : 4, n = base[z].dim() == 4 ? base[z].size(0) : -1;
    if (base[z].device() != x.device() || (n != 1 && n != N) || !shape_is(base[z], n, H, E, w) || !state_ok(base[z]))
      return false;
    if (shift[0].defined() != shift[z].defined()) return false;
    if (shift[z].defined() &&
        (shift[z].device() != x.device() || !shape_is(shift[z], N, H, E, w) || !state_ok(shift[z])))
      return false;
  }
  if (done.defined() && (done.device() != x.device() || done.dim() != 2 || done.size(0) != N ||
                         done.size(1) != x.size(2) || done.element_size() != 1 ||
                         (done.scalar_type() != at::kBool && done.scalar_type() != at::kByte)))
    return false;
  return true;
}

// (out, four shifts), with autograd where something wants a gradient
inline variable_list srwm_layer(const Tensor& x, const Four& base, const Four& shift, const Tensor& done,
                                bool input_softmax, bool detach) {
  const bool has_shift = shift[0].defined();
  if (!wants_grad({&x, &base[0], &base[1], &base[2], &base[3], &shift[0], &shift[1], &shift[2], &shift[3]})) {
    Four so;
    for (int z = 0; z < 4; ++z) so[z] = state_like(x, x.size(0), x.size(1), x.size(3), z < 3 ? x.size(3) : 4);
    Tensor out = srwm_forward(x, so, &base, has_shift ? &shift : nullptr, done, input_softmax, nullptr);
    return {out, so[0], so[1], so[2], so[3]};
  }
  auto opt = [](const Tensor& t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; };
  return SrwmLayer::apply(x, base[0], base[1], base[2], base[3], opt(shift[0]), opt(shift[1]), opt(shift[2]),
                          opt(shift[3]), opt(done), input_softmax, detach);
}

}  // namespace host
