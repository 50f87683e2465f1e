// The agents' layer steps without gradients as one call: what SRlayer / FastFFlayer do around the recurrence in
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
// (out, four states), or nothing where the parts decline
inline variable_list sr_step(const Tensor& h, const Four& base, const Four& state, const Tensor& out_w) {
  const int64_t H = base[0].size(1), d = base[0].size(2);
  const Tensor x = heads(h, H, d);
  if (!layer_args_ok(x, base, state, Tensor())) return {};
  if (!linear_args_ok(h, out_w, h)) return {};
  variable_list r = srwm_layer(x, base, state, Tensor(), true, false);
  // the output follows the view's memory order: it is [L, B, H d] as it lies
  const Tensor merged = r[0].as_strided(h.sizes(), h.strides());
  r[0] = linear_forward(merged, out_w, h);
  return r;
}

// x [L, B, in]; the layer norm's weight and bias, the slow net's rows, fast weights W [B, H, d, d] (left final), out_w
inline Tensor ff_step(const Tensor& x, const Tensor& lw, const Tensor& lb, double ln_eps, const Tensor& slow_w, const Tensor& W,
                      double norm_eps, bool zero_init, const Tensor& out_w) {
  if (!plain_f32(x) || x.dim() != 3 || x.numel() == 0 || W.dim() != 4 || slow_w.dim() != 2 || out_w.dim() != 2 ||
      !norm_args_ok(x, lw, lb) || !linear_args_ok(x, slow_w, Tensor()))
    return Tensor();
  const int64_t H = W.size(1), d = W.size(2), L = x.size(0), B = x.size(1);
  if (slow_w.size(0) != H * (3 * d + 1) || out_w.size(1) != H * d || out_w.size(0) != x.size(2) || W.size(0) != B ||
      W.device() != x.device() ||
      out_w.device() != x.device() || !head_dim_ok(d) || !state_ok(W) || !plain_f32(out_w) || (H * d) % 4 || x.size(2) % 4)
    return Tensor();
  const Tensor rows = linear_forward(norm_forward(x, lw, lb, ln_eps, nullptr), slow_w, Tensor());
  const Tensor view = heads(rows, H, 3 * d + 1);
  if (!packed_args_ok(view, W)) return Tensor();
  const Tensor out = packed_forward(view, W, norm_eps, zero_init, nullptr);   // laid out [L, B, H, d]
  return linear_forward(out.as_strided({L, B, H * d}, {B * H * d, H * d, 1}), out_w, x);
}

}  // namespace host
