// Native host path of the Python entry points: argument checks, output allocation, autograd
// nodes and launches in C++ (host.cpp builds it into srwm_b200/_host.so).
//
// A training step of the small configurations is some 90 us of kernels; the same work done in
// Python (tensor checks, ctypes structures, two Python autograd nodes) took 390 us a step on a
// B200 box, and an actor's step 110 us around 6 us of kernel.  The C ABI stays the boundary: this
// file only fills its argument blocks.  Everything unusual (another device or dtype, an unaligned
// row, a state that is not dense) is declined -- the entry points return NotImplemented and the
// Python code, which raises the errors and makes the copies, takes the call.
#pragma once
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/python_variable.h>

#include "srwm_b200.h"

namespace host {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// Entry points of the loaded library, bound by name from Python (so that the debug build of the
// library is used where the Python side chose it).
#define SRWM_HOST_API(X)                                                                              \
  X(srwm_b200_srwm_layer_forward)                                                                     \
  X(srwm_b200_srwm_layer_backward)                                                                    \
  X(srwm_b200_srwm_backward_detached)                                                                 \
  X(srwm_b200_delta_forward)                                                                          \
  X(srwm_b200_delta_backward)                                                                         \
  X(srwm_b200_delta_packed_forward)                                                                   \
  X(srwm_b200_delta_packed_backward)                                                                  \
  X(srwm_b200_reduce_states)                                                                          \
  X(srwm_b200_copy_states)                                                                            \
  X(srwm_b200_gemm_scratch_bytes)                                                                     \
  X(srwm_b200_gemm_few_rows)                                                                          \
  X(srwm_b200_gemm_f32)                                                                               \
  X(srwm_b200_norm_forward)                                                                           \
  X(srwm_b200_norm_scratch_bytes)                                                                     \
  X(srwm_b200_norm_backward)                                                                          \
  X(srwm_b200_block_fits)                                                                             \
  X(srwm_b200_block_forward)

struct Api {
#define X(name) decltype(&::name) name = nullptr;
  SRWM_HOST_API(X)
#undef X
};
inline Api& api() {
  static Api a;
  return a;
}

// Raises srwm_b200._lib.SrwmError(code, what), as the Python layer does.
[[noreturn]] inline void raise_code(int code, const char* what) {
  PyGILState_STATE g = PyGILState_Ensure();
  PyObject* mod = PyImport_ImportModule("srwm_b200._lib");
  if (mod) {
    PyObject* cls = PyObject_GetAttrString(mod, "SrwmError");
    PyObject* err = cls ? PyObject_CallFunction(cls, "is", code, what) : nullptr;
    if (err) PyErr_SetObject(cls, err);
    Py_XDECREF(err);
    Py_XDECREF(cls);
    Py_DECREF(mod);
  }
  python_error e;
  e.persist();
  PyGILState_Release(g);
  throw e;
}
inline void check(int code, const char* what) {
  if (code != 0) raise_code(code, what);
}

inline bool head_dim_ok(int64_t E) { return E == 8 || E == 16 || E == 32 || E == 64; }
inline bool io_ok(const Tensor& t) {
  return t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16;
}
inline int io_code(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? SRWM_B200_BF16 : SRWM_B200_F32; }

// Innermost contiguous, every row on a 16-byte boundary (strides of size-1 dimensions ignored).
inline bool seq_ok(const Tensor& t) {
  const int64_t es = t.element_size();
  const auto sh = t.sizes();
  const auto st = t.strides();
  if (sh[3] > 1 && st[3] != 1) return false;
  if (reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16) return false;
  for (int d = 0; d < 3; ++d)
    if (sh[d] > 1 && (st[d] * es) % 16) return false;
  return true;
}
inline srwm_b200_seq seq(const Tensor& t) {
  const auto sh = t.sizes();
  const auto st = t.strides();
  return {const_cast<void*>(t.const_data_ptr()), sh[0] > 1 ? st[0] : 0, sh[1] > 1 ? st[1] : 0, sh[2] > 1 ? st[2] : 0};
}
// Dense [N,H,L,w] rows inside a buffer of saved activations.
inline srwm_b200_seq dense_seq(float* base, int64_t H, int64_t L, int64_t w) { return {base, H * L * w, L * w, w}; }

inline bool state_ok(const Tensor& t) {
  if (t.scalar_type() != at::kFloat || reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16) return false;
  const auto sh = t.sizes();
  const auto st = t.strides();
  if (st[3] != 1 || st[2] != sh[3]) return false;
  for (int d = 0; d < 2; ++d)
    if (sh[d] > 1 && (st[d] * 4) % 16) return false;
  return true;
}
inline srwm_b200_state state(const Tensor& t) {
  const auto sh = t.sizes();
  const auto st = t.strides();
  return {static_cast<float*>(const_cast<void*>(t.const_data_ptr())), sh[0] > 1 ? st[0] : 0, sh[1] > 1 ? st[1] : 0};
}
inline bool shape_is(const Tensor& t, int64_t a, int64_t b, int64_t c, int64_t d) {
  return t.dim() == 4 && t.size(0) == a && t.size(1) == b && t.size(2) == c && t.size(3) == d;
}
inline Tensor floats(const Tensor& like, at::IntArrayRef shape) {
  return at::empty(shape, like.options().dtype(at::kFloat));
}
inline Tensor state_like(const Tensor& x, int64_t N, int64_t H, int64_t E, int64_t w) { return floats(x, {N, H, E, w}); }

// Output with the memory order of the input view, optionally with another last dimension.
inline Tensor like(const Tensor& t, int64_t last) {
  if (last == t.size(3)) return at::empty_like(t);
  int order[3] = {0, 1, 2};   // outer to inner in memory
  std::stable_sort(order, order + 3, [&](int a, int b) { return t.stride(a) > t.stride(b); });
  int64_t st[4] = {0, 0, 0, 1}, run = last;
  for (int i = 2; i >= 0; --i) {
    st[order[i]] = run;
    run *= t.size(order[i]);
  }
  return at::empty_strided({t.size(0), t.size(1), t.size(2), last}, at::IntArrayRef(st, 4), t.options());
}

// Gradient of an output as rows the kernels can read.
inline Tensor grad_rows(const Tensor& g, const Tensor& x) {
  if (!g.defined()) return at::zeros_like(x);
  Tensor r = g.scalar_type() == x.scalar_type() ? g : g.to(x.scalar_type());
  return seq_ok(r) ? r : r.contiguous();
}

// Gradients, and tensors that come back from a SavedVariable (saved-tensor hooks may have replaced them: same values,
// other strides or another alignment than those the forward has checked), as the kernels can read them.
inline Tensor dense(const Tensor& t) {
  Tensor r = t.contiguous();
  return reinterpret_cast<uintptr_t>(r.const_data_ptr()) % 16 ? r.clone() : r;
}
inline Tensor saved_rows(const Tensor& t) { return seq_ok(t) ? t : dense(t); }
inline Tensor saved_state(const Tensor& t) { return state_ok(t) ? t : dense(t); }

inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

inline bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// A plain tensor argument (a tensor or parameter object, no subclass with overridden behaviour).
inline bool plain(PyObject* o) { return THPVariable_CheckExact(o); }

// Inside a level of forward-mode AD tensors may have tangents, which only torch's own operators carry on and the Python nodes
// refuse.  (Asked once per call: every tensor's own tangent is behind a lock.)
inline bool forward_ad() { return torch::autograd::ForwardADLevel::try_get_by_idx(0) != nullptr; }

}  // namespace host
