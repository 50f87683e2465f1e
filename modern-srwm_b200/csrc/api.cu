// C ABI of libsrwm_b200.so (see include/srwm_b200.h): argument validation, conversion of
// element strides to the kernels' byte strides, dispatch to the compiled configuration.
// All validation happens before the first CUDA call.
#include "srwm_b200.h"

#include "configs.h"
#include "block.h"
#include "gemm.h"
#include "launch.h"
#include "norm.h"

#ifdef SRWM_DEBUG_CHECKS
// Status word of the debug build's row checks (common.cuh::bad_rows), one per device.
__device__ unsigned long long g_debug_status = 0ull;
#endif

namespace {

thread_local int g_last_cuda_error = 0;

// Device address of the status word (debug build), null in the ordinary build.
inline unsigned long long* debug_word() {
#ifdef SRWM_DEBUG_CHECKS
  unsigned long long* ptr = nullptr;
  if (cudaGetSymbolAddress((void**)&ptr, g_debug_status) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  return ptr;
#else
  return nullptr;
#endif
}

inline int esize(int dtype) { return dtype == SRWM_B200_BF16 ? 2 : 4; }

inline bool head_dim_ok(int E) { return E == 8 || E == 16 || E == 32 || E == 64; }

// Every row of a streamed tensor must start on a 16-byte boundary.
inline bool seq_aligned(const srwm_b200_seq& t, int es) {
  return ((uintptr_t)t.data % 16 == 0) && ((t.stride_n * es) % 16 == 0) && ((t.stride_h * es) % 16 == 0) &&
         ((t.stride_l * es) % 16 == 0);
}
inline bool state_aligned(const srwm_b200_state& t) {
  return ((uintptr_t)t.data % 16 == 0) && ((t.stride_n * 4) % 16 == 0) && ((t.stride_h * 4) % 16 == 0);
}
inline srwm::SeqView view(const srwm_b200_seq& t, int es) {
  srwm::SeqView v;
  v.base = reinterpret_cast<char*>(t.data);
  v.sn = t.stride_n * es;
  v.sh = t.stride_h * es;
  v.sl = t.stride_l * es;
  return v;
}
inline srwm::StateView view(const srwm_b200_state& t) {
  srwm::StateView v;
  v.base = t.data;
  v.sn = t.stride_n;
  v.sh = t.stride_h;
  return v;
}

inline int check_dims(int N, int H, int L, long long* grid) {
  if (N < 0 || H < 0 || L < 0) return SRWM_B200_ERR_SHAPE;
  const long long g = (long long)N * H;
  if (g > 0x7fffffffLL) return SRWM_B200_ERR_SHAPE;
  *grid = g;
  return 0;
}

// Extension block of the layer-level calls: all four base_* or none; shift and done need a
// base.  Sets the kernels' flag bits.
inline int check_ext(const srwm_b200_srwm_ext* x, bool forward, unsigned* flags) {
  *flags = 0;
  if (!x) return 0;
  const int nb = (x->base_W_y.data != nullptr) + (x->base_W_q.data != nullptr) + (x->base_W_k.data != nullptr) +
                 (x->base_w_b.data != nullptr);
  const int ns = (x->shift_W_y.data != nullptr) + (x->shift_W_q.data != nullptr) + (x->shift_W_k.data != nullptr) +
                 (x->shift_w_b.data != nullptr);
  if (nb != 0 && nb != 4) return SRWM_B200_ERR_NULL;
  if (ns != 0 && ns != 4) return SRWM_B200_ERR_NULL;
  if (nb == 0) return (ns != 0 || x->done != nullptr) ? SRWM_B200_ERR_NULL : 0;
  if (!state_aligned(x->base_W_y) || !state_aligned(x->base_W_q) || !state_aligned(x->base_W_k) ||
      !state_aligned(x->base_w_b))
    return SRWM_B200_ERR_ALIGN;
  *flags |= srwm::F_BASE;
  if (forward && ns == 4) {
    if (!state_aligned(x->shift_W_y) || !state_aligned(x->shift_W_q) || !state_aligned(x->shift_W_k) ||
        !state_aligned(x->shift_w_b))
      return SRWM_B200_ERR_ALIGN;
    *flags |= srwm::F_SHIFT_IN;
  }
  if (forward && x->done) *flags |= srwm::F_DONE;
  // a reverse-time backward cannot cross an in-kernel reset (the pre-reset state is gone)
  if (!forward && x->done) return SRWM_B200_ERR_UNSUPPORTED;
  return 0;
}

inline int finish(int rc, int cuda_err) {
  if (rc == -7) {
    g_last_cuda_error = cuda_err;
    return SRWM_B200_ERR_CUDA;
  }
  if (rc == -6) return SRWM_B200_ERR_VARIANT;
  if (rc == -3) return SRWM_B200_ERR_HEAD_DIM;
  return rc;
}

}  // namespace

extern "C" {

int srwm_b200_abi_version(void) { return SRWM_B200_ABI_VERSION; }

int srwm_b200_head_dim_supported(int32_t E) { return head_dim_ok(E) ? 1 : 0; }

int srwm_b200_last_cuda_error(void) { return g_last_cuda_error; }

const char* srwm_b200_strerror(int code) {
  switch (code) {
    case SRWM_B200_OK: return "ok";
    case SRWM_B200_ERR_NULL: return "a required pointer is NULL";
    case SRWM_B200_ERR_SHAPE: return "invalid shape (negative size or N*H too large)";
    case SRWM_B200_ERR_HEAD_DIM: return "head dimension not supported (E must be 8, 16, 32 or 64; delta rule needs M == E)";
    case SRWM_B200_ERR_DTYPE: return "unknown io_dtype";
    case SRWM_B200_ERR_ALIGN: return "a tensor row does not start on a 16-byte boundary";
    case SRWM_B200_ERR_VARIANT: return "kernel variant not compiled in";
    case SRWM_B200_ERR_CUDA: return "CUDA runtime error (see srwm_b200_last_cuda_error)";
    case SRWM_B200_ERR_TOO_LARGE: return "size exceeds the fixed capacity of this entry point";
    case SRWM_B200_ERR_TIMEOUT: return "a kernel of an earlier call gave up waiting; results of that call are NaN";
    case SRWM_B200_ERR_UNSUPPORTED: return "this combination of arguments is not supported by the entry point";
    default: return "unknown error code";
  }
}

int srwm_b200_describe_for_grid(int32_t op, int32_t E, int32_t io_dtype, int32_t variant, int64_t grid,
                                int32_t num_sms, int32_t out[5]) {
  if (!out) return SRWM_B200_ERR_NULL;
  if (io_dtype != SRWM_B200_F32 && io_dtype != SRWM_B200_BF16) return SRWM_B200_ERR_DTYPE;
  if (grid < 0 || grid > 0x7fffffffLL) return SRWM_B200_ERR_SHAPE;
  srwm::KernelInfo info = {0, 0, 0, 0, 0};
  int ce = 0, rc;
  const bool bf = io_dtype == SRWM_B200_BF16;
  const int g = (int)grid, sms = num_sms > 0 ? num_sms : srwm::DEFAULT_SMS;
  switch (op) {
    case srwm::OP_SRWM_FWD: {
      srwm::SrwmFwdParams p = {};
      rc = bf ? srwm::dispatch_srwm_fwd_bf16(E, variant, p, g, 0, &info, 1, &ce, sms)
              : srwm::dispatch_srwm_fwd_f32(E, variant, p, g, 0, &info, 1, &ce, sms);
      break;
    }
    case srwm::OP_SRWM_BWD: {
      srwm::SrwmBwdParams p = {};
      rc = bf ? srwm::dispatch_srwm_bwd_bf16(E, variant, p, g, 0, &info, 1, &ce, sms)
              : srwm::dispatch_srwm_bwd_f32(E, variant, p, g, 0, &info, 1, &ce, sms);
      break;
    }
    case srwm::OP_SRWM_BWD_DET: {
      srwm::SrwmBwdDetParams p = {};
      rc = bf ? srwm::dispatch_srwm_bwd_det_bf16(E, variant, p, g, 0, &info, 1, &ce, sms)
              : srwm::dispatch_srwm_bwd_det_f32(E, variant, p, g, 0, &info, 1, &ce, sms);
      break;
    }
    case srwm::OP_DELTA_FWD: {
      srwm::DeltaFwdParams p = {};
      rc = bf ? srwm::dispatch_delta_fwd_bf16(E, variant, p, g, 0, &info, 1, &ce, sms)
              : srwm::dispatch_delta_fwd_f32(E, variant, p, g, 0, &info, 1, &ce, sms);
      break;
    }
    case srwm::OP_DELTA_BWD: {
      srwm::DeltaBwdParams p = {};
      rc = bf ? srwm::dispatch_delta_bwd_bf16(E, variant, p, g, 0, &info, 1, &ce, sms)
              : srwm::dispatch_delta_bwd_f32(E, variant, p, g, 0, &info, 1, &ce, sms);
      break;
    }
    default:
      return SRWM_B200_ERR_SHAPE;
  }
  if (rc != 0) return finish(rc, ce);
  out[0] = info.P; out[1] = info.R; out[2] = info.T; out[3] = info.smem; out[4] = info.id;
  return 0;
}

int srwm_b200_describe(int32_t op, int32_t E, int32_t io_dtype, int32_t variant, int32_t out[4]) {
  if (!out) return SRWM_B200_ERR_NULL;
  int32_t o5[5];
  // a grid large enough to fill any GPU: the configuration of full waves
  const int rc = srwm_b200_describe_for_grid(op, E, io_dtype, variant, 1 << 20, 0, o5);
  if (rc != 0) return rc;
  out[0] = o5[0]; out[1] = o5[1]; out[2] = o5[2]; out[3] = o5[3];
  return 0;
}

int srwm_b200_num_variants(int32_t op, int32_t E) {
  int n = 0;
  int32_t tmp[4];
  while (n < 64 && srwm_b200_describe(op, E, SRWM_B200_F32, n, tmp) == 0) ++n;
  return n;
}

// ---------------------------------------------------------------------------------------
int srwm_b200_srwm_forward(const srwm_b200_srwm_fwd_args* a, void* stream) {
  return srwm_b200_srwm_layer_forward(a, nullptr, stream);
}

int srwm_b200_srwm_backward(const srwm_b200_srwm_bwd_args* a, void* stream) {
  return srwm_b200_srwm_layer_backward(a, nullptr, stream);
}

int srwm_b200_srwm_layer_forward(const srwm_b200_srwm_fwd_args* a, const srwm_b200_srwm_ext* x, void* stream) {
  if (!a) return SRWM_B200_ERR_NULL;
  long long grid;
  if (int rc = check_dims(a->N, a->H, a->L, &grid)) return rc;
  if (!head_dim_ok(a->E)) return SRWM_B200_ERR_HEAD_DIM;
  if (a->io_dtype != SRWM_B200_F32 && a->io_dtype != SRWM_B200_BF16) return SRWM_B200_ERR_DTYPE;
  if (grid == 0 || a->L == 0) return 0;
  const bool save = !(a->flags & SRWM_B200_FLAG_NO_SAVE);
  if (!a->x.data || !a->out.data || !a->W_y.data || !a->W_q.data || !a->W_k.data || !a->w_b.data)
    return SRWM_B200_ERR_NULL;
  if (save && (!a->q.data || !a->k.data || !a->beta.data || !a->y_diff.data || !a->q_diff.data ||
               !a->k_diff.data || !a->beta_diff.data))
    return SRWM_B200_ERR_NULL;
  const int es = esize(a->io_dtype);
  bool ok = seq_aligned(a->x, es) && seq_aligned(a->out, es) && state_aligned(a->W_y) && state_aligned(a->W_q) &&
            state_aligned(a->W_k) && state_aligned(a->w_b);
  if (save)
    ok = ok && seq_aligned(a->q, 4) && seq_aligned(a->k, 4) && seq_aligned(a->beta, 4) && seq_aligned(a->y_diff, 4) &&
         seq_aligned(a->q_diff, 4) && seq_aligned(a->k_diff, 4) && seq_aligned(a->beta_diff, 4);
  if (!ok) return SRWM_B200_ERR_ALIGN;
  unsigned ext_flags = 0;
  if (int rc = check_ext(x, /*forward=*/true, &ext_flags)) return rc;

  srwm::SrwmFwdParams p = {};
  p.dbg = debug_word();
  p.N = a->N; p.H = a->H; p.L = a->L;
  p.flags = (a->flags & (SRWM_B200_FLAG_NO_SAVE | SRWM_B200_FLAG_INPUT_SOFTMAX)) | ext_flags;
  if (ext_flags & srwm::F_BASE) {
    p.bWy = view(x->base_W_y); p.bWq = view(x->base_W_q); p.bWk = view(x->base_W_k); p.bwb = view(x->base_w_b);
    p.sWy = view(x->shift_W_y); p.sWq = view(x->shift_W_q); p.sWk = view(x->shift_W_k); p.swb = view(x->shift_w_b);
    p.done = x->done; p.done_sn = x->done_stride_n; p.done_sl = x->done_stride_l;
  }
  p.x = view(a->x, es); p.out = view(a->out, es);
  p.q = view(a->q, 4); p.k = view(a->k, 4); p.beta = view(a->beta, 4);
  p.yd = view(a->y_diff, 4); p.qd = view(a->q_diff, 4); p.kd = view(a->k_diff, 4); p.bd = view(a->beta_diff, 4);
  p.Wy = view(a->W_y); p.Wq = view(a->W_q); p.Wk = view(a->W_k); p.wb = view(a->w_b);
  int ce = 0;
  const int rc = a->io_dtype == SRWM_B200_BF16
                     ? srwm::dispatch_srwm_fwd_bf16(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0)
                     : srwm::dispatch_srwm_fwd_f32(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0);
  return finish(rc, ce);
}

namespace {
// group size of the fused batch reduction, and the scratch it needs: [H][ng+1] counters (padded to 256
// bytes), then [H][ng] partial states when there is more than one group
constexpr int REDUCE_GROUP = 32;
inline int reduce_groups(int N) { return N <= 2 * REDUCE_GROUP ? 1 : (N + REDUCE_GROUP - 1) / REDUCE_GROUP; }
inline int reduce_group_size(int N) { return N <= 2 * REDUCE_GROUP ? (N > 0 ? N : 1) : REDUCE_GROUP; }
inline size_t reduce_counter_bytes(int N, int H) {
  return (((size_t)H * (reduce_groups(N) + 1) * 4) + 255) / 256 * 256;
}
inline size_t reduce_scratch_bytes(int N, int H, int E) {
  const int ng = reduce_groups(N);
  return reduce_counter_bytes(N, H) + (ng > 1 ? (size_t)H * ng * (3 * E * E + 4 * E) * 4 : 0);
}
int layer_backward_impl(const srwm_b200_srwm_bwd_args* a, const srwm_b200_srwm_ext* x,
                        const srwm_b200_srwm_reduce* red, void* scratch, void* stream);
}  // namespace

size_t srwm_b200_srwm_reduce_scratch_bytes(int32_t N, int32_t H, int32_t E) {
  if (N < 0 || H < 0 || !head_dim_ok(E)) return 0;
  return reduce_scratch_bytes(N, H, E);
}

int srwm_b200_srwm_layer_backward(const srwm_b200_srwm_bwd_args* a, const srwm_b200_srwm_ext* x, void* stream) {
  return layer_backward_impl(a, x, nullptr, nullptr, stream);
}

int srwm_b200_srwm_layer_backward_reduced(const srwm_b200_srwm_bwd_args* a, const srwm_b200_srwm_ext* x,
                                          const srwm_b200_srwm_reduce* red, void* stream) {
  if (!red) return SRWM_B200_ERR_NULL;
  if (a && a->N > 0 && a->H > 0 && head_dim_ok(a->E)) {
    if (!red->scratch) return SRWM_B200_ERR_NULL;
    if ((uintptr_t)red->scratch % 256) return SRWM_B200_ERR_ALIGN;
    if (red->scratch_bytes < 0 || (size_t)red->scratch_bytes < reduce_scratch_bytes(a->N, a->H, a->E))
      return SRWM_B200_ERR_TOO_LARGE;
  }
  return layer_backward_impl(a, x, red, red->scratch, stream);
}

// ---------------------------------------------------------------------------------------
// The same call for hosts that cannot allocate device memory.  Its working memory is this
// array, which is part of the library image: every GPU that loads the library sets the
// SRWM_B200_STATIC_SCRATCH_BYTES aside until the process exits, whether or not the entry point
// is ever called.  In host code the array's name is only a handle for the runtime, not a
// device address, so the address is looked up with cudaGetSymbolAddress -- once per device,
// with that device current -- and that pointer is what the kernel receives.
// ---------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_static_reduce_scratch[SRWM_B200_STATIC_SCRATCH_BYTES];

namespace {
// Device address of the array on the current device; looked up on the first call per device and
// remembered (the look-up allocates nothing, but it is a runtime call that should not fall inside
// a stream capture, which is why the first call on a device should be made outside one).
void* static_scratch_address(int* cuda_err) {
  static void* cache[64] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) { *cuda_err = (int)e; return nullptr; }
  if (dev < 0 || dev >= 64) { *cuda_err = (int)cudaErrorInvalidDevice; return nullptr; }
  void* ptr = __atomic_load_n(&cache[dev], __ATOMIC_ACQUIRE);
  if (ptr) return ptr;
  e = cudaGetSymbolAddress((void**)&ptr, g_static_reduce_scratch);
  if (e != cudaSuccess || !ptr) {
    *cuda_err = (int)(e != cudaSuccess ? e : cudaErrorInvalidSymbol);
    (void)cudaGetLastError();
    return nullptr;
  }
  __atomic_store_n(&cache[dev], ptr, __ATOMIC_RELEASE);
  return ptr;
}
}  // namespace

int srwm_b200_srwm_layer_backward_reduced_static(const srwm_b200_srwm_bwd_args* a, const srwm_b200_srwm_ext* x,
                                                 const srwm_b200_srwm_reduce* red, void* stream) {
  if (!a || !red) return SRWM_B200_ERR_NULL;
  void* ptr = nullptr;
  if (a->N > 0 && a->H > 0 && head_dim_ok(a->E)) {
    // sizes first: a call that does not fit is refused before anything touches the device
    if (reduce_scratch_bytes(a->N, a->H, a->E) > (size_t)SRWM_B200_STATIC_SCRATCH_BYTES) return SRWM_B200_ERR_TOO_LARGE;
    int ce = 0;
    ptr = static_scratch_address(&ce);
    if (!ptr) {
      g_last_cuda_error = ce;
      return SRWM_B200_ERR_CUDA;
    }
  }
  // red->scratch / scratch_bytes are not looked at.  The shared routine clears the counters at the head
  // of the array on the caller's stream (cudaMemsetAsync) before the kernel runs: whatever the
  // previous call left in the array is either cleared (counters) or overwritten before it is read
  // (group partials).
  return layer_backward_impl(a, x, red, ptr, stream);
}

namespace {
int layer_backward_impl(const srwm_b200_srwm_bwd_args* a, const srwm_b200_srwm_ext* x,
                        const srwm_b200_srwm_reduce* red, void* scratch, void* stream) {
  if (!a) return SRWM_B200_ERR_NULL;
  long long grid;
  if (int rc = check_dims(a->N, a->H, a->L, &grid)) return rc;
  if (!head_dim_ok(a->E)) return SRWM_B200_ERR_HEAD_DIM;
  if (a->io_dtype != SRWM_B200_F32 && a->io_dtype != SRWM_B200_BF16) return SRWM_B200_ERR_DTYPE;
  if (grid == 0) return 0;
  if (!a->W_y.data || !a->W_q.data || !a->W_k.data || !a->w_b.data || !a->grad_W_y.data || !a->grad_W_q.data ||
      !a->grad_W_k.data || !a->grad_w_b.data)
    return SRWM_B200_ERR_NULL;
  if (a->L > 0 && (!a->x.data || !a->q.data || !a->k.data || !a->beta.data || !a->y_diff.data || !a->q_diff.data ||
                   !a->k_diff.data || !a->beta_diff.data || !a->grad_out.data || !a->grad_x.data))
    return SRWM_B200_ERR_NULL;
  const int es = esize(a->io_dtype);
  bool ok = state_aligned(a->W_y) && state_aligned(a->W_q) && state_aligned(a->W_k) && state_aligned(a->w_b) &&
            state_aligned(a->grad_W_y) && state_aligned(a->grad_W_q) && state_aligned(a->grad_W_k) &&
            state_aligned(a->grad_w_b);
  if (a->L > 0)
    ok = ok && seq_aligned(a->x, es) && seq_aligned(a->grad_out, es) && seq_aligned(a->grad_x, es) &&
         seq_aligned(a->q, 4) && seq_aligned(a->k, 4) && seq_aligned(a->beta, 4) && seq_aligned(a->y_diff, 4) &&
         seq_aligned(a->q_diff, 4) && seq_aligned(a->k_diff, 4) && seq_aligned(a->beta_diff, 4);
  if (!ok) return SRWM_B200_ERR_ALIGN;
  unsigned ext_flags = 0;
  if (int rc = check_ext(x, /*forward=*/false, &ext_flags)) return rc;

  srwm::SrwmBwdParams p = {};
  p.dbg = debug_word();
  p.N = a->N; p.H = a->H; p.L = a->L;
  p.flags = (a->flags & (SRWM_B200_FLAG_STATE_GRAD_IN | SRWM_B200_FLAG_RESTORE_STATE | SRWM_B200_FLAG_INPUT_SOFTMAX)) |
            ext_flags;
  if (ext_flags & srwm::F_BASE) {
    p.bWy = view(x->base_W_y); p.bWq = view(x->base_W_q); p.bWk = view(x->base_W_k); p.bwb = view(x->base_w_b);
  }
  p.x = view(a->x, es); p.gout = view(a->grad_out, es); p.gx = view(a->grad_x, es);
  p.q = view(a->q, 4); p.k = view(a->k, 4); p.beta = view(a->beta, 4);
  p.yd = view(a->y_diff, 4); p.qd = view(a->q_diff, 4); p.kd = view(a->k_diff, 4); p.bd = view(a->beta_diff, 4);
  p.Wy = view(a->W_y); p.Wq = view(a->W_q); p.Wk = view(a->W_k); p.wb = view(a->w_b);
  p.gWy = view(a->grad_W_y); p.gWq = view(a->grad_W_q); p.gWk = view(a->grad_W_k); p.gwb = view(a->grad_w_b);
  if (red) {
    if (!red->grad_base_W_y.data || !red->grad_base_W_q.data || !red->grad_base_W_k.data || !red->grad_base_w_b.data)
      return SRWM_B200_ERR_NULL;
    if (!state_aligned(red->grad_base_W_y) || !state_aligned(red->grad_base_W_q) ||
        !state_aligned(red->grad_base_W_k) || !state_aligned(red->grad_base_w_b))
      return SRWM_B200_ERR_ALIGN;
    p.flags |= srwm::F_REDUCE;
    p.red.oWy = view(red->grad_base_W_y); p.red.oWq = view(red->grad_base_W_q);
    p.red.oWk = view(red->grad_base_W_k); p.red.owb = view(red->grad_base_w_b);
    p.red.gs = reduce_group_size(a->N);
    p.red.ng = reduce_groups(a->N);
    p.red.accumulate = red->accumulate != 0;
    p.red.cnt = reinterpret_cast<unsigned*>(scratch);
    p.red.part = reinterpret_cast<float*>(reinterpret_cast<char*>(scratch) + reduce_counter_bytes(a->N, a->H));
    // the counters start at zero (the kernel leaves them at zero too; clearing them here keeps a call
    // independent of what an aborted earlier call may have left behind)
    const cudaError_t e = cudaMemsetAsync(scratch, 0, reduce_counter_bytes(a->N, a->H), (cudaStream_t)stream);
    if (e != cudaSuccess) {
      g_last_cuda_error = (int)e;
      return SRWM_B200_ERR_CUDA;
    }
  }
  int ce = 0;
  const int rc = a->io_dtype == SRWM_B200_BF16
                     ? srwm::dispatch_srwm_bwd_bf16(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0)
                     : srwm::dispatch_srwm_bwd_f32(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0);
  return finish(rc, ce);
}
}  // namespace

int srwm_b200_srwm_backward_detached(const srwm_b200_srwm_bwd_detached_args* a, void* stream) {
  if (!a) return SRWM_B200_ERR_NULL;
  long long grid;
  if (int rc = check_dims(a->N, a->H, a->L, &grid)) return rc;
  if (!head_dim_ok(a->E)) return SRWM_B200_ERR_HEAD_DIM;
  if (a->io_dtype != SRWM_B200_F32 && a->io_dtype != SRWM_B200_BF16) return SRWM_B200_ERR_DTYPE;
  if (grid == 0) return 0;
  if (!a->base_W_y.data || !a->grad_W_y.data) return SRWM_B200_ERR_NULL;
  if (a->L > 0 && (!a->x.data || !a->k.data || !a->beta.data || !a->y_diff.data || !a->grad_out.data || !a->grad_x.data))
    return SRWM_B200_ERR_NULL;
  const int es = esize(a->io_dtype);
  bool ok = state_aligned(a->base_W_y) && state_aligned(a->grad_W_y) &&
            (a->shift_W_y.data == nullptr || state_aligned(a->shift_W_y));
  if (a->L > 0)
    ok = ok && seq_aligned(a->x, es) && seq_aligned(a->grad_out, es) && seq_aligned(a->grad_x, es) &&
         seq_aligned(a->k, 4) && seq_aligned(a->beta, 4) && seq_aligned(a->y_diff, 4);
  if (!ok) return SRWM_B200_ERR_ALIGN;

  srwm::SrwmBwdDetParams p = {};
  p.dbg = debug_word();
  p.N = a->N; p.H = a->H; p.L = a->L;
  p.flags = (a->flags & SRWM_B200_FLAG_INPUT_SOFTMAX) | (a->shift_W_y.data ? srwm::F_SHIFT_IN : 0u) |
            (a->done ? srwm::F_DONE : 0u);
  p.x = view(a->x, es); p.gout = view(a->grad_out, es); p.gx = view(a->grad_x, es);
  p.k = view(a->k, 4); p.beta = view(a->beta, 4); p.yd = view(a->y_diff, 4);
  p.bWy = view(a->base_W_y); p.sWy = view(a->shift_W_y); p.gWy = view(a->grad_W_y);
  p.done = a->done; p.done_sn = a->done_stride_n; p.done_sl = a->done_stride_l;
  int ce = 0;
  const int rc = a->io_dtype == SRWM_B200_BF16
                     ? srwm::dispatch_srwm_bwd_det_bf16(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0)
                     : srwm::dispatch_srwm_bwd_det_f32(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0);
  return finish(rc, ce);
}

int srwm_b200_delta_forward(const srwm_b200_delta_fwd_args* a, void* stream) {
  if (!a) return SRWM_B200_ERR_NULL;
  long long grid;
  if (int rc = check_dims(a->N, a->H, a->L, &grid)) return rc;
  if (!head_dim_ok(a->E) || a->M != a->E) return SRWM_B200_ERR_HEAD_DIM;
  if (a->io_dtype != SRWM_B200_F32 && a->io_dtype != SRWM_B200_BF16) return SRWM_B200_ERR_DTYPE;
  if (grid == 0 || a->L == 0) return 0;
  const bool save = !(a->flags & SRWM_B200_FLAG_NO_SAVE);
  if (!a->Q.data || !a->K.data || !a->V.data || !a->beta.data || !a->W.data || !a->out.data) return SRWM_B200_ERR_NULL;
  if (save && (!a->v_old.data || !a->v_insert.data)) return SRWM_B200_ERR_NULL;
  const int es = esize(a->io_dtype);
  bool ok = seq_aligned(a->Q, es) && seq_aligned(a->K, es) && seq_aligned(a->V, es) && seq_aligned(a->out, es) &&
            state_aligned(a->W) && ((uintptr_t)a->beta.data % es == 0);
  if (save) ok = ok && seq_aligned(a->v_old, 4) && seq_aligned(a->v_insert, 4);
  if (!ok) return SRWM_B200_ERR_ALIGN;

  srwm::DeltaFwdParams p = {};
  p.dbg = debug_word();
  p.N = a->N; p.H = a->H; p.L = a->L; p.flags = a->flags & SRWM_B200_FLAG_NO_SAVE;
  p.Q = view(a->Q, es); p.K = view(a->K, es); p.V = view(a->V, es); p.beta = view(a->beta, es);
  p.out = view(a->out, es); p.v_old = view(a->v_old, 4); p.v_ins = view(a->v_insert, 4);
  p.W = view(a->W);
  int ce = 0;
  const int rc = a->io_dtype == SRWM_B200_BF16
                     ? srwm::dispatch_delta_fwd_bf16(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0)
                     : srwm::dispatch_delta_fwd_f32(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0);
  return finish(rc, ce);
}

int srwm_b200_delta_backward(const srwm_b200_delta_bwd_args* a, void* stream) {
  if (!a) return SRWM_B200_ERR_NULL;
  long long grid;
  if (int rc = check_dims(a->N, a->H, a->L, &grid)) return rc;
  if (!head_dim_ok(a->E) || a->M != a->E) return SRWM_B200_ERR_HEAD_DIM;
  if (a->io_dtype != SRWM_B200_F32 && a->io_dtype != SRWM_B200_BF16) return SRWM_B200_ERR_DTYPE;
  if (grid == 0) return 0;
  if (!a->W.data) return SRWM_B200_ERR_NULL;
  if (a->L > 0 && (!a->Q.data || !a->K.data || !a->V.data || !a->beta.data || !a->v_old.data || !a->v_insert.data ||
                   !a->grad_out.data || !a->grad_Q.data || !a->grad_K.data || !a->grad_V.data || !a->grad_beta.data))
    return SRWM_B200_ERR_NULL;
  const int es = esize(a->io_dtype);
  bool ok = state_aligned(a->W) && (a->grad_W0.data == nullptr || state_aligned(a->grad_W0));
  if (a->L > 0)
    ok = ok && seq_aligned(a->Q, es) && seq_aligned(a->K, es) && seq_aligned(a->V, es) && seq_aligned(a->grad_out, es) &&
         seq_aligned(a->grad_Q, es) && seq_aligned(a->grad_K, es) && seq_aligned(a->grad_V, es) &&
         seq_aligned(a->v_old, 4) && seq_aligned(a->v_insert, 4) && ((uintptr_t)a->beta.data % es == 0) &&
         ((uintptr_t)a->grad_beta.data % es == 0);
  if (!ok) return SRWM_B200_ERR_ALIGN;

  srwm::DeltaBwdParams p = {};
  p.dbg = debug_word();
  p.N = a->N; p.H = a->H; p.L = a->L; p.flags = 0;
  p.Q = view(a->Q, es); p.K = view(a->K, es); p.V = view(a->V, es); p.beta = view(a->beta, es);
  p.v_old = view(a->v_old, 4); p.v_ins = view(a->v_insert, 4); p.gout = view(a->grad_out, es);
  p.gQ = view(a->grad_Q, es); p.gK = view(a->grad_K, es); p.gV = view(a->grad_V, es); p.gbeta = view(a->grad_beta, es);
  p.W = view(a->W); p.gW0 = view(a->grad_W0);
  int ce = 0;
  const int rc = a->io_dtype == SRWM_B200_BF16
                     ? srwm::dispatch_delta_bwd_bf16(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0)
                     : srwm::dispatch_delta_bwd_f32(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0);
  return finish(rc, ce);
}

int srwm_b200_delta_packed_forward(const srwm_b200_delta_packed_fwd_args* a, void* stream) {
  if (!a) return SRWM_B200_ERR_NULL;
  long long grid;
  if (int rc = check_dims(a->N, a->H, a->L, &grid)) return rc;
  if (!head_dim_ok(a->E)) return SRWM_B200_ERR_HEAD_DIM;
  if (a->io_dtype != SRWM_B200_F32 && a->io_dtype != SRWM_B200_BF16) return SRWM_B200_ERR_DTYPE;
  if (grid == 0 || a->L == 0) return 0;
  const bool save = !(a->flags & SRWM_B200_FLAG_NO_SAVE);
  if (!a->qkvb.data || !a->W.data || !a->out.data) return SRWM_B200_ERR_NULL;
  if (save && (!a->v_old.data || !a->v_insert.data)) return SRWM_B200_ERR_NULL;
  const int es = esize(a->io_dtype);
  bool ok = ((uintptr_t)a->qkvb.data % es == 0) && seq_aligned(a->out, es) && state_aligned(a->W);
  if (save) ok = ok && seq_aligned(a->v_old, 4) && seq_aligned(a->v_insert, 4);
  if (!ok) return SRWM_B200_ERR_ALIGN;

  srwm::DeltaFwdParams p = {};
  p.dbg = debug_word();
  p.N = a->N; p.H = a->H; p.L = a->L;
  p.flags = (a->flags & SRWM_B200_FLAG_NO_SAVE) | srwm::F_PACKED |
            ((a->flags & SRWM_B200_FLAG_ZERO_INIT) ? srwm::F_ZERO_INIT : 0u);
  p.eps = a->norm_eps;
  p.Q = view(a->qkvb, es);
  p.out = view(a->out, es); p.v_old = view(a->v_old, 4); p.v_ins = view(a->v_insert, 4);
  p.W = view(a->W);
  int ce = 0;
  const int rc = a->io_dtype == SRWM_B200_BF16
                     ? srwm::dispatch_delta_fwd_bf16(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0)
                     : srwm::dispatch_delta_fwd_f32(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0);
  return finish(rc, ce);
}

int srwm_b200_delta_packed_backward(const srwm_b200_delta_packed_bwd_args* a, void* stream) {
  if (!a) return SRWM_B200_ERR_NULL;
  long long grid;
  if (int rc = check_dims(a->N, a->H, a->L, &grid)) return rc;
  if (!head_dim_ok(a->E)) return SRWM_B200_ERR_HEAD_DIM;
  if (a->io_dtype != SRWM_B200_F32 && a->io_dtype != SRWM_B200_BF16) return SRWM_B200_ERR_DTYPE;
  if (grid == 0) return 0;
  if (!a->W.data) return SRWM_B200_ERR_NULL;
  if (a->L > 0 && (!a->qkvb.data || !a->v_old.data || !a->v_insert.data || !a->grad_out.data || !a->grad_qkvb.data))
    return SRWM_B200_ERR_NULL;
  const int es = esize(a->io_dtype);
  bool ok = state_aligned(a->W) && (a->grad_W0.data == nullptr || state_aligned(a->grad_W0));
  if (a->L > 0)
    ok = ok && ((uintptr_t)a->qkvb.data % es == 0) && ((uintptr_t)a->grad_qkvb.data % es == 0) &&
         seq_aligned(a->grad_out, es) && seq_aligned(a->v_old, 4) && seq_aligned(a->v_insert, 4);
  if (!ok) return SRWM_B200_ERR_ALIGN;

  srwm::DeltaBwdParams p = {};
  p.dbg = debug_word();
  p.N = a->N; p.H = a->H; p.L = a->L;
  p.flags = srwm::F_PACKED;
  p.eps = a->norm_eps;
  p.Q = view(a->qkvb, es); p.gQ = view(a->grad_qkvb, es);
  p.v_old = view(a->v_old, 4); p.v_ins = view(a->v_insert, 4); p.gout = view(a->grad_out, es);
  p.W = view(a->W); p.gW0 = view(a->grad_W0);
  int ce = 0;
  const int rc = a->io_dtype == SRWM_B200_BF16
                     ? srwm::dispatch_delta_bwd_bf16(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0)
                     : srwm::dispatch_delta_bwd_f32(a->E, a->variant, p, (int)grid, (cudaStream_t)stream, nullptr, 0, &ce, 0);
  return finish(rc, ce);
}

#ifdef SRWM_DEBUG_CHECKS
namespace {
__global__ void debug_selftest_kernel(unsigned long long* dbg) {
  // a chunk that starts before the sequence, seen by the second warp: must be recorded and reported as bad, touching nothing
  if (threadIdx.x >= 32) (void)SRWM_BAD_ROWS(dbg, 255, -16, 16, 0, 16);
}
}  // namespace
#endif

int srwm_b200_debug_status(uint64_t* status) {
  if (!status) return SRWM_B200_ERR_NULL;
  *status = 0;
#ifdef SRWM_DEBUG_CHECKS
  unsigned long long w = 0ull, zero = 0ull;
  cudaError_t e = cudaMemcpyFromSymbol(&w, g_debug_status, sizeof(w));   // waits for the kernels in flight
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_debug_status, &zero, sizeof(zero));
  if (e != cudaSuccess) {
    g_last_cuda_error = (int)e;
    return SRWM_B200_ERR_CUDA;
  }
  *status = w;
  return 0;
#else
  return 1;
#endif
}

int srwm_b200_debug_selftest(void* stream) {
#ifdef SRWM_DEBUG_CHECKS
  unsigned long long* w = debug_word();
  if (!w) return SRWM_B200_ERR_CUDA;
  debug_selftest_kernel<<<1, 64, 0, (cudaStream_t)stream>>>(w);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    g_last_cuda_error = (int)e;
    return SRWM_B200_ERR_CUDA;
  }
  return 0;
#else
  (void)stream;
  return 1;
#endif
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Batch reduction: dst[i] (+)= sum_n src[n*stride_n + i].  A block of 1024 threads covers 128
// outputs (32 lanes x float4) and splits the batch over its 32 warps (four independent loads
// in flight per thread); the 32 partial sums are combined through shared memory in a fixed
// order, so the result does not depend on timing.  Reads are 16-byte and coalesced.
// ---------------------------------------------------------------------------------------
namespace {
constexpr int RB_SLICES = 32;
__device__ __forceinline__ void add4(float4& a, const float4& v) { a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w; }

__global__ void __launch_bounds__(32 * RB_SLICES) reduce_batch_kernel(const float* __restrict__ src, long long stride_n,
                                                                      int N, long long count, float* __restrict__ dst,
                                                                      int accumulate) {
  __shared__ float4 part[RB_SLICES][32];
  const int lane = threadIdx.x % 32, slice = threadIdx.x / 32;
  const long long i = ((long long)blockIdx.x * 32 + lane) * 4;
  const bool full = i + 4 <= count;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (full) {
    const float* s0 = src + i;
    int n = slice;
    for (; n + 3 * RB_SLICES < N; n += 4 * RB_SLICES) {
      const float4 v0 = *reinterpret_cast<const float4*>(s0 + (long long)n * stride_n);
      const float4 v1 = *reinterpret_cast<const float4*>(s0 + (long long)(n + RB_SLICES) * stride_n);
      const float4 v2 = *reinterpret_cast<const float4*>(s0 + (long long)(n + 2 * RB_SLICES) * stride_n);
      const float4 v3 = *reinterpret_cast<const float4*>(s0 + (long long)(n + 3 * RB_SLICES) * stride_n);
      add4(acc, v0); add4(acc, v1); add4(acc, v2); add4(acc, v3);
    }
    for (; n < N; n += RB_SLICES) add4(acc, *reinterpret_cast<const float4*>(s0 + (long long)n * stride_n));
  }
  part[slice][lane] = acc;
  __syncthreads();
  if (slice != 0 || i >= count) return;
  if (full) {
    float4 t = accumulate ? *reinterpret_cast<const float4*>(dst + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int s8 = 0; s8 < RB_SLICES; ++s8) add4(t, part[s8][lane]);
    *reinterpret_cast<float4*>(dst + i) = t;
  } else {   // ragged end: fewer than four outputs left
    for (long long j = i; j < count; ++j) {
      float t = accumulate ? dst[j] : 0.f;
      for (int n = 0; n < N; ++n) t += src[(long long)n * stride_n + j];
      dst[j] = t;
    }
  }
}

// Four state blocks in one launch (blocks of CTAs per state block z = blockIdx.y); per output the same
// two-level sum as above.  A layer's four slow-weight gradients are 40-400 KB: the launches, not the
// bytes, were the cost of four separate calls.
struct ReduceStates {
  srwm_b200_state src[4], sub[4];
  float* dst[4];
  int N, H, E;
};
__device__ __forceinline__ float4 sum_samples(const srwm_b200_state& s, int h, int off, int N, int slice) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* p = s.data + (long long)h * s.stride_h + off;
  int n = slice;
  for (; n + 3 * RB_SLICES < N; n += 4 * RB_SLICES) {
    const float4 v0 = *reinterpret_cast<const float4*>(p + (long long)n * s.stride_n);
    const float4 v1 = *reinterpret_cast<const float4*>(p + (long long)(n + RB_SLICES) * s.stride_n);
    const float4 v2 = *reinterpret_cast<const float4*>(p + (long long)(n + 2 * RB_SLICES) * s.stride_n);
    const float4 v3 = *reinterpret_cast<const float4*>(p + (long long)(n + 3 * RB_SLICES) * s.stride_n);
    add4(acc, v0); add4(acc, v1); add4(acc, v2); add4(acc, v3);
  }
  for (; n < N; n += RB_SLICES) add4(acc, *reinterpret_cast<const float4*>(p + (long long)n * s.stride_n));
  return acc;
}
__global__ void __launch_bounds__(32 * RB_SLICES) reduce_states_kernel(const ReduceStates p) {
  __shared__ float4 part[RB_SLICES][32];
  const int z = blockIdx.y, per_head = z < 3 ? p.E * p.E : 4 * p.E;
  const int lane = threadIdx.x % 32, slice = threadIdx.x / 32;
  const int i = (blockIdx.x * 32 + lane) * 4;      // a multiple of four values of one head
  if (p.dst[z] == nullptr || blockIdx.x * 128 >= p.H * per_head) return;
  const bool in = i < p.H * per_head;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (in) {
    const int h = i / per_head, off = i % per_head;
    acc = sum_samples(p.src[z], h, off, p.N, slice);
    if (p.sub[z].data != nullptr) {
      const float4 b = sum_samples(p.sub[z], h, off, p.N, slice);
      acc.x -= b.x; acc.y -= b.y; acc.z -= b.z; acc.w -= b.w;
    }
  }
  part[slice][lane] = acc;
  __syncthreads();
  if (slice != 0 || !in) return;
  float4 t = part[0][lane];
#pragma unroll
  for (int k = 1; k < RB_SLICES; ++k) add4(t, part[k][lane]);
  *reinterpret_cast<float4*>(p.dst[z] + i) = t;
}

// Up to four states copied or zeroed in one launch: as four copies (or fills) they are bound by the host, some 6 us each
// beside 2 us on the GPU.
struct CopyStates {
  srwm_b200_state src[4];
  float* dst[4];
  int N, H, E;
};
__global__ void __launch_bounds__(256) copy_states_kernel(const CopyStates p) {
  const int z = blockIdx.y, per_head = z < 3 ? p.E * p.E : 4 * p.E;
  if (p.dst[z] == nullptr) return;
  const long long quads = (long long)p.N * p.H * (per_head / 4);
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < quads; i += (long long)gridDim.x * 256) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.src[z].data != nullptr) {
      const int seq = (int)(i / (per_head / 4)), off = (int)(i % (per_head / 4)) * 4;
      v = *reinterpret_cast<const float4*>(p.src[z].data + (seq / p.H) * p.src[z].stride_n + (seq % p.H) * p.src[z].stride_h + off);
    }
    *reinterpret_cast<float4*>(p.dst[z] + i * 4) = v;
  }
}
}  // namespace

extern "C" int srwm_b200_reduce_batch(const float* src, int64_t stride_n, int32_t N, int64_t count, float* dst,
                                      int32_t accumulate, void* stream) {
  if (N < 0 || count < 0) return SRWM_B200_ERR_SHAPE;
  if (count == 0) return 0;
  if (!dst || (N > 0 && !src)) return SRWM_B200_ERR_NULL;
  if ((uintptr_t)src % 16 || (uintptr_t)dst % 16 || (stride_n * 4) % 16) return SRWM_B200_ERR_ALIGN;
  const long long blocks = (count + 127) / 128;
  if (blocks > 0x7fffffffLL) return SRWM_B200_ERR_SHAPE;
  reduce_batch_kernel<<<(unsigned)blocks, 32 * RB_SLICES, 0, (cudaStream_t)stream>>>(src, stride_n, N, count, dst, accumulate);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    g_last_cuda_error = (int)e;
    return SRWM_B200_ERR_CUDA;
  }
  return 0;
}

extern "C" int srwm_b200_reduce_states(const srwm_b200_state* src, const srwm_b200_state* sub, float* const* dst, int32_t N,
                                       int32_t H, int32_t E, void* stream) {
  if (N < 0 || H < 0) return SRWM_B200_ERR_SHAPE;
  if (!head_dim_ok(E)) return SRWM_B200_ERR_HEAD_DIM;
  if (!src || !sub || !dst) return SRWM_B200_ERR_NULL;
  if ((long long)H * E * E > 0x7fffffffLL - 128) return SRWM_B200_ERR_SHAPE;
  ReduceStates p;
  p.N = N; p.H = H; p.E = E;
  bool any = false;
  for (int z = 0; z < 4; ++z) {
    p.src[z] = src[z]; p.sub[z] = sub[z]; p.dst[z] = dst[z];
    if (!dst[z]) continue;
    any = true;
    if (N > 0 && !src[z].data) return SRWM_B200_ERR_NULL;
    if (!state_aligned(src[z]) || !state_aligned(sub[z]) || (uintptr_t)dst[z] % 16) return SRWM_B200_ERR_ALIGN;
  }
  if (!any || H == 0) return 0;
  reduce_states_kernel<<<dim3((unsigned)((H * E * E + 127) / 128), 4), 32 * RB_SLICES, 0, (cudaStream_t)stream>>>(p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    g_last_cuda_error = (int)e;
    return SRWM_B200_ERR_CUDA;
  }
  return 0;
}

static int cuda_result(cudaError_t e) {
  if (e == cudaSuccess) return 0;
  g_last_cuda_error = (int)e;
  return SRWM_B200_ERR_CUDA;
}

extern "C" int srwm_b200_copy_states(const srwm_b200_state* src, float* const* dst, int32_t N, int32_t H, int32_t E,
                                     void* stream) {
  if (N < 0 || H < 0 || (long long)N * H > 0x7fffffffLL) return SRWM_B200_ERR_SHAPE;
  if (!head_dim_ok(E)) return SRWM_B200_ERR_HEAD_DIM;
  if (!src || !dst) return SRWM_B200_ERR_NULL;
  CopyStates p;
  p.N = N; p.H = H; p.E = E;
  bool any = false;
  for (int z = 0; z < 4; ++z) {
    p.src[z] = src[z]; p.dst[z] = dst[z];
    if (!dst[z]) continue;
    any = true;
    if (!state_aligned(src[z]) || (uintptr_t)dst[z] % 16) return SRWM_B200_ERR_ALIGN;
  }
  if (!any || N == 0 || H == 0) return 0;
  const long long blocks = ((long long)N * H * E * E / 4 + 255) / 256, most = 8 * srwm::common_sms();
  copy_states_kernel<<<dim3((unsigned)(blocks < most ? blocks : most), 4), 256, 0, (cudaStream_t)stream>>>(p);
  return cuda_result(cudaGetLastError());
}

extern "C" size_t srwm_b200_gemm_scratch_bytes(int32_t M, int32_t N, int32_t K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const int parts = srwm::gemm_is_skinny(M, N, K) ? 1 : srwm::gemm_parts(M, N, K);
  return parts > 1 ? (size_t)parts * M * N * 4 : 0;
}

extern "C" int32_t srwm_b200_gemm_few_rows(int32_t M, int32_t N, int32_t K) {
  return M > 0 && N > 0 && K > 0 && srwm::gemm_is_skinny(M, N, K);
}

extern "C" int srwm_b200_gemm_f32(const srwm_b200_gemm_args* a, void* stream) {
  if (!a) return SRWM_B200_ERR_NULL;
  if (srwm::gemm_gave_up()) return SRWM_B200_ERR_TIMEOUT;
  if (a->M < 0 || a->N < 0 || a->K <= 0 || (a->M + 127ll) / 128 > 65535) return SRWM_B200_ERR_SHAPE;
  if (a->M == 0 || a->N == 0) return 0;
  if (!a->A || !a->B || !a->C) return SRWM_B200_ERR_NULL;
  if ((uintptr_t)a->A % 16 || (uintptr_t)a->B % 16 || (uintptr_t)a->C % 16 || (uintptr_t)a->add % 16 || a->lda % 4 ||
      a->ldb % 4 || a->ldc % 4 || a->ldadd % 4 || a->N % 4 || ((!a->trans_a || !a->trans_b) && a->K % 4))
    return SRWM_B200_ERR_ALIGN;
  srwm::GemmParams p = {};
  p.A = a->A; p.B = a->B; p.add = a->add; p.C = a->C;
  p.lda = a->lda; p.ldb = a->ldb; p.ldc = a->ldc; p.ldadd = a->ldadd;
  p.M = a->M; p.N = a->N; p.K = a->K;
  const bool ta = a->trans_a != 0, tb = a->trans_b != 0;
  p.relu = a->relu != 0;
  if (p.relu && !srwm::gemm_is_skinny(a->M, a->N, a->K)) return SRWM_B200_ERR_SHAPE;
  if (srwm::gemm_is_skinny(a->M, a->N, a->K)) return cuda_result(srwm::gemm_skinny_launch(p, ta, tb, (cudaStream_t)stream));
  const int parts = srwm::gemm_parts(a->M, a->N, a->K);
  if (parts > 1 && (!a->scratch || a->scratch_bytes < (int64_t)parts * a->M * a->N * 4 || a->ldc != a->N ||
                    (a->add && a->ldadd != a->N) || (uintptr_t)a->scratch % 16))
    return SRWM_B200_ERR_NULL;
  return cuda_result(srwm::gemm_launch(p, ta, tb, parts > 1 ? (float*)a->scratch : nullptr, (cudaStream_t)stream));
}

extern "C" int32_t srwm_b200_gemm_timeouts(void) { return (int32_t)srwm::gemm_timeouts(); }

extern "C" int srwm_b200_debug_gemm_tries(int32_t tries) {
#ifdef SRWM_DEBUG_CHECKS
  srwm::gemm_tries = tries;
  return 0;
#else
  (void)tries;
  return 1;
#endif
}

static int norm_check(const void* a, const void* b, const void* c, const void* d, int64_t rows, int32_t D) {
  if (rows < 0 || D <= 0 || D > 1024) return SRWM_B200_ERR_SHAPE;
  if (rows == 0) return 0;
  if (!a || !b || !c || !d) return SRWM_B200_ERR_NULL;
  if (D % 4 || (uintptr_t)a % 16 || (uintptr_t)b % 16 || (uintptr_t)c % 16 || (uintptr_t)d % 16) return SRWM_B200_ERR_ALIGN;
  return 0;
}

extern "C" int srwm_b200_norm_forward(const float* x, const float* gamma, const float* beta, float* y, float* mean, float* rstd,
                                      int64_t rows, int32_t D, float eps, void* stream) {
  if (int rc = norm_check(x, gamma, beta, y, rows, D)) return rc;
  if (rows == 0) return 0;
  if ((mean == nullptr) != (rstd == nullptr)) return SRWM_B200_ERR_NULL;
  srwm::NormParams p = {};
  p.x = x; p.gamma = gamma; p.beta = beta; p.y = y; p.mean = mean; p.rstd = rstd;
  p.rows = rows; p.D = D; p.eps = eps;
  return cuda_result(srwm::norm_forward(p, (cudaStream_t)stream));
}

extern "C" size_t srwm_b200_norm_scratch_bytes(int64_t rows, int32_t D) {
  return rows <= 0 || D <= 0 ? 0 : (size_t)srwm::norm_blocks(rows) * 2 * D * 4;
}

extern "C" int srwm_b200_norm_backward(const float* x, const float* gamma, const float* dy, const float* mean, const float* rstd,
                                       float* dx, float* dgamma, float* dbeta, int64_t rows, int32_t D, void* scratch,
                                       int64_t scratch_bytes, void* stream) {
  if (int rc = norm_check(x, gamma, dy, dx, rows, D)) return rc;
  if (rows == 0) return 0;
  if (!mean || !rstd || !dgamma || !dbeta || !scratch || scratch_bytes < (int64_t)srwm_b200_norm_scratch_bytes(rows, D))
    return SRWM_B200_ERR_NULL;
  if ((uintptr_t)scratch % 16) return SRWM_B200_ERR_ALIGN;
  srwm::NormParams p = {};
  p.x = x; p.gamma = gamma; p.dy = dy; p.y = dx;
  p.mean = const_cast<float*>(mean); p.rstd = const_cast<float*>(rstd);
  p.part = (float*)scratch;
  p.rows = rows; p.D = D;
  return cuda_result(srwm::norm_backward(p, dgamma, dbeta, (cudaStream_t)stream));
}

extern "C" int32_t srwm_b200_block_fits(int32_t rows, int32_t K0, int32_t D, int32_t F, int32_t N) {
  return K0 > 0 && D > 0 && F > 0 && N > 0 && srwm::block_pays(rows, K0, D, F, N);
}

extern "C" int srwm_b200_block_forward(const srwm_b200_block_args* a, void* stream) {
  if (!a) return SRWM_B200_ERR_NULL;
  if (a->rows < 0 || a->K0 <= 0 || a->D <= 0 || a->F <= 0 || a->N <= 0) return SRWM_B200_ERR_SHAPE;
  if (a->rows == 0) return 0;
  if (!srwm::block_fits(a->K0, a->D, a->F, a->N)) return SRWM_B200_ERR_SHAPE;
  if (!a->att || !a->res || !a->wo || !a->gamma || !a->beta || !a->w1 || !a->w2 || !a->y) return SRWM_B200_ERR_NULL;
  for (const void* p : {(const void*)a->att, (const void*)a->res, (const void*)a->wo, (const void*)a->gamma, (const void*)a->beta,
                        (const void*)a->w1, (const void*)a->b1, (const void*)a->w2, (const void*)a->b2, (const void*)a->y})
    if ((uintptr_t)p % 16) return SRWM_B200_ERR_ALIGN;
  srwm::BlockParams p = {};
  p.att = a->att; p.res = a->res; p.wo = a->wo; p.gamma = a->gamma; p.beta = a->beta;
  p.w1 = a->w1; p.b1 = a->b1; p.w2 = a->w2; p.b2 = a->b2; p.y = a->y;
  p.rows = a->rows; p.K0 = a->K0; p.D = a->D; p.F = a->F; p.N = a->N;
  p.eps = a->eps;
  return cuda_result(srwm::block_launch(p, (cudaStream_t)stream));
}
