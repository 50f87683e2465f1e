// Python module srwm_b200._host: see host_common.h.
#include "host_layers.h"

namespace {
using namespace host;

// (The structures are sized by the declarations of the bound functions.)
PyObject* bind(PyObject*, PyObject* dict) {   // {name: address}
  Api& a = api();
#define X(name)                                                                              \
  {                                                                                          \
    PyObject* v = PyDict_GetItemString(dict, #name);                                         \
    void* p = v ? PyLong_AsVoidPtr(v) : nullptr;                                             \
    if (!p) {                                                                                \
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "missing library symbol " #name); \
      return nullptr;                                                                        \
    }                                                                                        \
    a.name = reinterpret_cast<decltype(a.name)>(p);                                          \
  }
  SRWM_HOST_API(X)
#undef X
  Py_RETURN_NONE;
}

// Tensor arguments [from, from + n); false if one is not a plain tensor (None: left undefined if allowed).
bool take(PyObject* const* args, int from, int n, Tensor* out, bool none_ok = false) {
  for (int i = 0; i < n; ++i) {
    PyObject* o = args[from + i];
    if (none_ok && o == Py_None) continue;
    if (!plain(o)) return false;
    out[i] = THPVariable_Unpack(o);
  }
  return true;
}
PyObject* wrap(const variable_list& v) {
  PyObject* t = PyTuple_New((Py_ssize_t)v.size());
  if (!t) return nullptr;
  for (size_t i = 0; i < v.size(); ++i) PyTuple_SET_ITEM(t, (Py_ssize_t)i, THPVariable_Wrap(v[i]));
  return t;
}
PyObject* declined() { Py_RETURN_NOTIMPLEMENTED; }
bool arity(Py_ssize_t got, Py_ssize_t want) {
  if (got == want) return true;
  PyErr_SetString(PyExc_TypeError, "wrong number of arguments");
  return false;
}
struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};

PyObject* self_ref_impl(PyObject* const* args, Py_ssize_t n, bool stateful) {
  HANDLE_TH_ERRORS
  if (!arity(n, 5)) return nullptr;
  Tensor x;
  Four W;
  if (forward_ad() || !take(args, 0, 1, &x) || !take(args, 1, 4, W.data()) || !operator_args_ok(x, W)) return declined();
  variable_list r;
  const bool grad = wants_grad({&x, &W[0], &W[1], &W[2], &W[3]});
  {
    NoGil nogil;
    if (grad) r = SelfRef::apply(x, W[0], W[1], W[2], W[3], stateful);
    else r = {srwm_forward(x, W, nullptr, nullptr, Tensor(), false, nullptr)};
  }
  if (!stateful) return THPVariable_Wrap(r[0]);
  if (grad) return wrap(r);
  PyObject* out = THPVariable_Wrap(r[0]);   // without autograd the caller's own state tensors come back
  PyObject* t = PyTuple_Pack(5, out, args[1], args[2], args[3], args[4]);
  Py_DECREF(out);
  return t;
  END_HANDLE_TH_ERRORS
}
PyObject* self_ref(PyObject*, PyObject* const* args, Py_ssize_t n) { return self_ref_impl(args, n, false); }
PyObject* stateful_self_ref(PyObject*, PyObject* const* args, Py_ssize_t n) { return self_ref_impl(args, n, true); }

PyObject* fast_weight_delta(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 5)) return nullptr;
  Tensor t[5];
  if (forward_ad() || !take(args, 0, 5, t) || !delta_args_ok(t[0], t[1], t[2], t[3], t[4])) return declined();
  Tensor out;
  {
    NoGil nogil;
    if (wants_grad({&t[0], &t[1], &t[2], &t[3]})) out = Delta::apply(t[0], t[1], t[2], t[3], t[4])[0];
    else out = delta_forward(t[0], t[1], t[2], t[3], t[4], nullptr);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// (x, W_y, W_q, W_k, w_b, s_y, s_q, s_k, s_b, done, input_softmax, detach) -> five tensors
PyObject* layer(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 12)) return nullptr;
  Tensor x, done;
  Four base, shift;
  if (forward_ad() || !take(args, 0, 1, &x) || !take(args, 1, 4, base.data()) || !take(args, 5, 4, shift.data(), true) ||
      !take(args, 9, 1, &done, true) || !layer_args_ok(x, base, shift, done))
    return declined();
  const bool softmax = PyObject_IsTrue(args[10]), detach = PyObject_IsTrue(args[11]);
  if (done.defined() && !detach) return declined();   // an error the Python side words
  variable_list r;
  {
    NoGil nogil;
    r = srwm_layer(x, base, shift, done, softmax, detach);
  }
  return wrap(r);
  END_HANDLE_TH_ERRORS
}

// (qkvb, W, norm_eps, zero_init)
PyObject* delta_layer(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 4)) return nullptr;
  Tensor t[2];
  if (forward_ad() || !take(args, 0, 2, t) || !packed_args_ok(t[0], t[1])) return declined();
  const double eps = PyFloat_AsDouble(args[2]);
  if (eps == -1.0 && PyErr_Occurred()) return nullptr;
  const bool zero_init = PyObject_IsTrue(args[3]);
  Tensor out;
  {
    NoGil nogil;
    if (wants_grad({&t[0]})) out = DeltaLayer::apply(t[0], t[1], eps, zero_init)[0];
    else out = packed_forward(t[0], t[1], eps, zero_init, nullptr);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// (x, weight, residual or bias or None[, relu: without gradients])
PyObject* linear_py(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 && !arity(n, 3)) return nullptr;
  Tensor t[2], add;
  const bool relu = n == 4 && PyObject_IsTrue(args[3]);
  if (forward_ad() || !take(args, 0, 2, t) || !take(args, 2, 1, &add, true) || !linear_args_ok(t[0], t[1], add) ||
      (relu && wants_grad({&t[0], &t[1], &add})))
    return declined();
  Tensor out;
  {
    NoGil nogil;
    out = relu ? linear_forward(t[0], t[1], add, true) : linear(t[0], t[1], add);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// (x, weight, bias, eps)
PyObject* norm_py(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 4)) return nullptr;
  Tensor t[3];
  if (forward_ad() || !take(args, 0, 3, t) || !norm_args_ok(t[0], t[1], t[2])) return declined();
  const double eps = PyFloat_AsDouble(args[3]);
  if (eps == -1.0 && PyErr_Occurred()) return nullptr;
  Tensor out;
  {
    NoGil nogil;
    out = norm(t[0], t[1], t[2], eps);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// (h, W_y, W_q, W_k, w_b, s_y, s_q, s_k, s_b, done, unroll, out weight) -> five tensors.  With gradients only the
// unroll, whose state is detached; a step's is not.  An unroll has its done, which a step has not.
PyObject* sr_step_py(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 12)) return nullptr;
  Tensor h, done, w;
  Four base, state;
  if (forward_ad() || (at::GradMode::is_enabled() && !PyObject_IsTrue(args[10])) || !take(args, 0, 1, &h) || !take(args, 1, 4, base.data()) ||
      !take(args, 5, 4, state.data()) || !take(args, 9, 1, &done, true) || !take(args, 11, 1, &w) ||
      done.defined() != (PyObject_IsTrue(args[10]) != 0) || !sr_step_ok(h, base, state, w))
    return declined();
  variable_list r;
  {
    NoGil nogil;
    r = sr_step(h, base, state, done, w);
  }
  return r.empty() ? declined() : wrap(r);
  END_HANDLE_TH_ERRORS
}

// (x, layer norm weight, bias, eps, slow weight, W, norm_eps, zero_init, out weight) -> out, copy of W or None; without gradients
PyObject* ff_step_py(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 9)) return nullptr;
  Tensor x, ln[2], slow, W, out_w;
  if (forward_ad() || at::GradMode::is_enabled() || !take(args, 0, 1, &x) || !take(args, 1, 2, ln) || !take(args, 4, 1, &slow) ||
      !take(args, 5, 1, &W) || !take(args, 8, 1, &out_w))
    return declined();
  const double eps = PyFloat_AsDouble(args[3]), norm_eps = PyFloat_AsDouble(args[6]);
  if (PyErr_Occurred()) return nullptr;
  const bool zero_init = PyObject_IsTrue(args[7]);
  variable_list r;
  {
    NoGil nogil;
    r = ff_step(x, ln[0], ln[1], eps, slow, W, norm_eps, zero_init, out_w);
  }
  return r.empty() ? declined() : wrap(r);
  END_HANDLE_TH_ERRORS
}

// (att, h, out weight, norm weight, bias, eps, w1, b1 or None, w2, b2 or None) -> y; without gradients
PyObject* block_tail_py(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 10)) return nullptr;
  Tensor t[5], w1, b1, w2, b2;
  if (forward_ad() || at::GradMode::is_enabled() || !take(args, 0, 5, t) || !take(args, 6, 1, &w1) || !take(args, 7, 1, &b1, true) ||
      !take(args, 8, 1, &w2) || !take(args, 9, 1, &b2, true))
    return declined();
  const double eps = PyFloat_AsDouble(args[5]);
  if (PyErr_Occurred()) return nullptr;
  Tensor y;
  {
    NoGil nogil;
    y = block_tail(t[0], t[1], t[2], t[3], t[4], eps, w1, b1, w2, b2);
  }
  return y.defined() ? THPVariable_Wrap(y) : declined();
  END_HANDLE_TH_ERRORS
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr
PyMethodDef methods[] = {{"bind", bind, METH_O, nullptr},
                         {"self_ref_v0", FAST(self_ref)},
                         {"stateful_self_ref_v0", FAST(stateful_self_ref)},
                         {"fast_weight_delta", FAST(fast_weight_delta)},
                         {"srwm_layer", FAST(layer)},
                         {"delta_layer", FAST(delta_layer)},
                         {"linear", FAST(linear_py)},
                         {"sr_step", FAST(sr_step_py)},
                         {"ff_step", FAST(ff_step_py)},
                         {"layer_norm", FAST(norm_py)},
                         {"block_tail", FAST(block_tail_py)},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module_def); }
