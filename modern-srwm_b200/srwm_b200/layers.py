"""The reference's SRWM and delta-rule layers on top of the fused layer-level calls.

Same constructor arguments, parameter names (so a reference ``state_dict`` loads) and
``forward`` signatures as

* ``SRWMlayer``    supervised_learning/layer.py:112-209
* ``SRlayer``      reinforcement_learning/torchbeast/layer.py:340-421
* ``FastFFlayer``  supervised_learning/layer.py:49-108 (``norm_eps=0``, fresh zero fast weights
                   per call) and reinforcement_learning/torchbeast/layer.py:127-189
                   (``FastFFlayerRL``: ``norm_eps=1e-5``, fast weights carried as state)

but the per-call work around the operator -- input softmax, four ``W.repeat(bsz,1,1,1)``,
``shift + repeat``, the ``[L,B,H*d] -> [B,H,L,d]`` layout change and back, the four
``W_bc - W.repeat`` subtractions; for the delta rule the four-way split of the slow net's rows,
``elu + 1``, the sum normalisation and the sigmoid -- is done inside the kernels
(``layer_ops.srwm_layer`` / ``layer_ops.delta_layer``).
``SRlayer.unroll`` additionally runs the learner's one-step-at-a-time loop with episode
resets (reinforcement_learning/torchbeast_procgen/model.py:1180-1197) as ONE call.
"""
from __future__ import annotations

import math

import torch
import torch.nn as nn

from . import _lib as L
from .layer_ops import delta_layer, srwm_layer


# The modules' linear maps and layer norms run on this library's kernels (fp32 in and out; the products
# on the tensor cores at fp32 accuracy) where the module is the plain one built here and nothing asks for torch's
# own call: no hooks, no ``forward`` of the instance's own, no autocast, no tf32, no forward-mode AD; everything else goes
# through the module.
def _plain_input(x):
    return (x.is_cuda and x.dtype is torch.float32 and not torch.is_autocast_enabled("cuda")
            and not nn.modules.module._has_any_global_hook())


def _plain(mod, kind):
    d = mod.__dict__      # (half the time of attribute access, which an actor's step would notice)
    return type(mod) is kind and not (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"]
                                      or d["_backward_pre_hooks"] or "forward" in d)


def _direct(mod, kind, x):
    return _plain(mod, kind) and _plain_input(x)


def _norm(mod, x):
    if _direct(mod, nn.LayerNorm, x) and mod.bias is not None:
        r = L.host().layer_norm(x, mod.weight, mod.bias, mod.eps)
        if r is not NotImplemented:
            return r
    return mod(x)


def _linear(mod, x, residual=None):
    """``mod(x)``, plus ``residual`` where given."""
    if _direct(mod, nn.Linear, x) and mod.bias is None:
        r = L.host().linear(x, mod.weight, residual)
        if r is not NotImplemented:
            return r
    return mod(x) if residual is None else residual + mod(x)


def _feed_forward(mod, x):
    """``mod(x)`` without gradients; a plain stack of layer norms, linear maps and ReLUs runs on this library's kernels."""
    if not _plain(mod, nn.Sequential) or nn.modules.module._has_any_global_hook():
        return mod(x)
    mods, i = list(mod), 0
    while i < len(mods):
        m, r = mods[i], NotImplemented
        if _direct(m, nn.LayerNorm, x):
            r = _norm(m, x)
        elif _direct(m, nn.Linear, x):
            relu = i + 1 < len(mods) and _direct(mods[i + 1], nn.ReLU, x)   # in the product's epilogue
            r = L.host().linear(x, m.weight, m.bias, relu)
            i += r is not NotImplemented and relu
        x = m(x) if r is NotImplemented else r
        i += 1
    return x


def _idle(drop):
    d = drop.__dict__      # (and the same checks as _plain: one call less)
    return type(drop) is nn.Dropout and (d["p"] == 0.0 or not d["training"]) and not (
        d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"] or "forward" in d)


def _project(lin, drop, x, residual):
    """``residual + drop(lin(x))``; the sum in the product's epilogue while the dropout is idle."""
    if _idle(drop):
        return _linear(lin, x, residual)
    return residual + drop(_linear(lin, x))


def _block_tail(sr, ff, att, h):
    """What follows the recurrence in a block, without gradients: projection, residual, feed-forward part.  With few rows and a plain
    stack of layer norm, linear map, ReLU, linear map one kernel does all of it."""
    lin = sr.out_linear
    if (ff is not None and _plain(ff, nn.Sequential) and len(ff) == 4 and _idle(sr.drop) and _direct(lin, nn.Linear, att)
            and lin.bias is None and all(_plain(m, k) for m, k in zip(ff, (nn.LayerNorm, nn.Linear, nn.ReLU, nn.Linear)))
            and _plain_input(h)):
        norm, up, _, down = ff
        if norm.bias is not None:
            r = L.host().block_tail(att, h, lin.weight, norm.weight, norm.bias, norm.eps, up.weight, up.bias, down.weight, down.bias)
            if r is not NotImplemented:
                return r
    h = _project(lin, sr.drop, att, h)
    return h if ff is None else _feed_forward(ff, h)


def _heads(h, num_head, dim_head):
    """[L, B, H*d] -> the [B, H, L, d] view the operator reads in place."""
    slen, bsz, _ = h.shape
    return h.reshape(slen, bsz, num_head, dim_head).permute(1, 2, 0, 3)


def _merge(out):
    """[B, H, L, d] laid out like the input view -> [L, B, H*d] (a view, no copy)."""
    bsz, num_head, slen, dim_head = out.shape
    return out.transpose(1, 2).reshape(bsz, slen, num_head * dim_head).transpose(0, 1)


class SRWMlayer(nn.Module):
    """Self-referential weight matrix layer of the supervised-learning models."""

    def __init__(self, num_head, dim_head, in_dim, dropout, use_ln=True, use_input_softmax=False,
                 beta_init=-1.0, stateful=False):
        super().__init__()
        self.num_head, self.dim_head, self.in_dim = num_head, dim_head, in_dim
        self.use_ln, self.use_input_softmax, self.stateful = use_ln, use_input_softmax, stateful
        self.W_y = nn.Parameter(torch.empty(1, num_head, dim_head, dim_head))
        self.W_q = nn.Parameter(torch.empty(1, num_head, dim_head, dim_head))
        self.W_k = nn.Parameter(torch.empty(1, num_head, dim_head, dim_head))
        self.w_b = nn.Parameter(torch.empty(1, num_head, dim_head, 4))
        if use_ln:
            self.layer_norm = nn.LayerNorm(in_dim)
        self.out_linear = nn.Linear(num_head * dim_head, in_dim, bias=False)
        self.drop = nn.Dropout(dropout)
        self.reset_parameters(beta_init)

    def reset_parameters(self, beta_init):
        std = 1.0 / math.sqrt(self.dim_head)
        for w in (self.W_y, self.W_q, self.W_k):
            nn.init.normal_(w, mean=0.0, std=std)
        nn.init.normal_(self.w_b, mean=beta_init, std=std)

    def forward(self, h, state=None, get_state=False):
        x = _heads(h, self.num_head, self.dim_head)
        # stateful: gradients flow through the carried state (stateful_self_ref_v0); otherwise
        # the returned state carries none, as with the reference's in-place mutated buffers
        out, shift = srwm_layer(x, self.W_y, self.W_q, self.W_k, self.w_b, shift=state,
                                input_softmax=self.use_input_softmax)
        out = _project(self.out_linear, self.drop, _merge(out), _norm(self.layer_norm, h) if self.use_ln else h)
        if get_state:
            if not self.stateful:
                shift = tuple(s.detach() for s in shift)
            return out, shift
        return out


class SRlayer(nn.Module):
    """Self-referential weight matrix layer of the reinforcement-learning agents: the input
    softmax is always on, the state (shift from the slow weights) is required and comes
    back detached."""

    def __init__(self, num_head, dim_head, in_dim, dropout):
        super().__init__()
        self.num_head, self.dim_head, self.in_dim = num_head, dim_head, in_dim
        self.W_y = nn.Parameter(torch.empty(1, num_head, dim_head, dim_head))
        self.W_q = nn.Parameter(torch.empty(1, num_head, dim_head, dim_head))
        self.W_k = nn.Parameter(torch.empty(1, num_head, dim_head, dim_head))
        self.w_b = nn.Parameter(torch.empty(1, num_head, dim_head, 4))
        self.layer_norm = nn.LayerNorm(in_dim)
        self.out_linear = nn.Linear(num_head * dim_head, in_dim, bias=False)
        self.drop = nn.Dropout(dropout)
        self.reset_rec_parameters()

    def reset_rec_parameters(self):
        std = 1.0 / math.sqrt(self.dim_head)
        for w in (self.W_y, self.W_q, self.W_k, self.w_b):
            nn.init.normal_(w, mean=0.0, std=std)

    def forward(self, h, state=None):
        assert state is not None
        if not torch.is_grad_enabled():
            r = self._step(h, None, state, False)
            if r is not NotImplemented:
                return r[0], r[1:]
        x = _heads(h, self.num_head, self.dim_head)
        out, shift = srwm_layer(x, self.W_y, self.W_q, self.W_k, self.w_b, shift=state, input_softmax=True)
        out = _project(self.out_linear, self.drop, _merge(out), h)
        return out, tuple(s.detach() for s in shift)

    def _step(self, h, done, state, unroll):
        """The whole layer as one call; NotImplemented where it does not apply.  (Modules and parameters straight from
        their dictionaries: attribute access was 3 of an actor step's 20 us.)"""
        mods, own = self._modules, self._parameters
        lin = mods["out_linear"]
        if not _plain(lin, nn.Linear) or not _plain_input(h) or not _idle(mods["drop"]):
            return NotImplemented
        proj = lin._parameters
        if proj.get("bias") is not None:
            return NotImplemented
        return L.host().sr_step(h, own.get("W_y"), own.get("W_q"), own.get("W_k"), own.get("w_b"), *state, done, unroll,
                                proj.get("weight"))

    def unroll(self, h, done, state):
        """The learner's loop over ``h [T, B, D]`` with ``done [T, B]`` as one call: before
        step t the state of the samples with ``done[t]`` goes back to zero, every step sees a
        detached state.  Returns (out [T, B, D], state after the last step)."""
        assert state is not None
        r = self._step(h, done, state, True)
        if r is not NotImplemented:
            return r[0], r[1:]
        x = _heads(h, self.num_head, self.dim_head)
        out, shift = srwm_layer(x, self.W_y, self.W_q, self.W_k, self.w_b, shift=state, done=done.t(),
                                input_softmax=True, detach_state=True)
        out = _project(self.out_linear, self.drop, _merge(out), h)
        return out, shift


class FastFFlayer(nn.Module):
    """Delta-rule fast-weight layer of the supervised-learning models: layer norm, slow net,
    then -- in one call on the slow net's raw rows -- the q/k/beta preparation and the
    recurrence, starting from zero fast weights."""

    norm_eps = 0.0

    def __init__(self, num_head, dim_head, in_dim, dropout):
        super().__init__()
        self.num_head, self.dim_head, self.in_dim = num_head, dim_head, in_dim
        self.slow_net = nn.Linear(in_dim, num_head * (3 * dim_head + 1), bias=False)
        self.layer_norm = nn.LayerNorm(in_dim)
        self.out_linear = nn.Linear(num_head * dim_head, in_dim, bias=False)
        self.drop = nn.Dropout(dropout)

    def _rows(self, x):
        slen, bsz, _ = x.shape
        qkvb = _linear(self.slow_net, _norm(self.layer_norm, x))
        return qkvb.view(slen, bsz, self.num_head, 3 * self.dim_head + 1).permute(1, 2, 0, 3)

    def _step(self, x, W, zero_init):
        """The whole layer as one call where nothing needs a gradient; NotImplemented where it does not apply."""
        mods = self._modules
        ln, slow, lin = mods["layer_norm"], mods["slow_net"], mods["out_linear"]
        if (torch.is_grad_enabled() or not _plain_input(x) or not _plain(ln, nn.LayerNorm) or not _plain(slow, nn.Linear)
                or not _plain(lin, nn.Linear) or not _idle(mods["drop"])):
            return NotImplemented
        norm, rows, proj = ln._parameters, slow._parameters, lin._parameters
        if rows.get("bias") is not None or proj.get("bias") is not None:
            return NotImplemented
        return L.host().ff_step(x, norm.get("weight"), norm.get("bias"), ln.eps, rows.get("weight"), W, self.norm_eps,
                                zero_init, proj.get("weight"))

    def forward(self, x):
        if not torch.is_grad_enabled():
            W = torch.empty(x.shape[1], self.num_head, self.dim_head, self.dim_head, device=x.device)
            r = self._step(x, W, True)
            if r is not NotImplemented:
                return r[0]
        rows = self._rows(x)
        W = torch.empty(rows.shape[0], self.num_head, self.dim_head, self.dim_head, device=x.device)
        out = delta_layer(rows, W, norm_eps=self.norm_eps, zero_init=True)
        return _project(self.out_linear, self.drop, _merge(out), x)


class FastFFlayerRL(FastFFlayer):
    """The agents' variant: 1e-5 in the normalisers, the fast weights are the carried state
    (given, updated in place by the call, returned as a copy)."""

    norm_eps = 1e-5

    def forward(self, x, state=None):
        assert state is not None
        r = self._step(x, state, False)
        if r is not NotImplemented:
            return r
        out = delta_layer(self._rows(x), state, norm_eps=self.norm_eps)
        return _project(self.out_linear, self.drop, _merge(out), x), state.clone()

