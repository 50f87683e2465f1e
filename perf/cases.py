"""Cases that stand for what a user of this framework has it do, for timing.

Each case is one pass through the public entry points: the drop-in operators (``self_ref_v0``,
``stateful_self_ref_v0``, ``fast_weight_delta``), the layer-level calls and modules built on them
(``srwm_layer``, ``SRWMlayer``, ``SRlayer``, ``FastFFlayer``) and the captured actor step
(``GraphedSRStep``).  Sizes are those of the benchmark and test configurations (C1..C5 in the
names below), a GPU's share of the scale sweep for the largest, and odd ones in between.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "modern-srwm_b200"))

from srwm_b200 import fast_weight_delta, self_ref_v0, stateful_self_ref_v0  # noqa: E402
from srwm_b200.graphs import GraphedSRStep  # noqa: E402
from srwm_b200.layer_ops import srwm_layer  # noqa: E402
from srwm_b200.layers import FastFFlayer, FastFFlayerRL, SRlayer, SRWMlayer  # noqa: E402


def _case(name, kind, B, H, L, d, dtype="f32"):
    return {"name": name, "kind": kind, "B": B, "H": H, "L": L, "d": d, "dtype": dtype}


def listed():
    return [
        # one environment step of 48 actors through the agents' layer, state carried (C4): host-bound
        _case("actor step", "sr_step", 48, 8, 1, 32),
        # the same step of the two-layer agent as a captured graph
        _case("actor graph", "sr_graph", 48, 8, 1, 32),
        # one step of the delta-rule agents' layer, fast weights carried
        _case("delta actor step", "ff_step", 48, 8, 1, 32),
        # the single-layer operator training step with few, short sequences (C1): latency
        _case("srwm small train", "srwm_train", 4, 4, 64, 16),
        # the learner's unroll with episode resets, forward and backward (C4)
        _case("rl unroll train", "sr_unroll", 32, 8, 100, 32),
        # a few-shot layer's training step, input softmax and layer norm included (C3)
        _case("few-shot layer train", "srwm_layer_train", 128, 16, 128, 32),
        # gradient through a carried state, odd sizes, the largest head
        _case("stateful train", "srwm_stateful", 13, 8, 77, 64),
        # long sequences evaluated without gradients
        _case("srwm eval", "srwm_eval", 16, 16, 1000, 64, "bf16"),
        # the delta-rule operator's training step (C2)
        _case("delta train", "delta_train", 32, 8, 512, 64),
        # the delta-rule layer's training step on its slow net's packed rows
        _case("delta layer train", "ff_layer", 32, 8, 389, 64),
        # one GPU's share of the scale sweep over eight (C5): throughput
        _case("srwm sweep share", "srwm_slow", 128, 16, 2048, 64, "bf16"),
        _case("delta sweep share", "delta_train", 64, 16, 8192, 64, "bf16"),
    ]


# kind -> (head sizes, element types, largest B, largest L); B and L are drawn over their logarithm
_RANGES = {
    "sr_step": ((16, 32, 64), ("f32",), 256, 1),
    "sr_graph": ((16, 32, 64), ("f32",), 256, 1),
    "ff_step": ((16, 32, 64), ("f32",), 256, 1),
    "srwm_train": ((8, 16, 32, 64), ("f32", "bf16"), 64, 512),
    "sr_unroll": ((16, 32, 64), ("f32",), 64, 200),
    "srwm_layer_train": ((16, 32, 64), ("f32",), 128, 256),
    "srwm_stateful": ((8, 16, 32, 64), ("f32",), 64, 256),
    "srwm_eval": ((16, 32, 64), ("f32", "bf16"), 64, 2048),
    "delta_train": ((16, 32, 64), ("f32", "bf16"), 128, 4096),
    "ff_layer": ((16, 32, 64), ("f32", "bf16"), 64, 1024),
    "srwm_slow": ((32, 64), ("f32", "bf16"), 128, 2048),
}
_MIN_L = {"sr_step": 1, "sr_graph": 1, "ff_step": 1}


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(sorted(_RANGES))
        heads, types, b_most, l_most = _RANGES[kind]
        case = {"kind": kind, "B": _log_int(rng, 1, b_most), "H": rng.choice((4, 8, 16)),
                "L": _log_int(rng, _MIN_L.get(kind, 8), l_most), "d": rng.choice(heads), "dtype": rng.choice(types)}
        if work(case)["flops"] <= most and case["B"] * case["H"] * case["L"] * case["d"] <= 1.2e9 / 2:
            return case


def _dt(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float32


class _Rand:
    """Seeded inputs made on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def normal(self, *shape, dtype=torch.float32, scale=1.0):
        t = torch.empty(shape, device="cuda", dtype=torch.float32).normal_(generator=self.g)
        return (t.mul_(scale) if scale != 1.0 else t).to(dtype)

    def softmax(self, *shape, dtype=torch.float32):
        return torch.softmax(self.normal(*shape), -1).to(dtype)

    def sigmoid(self, *shape, dtype=torch.float32):
        return torch.sigmoid(self.normal(*shape)).to(dtype)

    def module(self, m):
        """A module on the GPU whose weights come from the seed: matrices N(0, 1/fan in), small biases."""
        m = m.to("cuda")
        with torch.no_grad():
            for name, p in m.named_parameters():
                if p.dim() > 1:
                    p.copy_(self.normal(*p.shape, scale=p.shape[-1] ** -0.5))
                elif name.endswith("bias"):
                    p.copy_(self.normal(*p.shape, scale=0.02))
        return m

    def slow_weights(self, H, d):
        """The un-repeated [1, H, d, .] slow weights, N(0, 1/d)."""
        return [self.normal(1, H, d, w, scale=d ** -0.5) for w in (d, d, d, 4)]

    def shift(self, B, H, d):
        """A carried state: what some steps have added to the slow weights."""
        return tuple(self.normal(B, H, d, w, scale=0.1 * d ** -0.5) for w in (d, d, d, 4))


def prepare(case, seed):
    r = _Rand(seed)
    B, H, L, d, kind = (case[k] for k in ("B", "H", "L", "d", "kind"))
    dt = _dt(case)
    s = {"kind": kind, "B": B}
    dim = H * d
    if kind in ("sr_step", "sr_graph", "sr_unroll"):
        s["h"] = r.normal(L, B, dim)
        s["state"] = r.shift(B, H, d)
        s["net"] = r.module(SRlayer(H, d, dim, 0.0))
        if kind == "sr_graph":
            blocks = []
            for net in (s["net"], r.module(SRlayer(H, d, dim, 0.0))):
                ff = torch.nn.Sequential(torch.nn.LayerNorm(dim), torch.nn.Linear(dim, 2 * dim), torch.nn.ReLU(),
                                         torch.nn.Linear(2 * dim, dim))
                blocks.append((net, r.module(ff)))
            s["step"] = GraphedSRStep(blocks, [s["state"], r.shift(B, H, d)], s["h"])
        if kind == "sr_unroll":
            s["h"].requires_grad_()
            s["gout"] = r.normal(L, B, dim)
            s["done"] = torch.rand(L, B, device="cuda", generator=r.g) < 0.02   # an episode ends now and then
    elif kind == "srwm_layer_train":
        s["h"] = r.normal(L, B, dim).requires_grad_()
        s["gout"] = r.normal(L, B, dim)
        s["net"] = r.module(SRWMlayer(H, d, dim, 0.0, use_ln=True, use_input_softmax=True))
    elif kind in ("ff_step", "ff_layer"):
        s["h"] = r.normal(L, B, dim, dtype=dt)
        s["net"] = r.module((FastFFlayerRL if kind == "ff_step" else FastFFlayer)(H, d, dim, 0.0)).to(dt)
        if kind == "ff_step":
            s["W"] = r.normal(B, H, d, d, scale=0.1)
        else:
            s["h"].requires_grad_()
            s["gout"] = r.normal(L, B, dim, dtype=dt)
    elif kind == "delta_train":
        s["qkvb"] = [t.requires_grad_() for t in (r.softmax(B, H, L, d, dtype=dt), r.softmax(B, H, L, d, dtype=dt),
                                                  r.normal(B, H, L, d, dtype=dt), r.sigmoid(B, H, L, 1, dtype=dt))]
        s["gout"] = r.normal(B, H, L, d, dtype=dt)
    else:
        s["x"] = r.normal(B, H, L, d, dtype=dt)
        s["W"] = r.slow_weights(H, d)
        if kind == "srwm_eval":
            s["x"] = torch.softmax(s["x"].float(), -1).to(dt)
        else:
            s["gout"] = r.normal(B, H, L, d, dtype=dt)
            for t in [s["x"]] + s["W"]:
                t.requires_grad_()
        if kind == "srwm_stateful":
            s["state"] = tuple(t.requires_grad_() for t in r.shift(B, H, d))
            s["gstate"] = r.shift(B, H, d)
    return s


def run(s):
    kind, B = s["kind"], s["B"]
    if kind == "sr_step":
        with torch.no_grad():
            return s["net"](s["h"], s["state"])
    if kind == "sr_graph":
        return s["step"](s["h"]), s["step"].state       # the state advances in place
    if kind == "ff_step":
        with torch.no_grad():
            return s["net"](s["h"], s["W"])             # so do the fast weights
    if kind == "sr_unroll":
        out, state = s["net"].unroll(s["h"], s["done"], s["state"])
        params = list(s["net"].parameters())
        return out, state, torch.autograd.grad(out, [s["h"]] + params, s["gout"], allow_unused=True)
    if kind in ("srwm_layer_train", "ff_layer"):
        out = s["net"](s["h"])
        return out, torch.autograd.grad(out, [s["h"]] + list(s["net"].parameters()), s["gout"])
    if kind == "delta_train":
        q = s["qkvb"][0]
        W = torch.zeros(q.shape[0], q.shape[1], q.shape[3], q.shape[3], device=q.device)
        out = fast_weight_delta(*s["qkvb"], W)
        return out, torch.autograd.grad(out, s["qkvb"], s["gout"])
    if kind == "srwm_slow":
        out, state = srwm_layer(s["x"], *s["W"], input_softmax=False)
        return out, [t.detach() for t in state], torch.autograd.grad(out, [s["x"]] + s["W"], s["gout"])
    # the operators take per-sample weights, repeated by the caller, and leave the final state in them
    W = [w.repeat(B, 1, 1, 1) for w in s["W"]]
    if kind == "srwm_eval":
        with torch.no_grad():
            return self_ref_v0(s["x"], *W), W
    if kind == "srwm_train":
        out = self_ref_v0(s["x"], *W)
        return out, [w.detach() for w in W], torch.autograd.grad(out, [s["x"]] + s["W"], s["gout"])
    W = [w + t for w, t in zip(W, s["state"])]
    out, *state = stateful_self_ref_v0(s["x"], *W)
    grads = torch.autograd.grad([out] + state, [s["x"]] + s["W"] + list(s["state"]), [s["gout"]] + list(s["gstate"]))
    return out, [t.detach() for t in state], grads


def work(case):
    """One pass: inputs read once, outputs written once; the recurrence's multiply-adds (a matrix-vector
    product per pass over the state) and the modules' matrix products."""
    B, H, L, d, kind = (case[k] for k in ("B", "H", "L", "d", "kind"))
    s = 2 if case["dtype"] == "bf16" else 4
    n, dim, D = B * H, H * d, 3 * d + 4
    rows = n * L
    srwm_state, delta_state = 4 * d * D, 4 * d * d        # bytes of one sequence's state
    slow = H * srwm_state
    if kind in ("sr_step", "sr_graph"):
        layers = 2 if kind == "sr_graph" else 1
        ff = 4 * dim * dim if kind == "sr_graph" else 0
        return {"bytes": layers * (2 * rows * d * s + 2 * n * srwm_state + slow + 4 * (dim * dim + ff)),
                "flops": layers * (6 * rows * d * D + 2 * B * L * (dim * dim + ff))}
    if kind == "ff_step":
        wide = H * (3 * d + 1)
        return {"bytes": 2 * rows * d * s + 3 * n * delta_state + 4 * dim * (dim + wide),
                "flops": 6 * rows * d * d + 2 * B * L * dim * (dim + wide)}
    if kind == "sr_unroll":
        return {"bytes": 4 * rows * d * s + 2 * n * srwm_state + 2 * slow + 2 * 4 * dim * dim,
                "flops": 6 * rows * d * D + 6 * rows * d * d + 6 * B * L * dim * dim}
    if kind == "srwm_layer_train":
        return {"bytes": 4 * rows * d * s + 2 * slow + 2 * 4 * dim * dim,
                "flops": 20 * rows * d * D + 6 * B * L * dim * dim}
    if kind == "ff_layer":
        wide = H * (3 * d + 1)
        return {"bytes": 4 * rows * d * s + 2 * s * dim * (dim + wide),
                "flops": 20 * rows * d * d + 6 * B * L * dim * (dim + wide)}
    if kind == "delta_train":
        return {"bytes": rows * (8 * d + 2) * s, "flops": 20 * rows * d * d}
    if kind == "srwm_eval":
        return {"bytes": 2 * rows * d * s + n * srwm_state + slow, "flops": 6 * rows * d * D}
    carried = n * srwm_state * {"srwm_train": 1, "srwm_slow": 1, "srwm_stateful": 4}[kind]
    return {"bytes": 4 * rows * d * s + 2 * slow + carried, "flops": 20 * rows * d * D}


def tolerance(case):
    """bf16 streams round every output to 8 bits; float32 rounding adds up along a sequence."""
    if case["dtype"] == "bf16":
        return {"rel": 1e-2, "max": 0.2}
    rel = 1e-5 * max(1.0, case["L"] / 256)
    return {"rel": min(rel, 1e-4), "max": min(40 * rel, 4e-3)}
