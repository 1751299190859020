"""What the framework is timed on: the calls that programs written against it make, at sizes from the smallest to the largest.

A case names a kind of call and its sizes.  `prepare` makes what such a program holds before the call (inputs, weights, a
bound graph), `run` makes the call through the public entry points, `exact` computes the same outputs in 64 bits with plain
torch, `work` counts the bytes and operations that the call cannot do without.

Kinds
  step       one training step through the graph API: dispatch_forward, dispatch_loss, dispatch_backward, dispatch_optim
  dense      the forward pass of one dense layer on f32 tensors: act(x W + b)
  dense_bwd  its backward pass: the gradients of x, W and b from dL/dy
  layer16    forward and backward of one dense layer on 16-bit tensors
  batched    forward and backward of a rank-3 product: T independent [M,K] x [K,N]
  softmax    row softmax, forward and backward
  ce         fused softmax + cross-entropy: loss, probabilities' gradient and the predicted class
  chain      a fused elementwise program, forward and backward, in any of the three storage types
"""
import math

import numpy as np
import torch

from ferrograd_b200 import GpuContext
from ferrograd_b200.mlp import GraphMLP

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
ADAMW = ("adamw", 1e-3, 0.9, 0.999, 1e-8, 0.01)
SGD = ("sgd", 1e-3)

# Elementwise programs: (op, operand, operand, constant) per instruction, operands are earlier instructions' indices.
PROGRAMS = {
    # the benchmark's chain: gelu(x * y) + x
    "gate": [("input", 0, 0, 0.0), ("input", 1, 0, 0.0), ("mul", 0, 1, 0.0), ("gelu", 2, 0, 0.0), ("add", 3, 0, 0.0)],
    # the smallest useful one: tanh(x + y)
    "add_tanh": [("input", 0, 0, 0.0), ("input", 1, 0, 0.0), ("add", 0, 1, 0.0), ("tanh", 2, 0, 0.0)],
    # x / (1 + exp(-x)) * y, spelled out in primitive operations
    "swish": [("input", 0, 0, 0.0), ("neg", 0, 0, 0.0), ("exp", 1, 0, 0.0), ("const", 0, 0, 1.0), ("add", 2, 3, 0.0),
              ("div", 0, 4, 0.0), ("input", 1, 0, 0.0), ("mul", 5, 6, 0.0)],
    # a residual with an elu and a scale: elu(x - y) * 0.5 + y
    "elu_residual": [("input", 0, 0, 0.0), ("input", 1, 0, 0.0), ("sub", 0, 1, 0.0), ("elu", 2, 0, 0.0),
                     ("const", 0, 0, 0.5), ("mul", 3, 4, 0.0), ("add", 5, 1, 0.0)],
}


def listed():
    return [
        # the 2-16-2 network of the smallest benchmark workload: nothing but launches
        {"name": "step_tiny", "kind": "step", "dims": "2-16-2", "batch": 64, "act": "tanh", "loss": "mse", "opt": "sgd"},
        # the network of the smoke run: a small classifier, kernels of a few microseconds
        {"name": "step_small", "kind": "step", "dims": "200-256-256-10", "batch": 384, "act": "gelu", "loss": "ce", "opt": "adamw"},
        # the headline workload: a full training step at 4096 samples
        {"name": "step_mlp", "kind": "step", "dims": "784-4096-4096-10", "batch": 4096, "act": "gelu", "loss": "ce", "opt": "adamw"},
        # the largest matrix product of the benchmark
        {"name": "dense_large", "kind": "dense", "m": 8192, "k": 8192, "n": 8192, "act": "relu"},
        # inference of a hundred requests through one wide layer: bound by reading the weights
        {"name": "dense_serve", "kind": "dense", "m": 100, "k": 4096, "n": 4096, "act": "gelu"},
        # a layer whose sizes are multiples of nothing, backward
        {"name": "dense_bwd_ragged", "kind": "dense_bwd", "m": 1000, "k": 777, "n": 1001, "act": "tanh"},
        # 16-bit storage: one hidden layer of a large network, forward and backward
        {"name": "layer_bf16", "kind": "layer16", "dtype": "bf16", "m": 2048, "k": 4096, "n": 4096, "act": "gelu"},
        # a rank-3 product of middling matrices, forward and backward
        {"name": "batched", "kind": "batched", "t": 16, "m": 384, "k": 512, "n": 320},
        # row softmax over an odd number of columns
        {"name": "softmax_ragged", "kind": "softmax", "rows": 4096, "cols": 10001},
        # the loss of the benchmark's 32000-class workload
        {"name": "softmax_ce", "kind": "ce", "rows": 8192, "cols": 32000},
        # a fused elementwise region of a graph, on tensors larger than the L2
        {"name": "chain_f32", "kind": "chain", "dtype": "f32", "n": 32 << 20, "program": "gate"},
        # the same on half-precision tensors of an odd length
        {"name": "chain_f16", "kind": "chain", "dtype": "f16", "n": 3000001, "program": "swish"},
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi]: any whole number, or a multiple of 8 or 64."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    g = rng.choice((1, 8, 64))
    return max(lo, min(hi, (v + g - 1) // g * g if v >= g else v))


def draw(rng):
    kind = rng.choice(("step", "dense", "dense_bwd", "layer16", "batched", "softmax", "ce", "chain"))
    act = rng.choice(("relu", "tanh", "gelu"))
    if kind == "step":
        hidden = [_size(rng, 16, 4096) for _ in range(rng.choice((1, 2, 2, 3)))]
        dims = [_size(rng, 2, 1024)] + hidden + [rng.randint(2, 100)]
        return {"kind": kind, "dims": "-".join(map(str, dims)), "batch": _size(rng, 32, 4096), "act": act,
                "loss": rng.choice(("ce", "mse")), "opt": rng.choice(("adamw", "sgd"))}
    if kind == "dense":
        return {"kind": kind, "m": _size(rng, 1, 8192), "k": _size(rng, 32, 8192), "n": _size(rng, 8, 8192), "act": act}
    if kind == "dense_bwd":
        return {"kind": kind, "m": _size(rng, 32, 4096), "k": _size(rng, 32, 4096), "n": _size(rng, 8, 4096), "act": act}
    if kind == "layer16":
        return {"kind": kind, "dtype": rng.choice(("bf16", "f16")), "m": _size(rng, 64, 4096), "k": _size(rng, 64, 4096),
                "n": _size(rng, 64, 4096), "act": act}
    if kind == "batched":
        return {"kind": kind, "t": rng.randint(2, 32), "m": _size(rng, 16, 512), "k": _size(rng, 16, 512), "n": _size(rng, 16, 512)}
    if kind == "softmax":
        cols = _size(rng, 10, 32768)
        return {"kind": kind, "rows": min(_size(rng, 32, 16384), max(32, 60_000_000 // cols)), "cols": cols}
    if kind == "ce":
        return {"kind": kind, "rows": _size(rng, 32, 8192), "cols": _size(rng, 10, 32000)}
    return {"kind": kind, "dtype": rng.choice(("f32", "f16", "bf16")), "n": _size(rng, 1000, 32 << 20),
            "program": rng.choice(sorted(PROGRAMS))}


# ---- inputs ----
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + 17)


def _normal(gen, shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=gen, device="cuda") * scale).to(dtype)


def _saved(gen, shape, act, dtype=torch.float32):
    """What the forward pass keeps for the backward pass: the output for relu and tanh, the pre-activation for gelu."""
    z = torch.randn(shape, generator=gen, device="cuda")
    return (torch.relu(z) if act == "relu" else torch.tanh(z) if act == "tanh" else z).to(dtype)


def _dims(case):
    return [int(d) for d in case["dims"].split("-")]


def _inputs(case, seed):
    """The input tensors of a case, a function of the seed alone."""
    gen, kind = _gen(seed), case["kind"]
    if kind == "step":
        dims, batch = _dims(case), case["batch"]
        t = {"x": torch.rand((batch, dims[0]), generator=gen, device="cuda") if case["loss"] == "ce" else _normal(gen, (batch, dims[0]))}
        if case["loss"] == "ce":
            t["target"] = torch.randint(0, dims[-1], (batch,), generator=gen, device="cuda").int()
        else:
            t["target"] = _normal(gen, (batch, dims[-1]))
        t["W"] = [_normal(gen, (a, b), math.sqrt(2.0 / a)) for a, b in zip(dims, dims[1:])]
        t["b"] = [_normal(gen, (b,), 0.1) for b in dims[1:]]
        return t
    if kind in ("dense", "dense_bwd", "layer16"):
        m, k, n, act = case["m"], case["k"], case["n"], case["act"]
        dt = DTYPES[case.get("dtype", "f32")]
        t = {"x": _normal(gen, (m, k), 1.0, dt), "w": _normal(gen, (k, n), k ** -0.5, dt), "b": _normal(gen, (n,), 0.1, dt)}
        if kind != "dense":
            t["dy"] = _normal(gen, (m, n), 1.0, dt)
        if kind == "dense_bwd":
            t["saved"] = _saved(gen, (m, n), act)
        return t
    if kind == "batched":
        t, m, k, n = (case[c] for c in "tmkn")
        return {"a": _normal(gen, (t, m, k)), "b": _normal(gen, (t, k, n), k ** -0.5), "dy": _normal(gen, (t, m, n))}
    if kind == "softmax":
        return {"x": _normal(gen, (case["rows"], case["cols"]), 2.0), "dy": _normal(gen, (case["rows"], case["cols"]))}
    if kind == "ce":
        return {"x": _normal(gen, (case["rows"], case["cols"]), 2.0),
                "labels": torch.randint(0, case["cols"], (case["rows"],), generator=gen, device="cuda").int()}
    dt = DTYPES[case["dtype"]]
    return {"in": [_normal(gen, (case["n"],), 1.0, dt) for _ in range(2)], "seed": _normal(gen, (case["n"],), 1.0, dt)}


_context = None


def _ctx():
    """One context per process, as a program has."""
    global _context
    if _context is None:
        _context = GpuContext(0)
    return _context


class _DeviceArray:
    """A buffer of the framework for torch.as_tensor, without a copy; the tensor keeps `owner` alive."""

    def __init__(self, buf, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (buf.ptr, False), "shape": tuple(shape), "typestr": typestr, "version": 2}


class _Net:
    """A bound graph with its weights; its device buffers go when neither the state nor an output refers to it."""

    def __init__(self, case, t):
        self.net = GraphMLP(_ctx(), _dims(case), case["batch"], case["act"], case["loss"], ADAMW if case["opt"] == "adamw" else SGD)
        self.net.set_params([w.cpu().numpy() for w in t["W"]], [b.cpu().numpy() for b in t["b"]])
        self.net.upload_batch(t["x"].cpu().numpy(), t["target"].cpu().numpy().view(np.uint32 if case["loss"] == "ce" else np.float32))

    def outputs(self):
        n = self.net
        view = lambda buf, shape: torch.as_tensor(_DeviceArray(buf, shape, "<f4", self), device="cuda")   # noqa: E731
        out = (n.batch, n.dims[-1])
        return {"prediction": view(n.tensors.forward_out, out), "loss": view(n.tensors.loss_t.data, out), "loss_sum": view(n.loss_out, (1,)),
                "W": [view(w.data, w.shape) for w in n.W], "b": [view(v.data, v.shape) for v in n.b]}

    def __del__(self):
        _ctx().sync()
        self.net.destroy()


def prepare(case, seed):
    ctx, kind, t = _ctx(), case["kind"], _inputs(case, seed)
    if kind == "step":
        net = _Net(case, t)
        state = {"net": net.net, "out": net.outputs()}
    else:
        like = lambda *names: {"d" + k: torch.empty_like(t[k]) for k in names}   # noqa: E731
        state = {"in": t}
        if kind == "dense":
            state["out"] = {"y": torch.empty((case["m"], case["n"]), device="cuda")}
        elif kind == "dense_bwd":
            state["out"] = like("x", "w", "b")
        elif kind == "layer16":
            y = torch.empty_like(t["dy"])
            state["out"] = {"y": y, "z": torch.empty_like(y), **like("x", "w", "b")}
        elif kind == "batched":
            state["out"] = {"y": torch.empty_like(t["dy"]), **like("a", "b")}
        elif kind == "softmax":
            state["out"] = {"y": torch.empty_like(t["x"]), "dx": torch.empty_like(t["x"])}
        elif kind == "ce":
            state["out"] = {"loss_row": torch.empty(case["rows"], device="cuda"), "loss_mean": torch.empty(1, device="cuda"),
                            "dx": torch.empty_like(t["x"]), "argmax": torch.empty(case["rows"], dtype=torch.int32, device="cuda")}
        else:
            state["out"] = {"y": torch.empty_like(t["seed"]), "dx": [torch.empty_like(v) for v in t["in"]]}
    state["case"], state["ctx"] = case, ctx
    torch.cuda.synchronize()
    return state


def run(state):
    case, c = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "step":
        state["net"].step()
        return state["out"]
    t, o = state["in"], state["out"]
    p = lambda v: v.data_ptr()   # noqa: E731
    if kind == "dense":
        c.gemm(p(t["x"]), p(t["w"]), p(o["y"]), case["m"], case["n"], case["k"], bias=p(t["b"]), act=case["act"])
    elif kind == "dense_bwd":
        c.gemm_bwd(p(t["x"]), p(t["w"]), p(t["dy"]), case["m"], case["n"], case["k"], act=case["act"], saved=p(t["saved"]),
                   dA=p(o["dx"]), dB=p(o["dw"]), dbias=p(o["db"]))
    elif kind == "layer16":
        saved = o["z"] if case["act"] == "gelu" else o["y"]
        c.gemm_lowp(p(t["x"]), p(t["w"]), p(o["y"]), case["m"], case["n"], case["k"], case["dtype"], bias=p(t["b"]),
                    act=case["act"], preact_out=p(o["z"]))
        c.gemm_bwd_lowp(p(t["x"]), p(t["w"]), p(t["dy"]), case["m"], case["n"], case["k"], case["dtype"], act=case["act"],
                        saved=p(saved), dA=p(o["dx"]), dB=p(o["dw"]), dbias=p(o["db"]))
    elif kind == "batched":
        c.gemm_batched(p(t["a"]), p(t["b"]), p(o["y"]), case["t"], case["m"], case["n"], case["k"])
        c.gemm_batched_bwd(p(t["a"]), p(t["b"]), p(t["dy"]), case["t"], case["m"], case["n"], case["k"], dA=p(o["da"]), dB=p(o["db"]))
    elif kind == "softmax":
        c.softmax_fwd(p(t["x"]), p(o["y"]), case["rows"], case["cols"])
        c.softmax_bwd(p(o["y"]), p(t["dy"]), p(o["dx"]), case["rows"], case["cols"])
    elif kind == "ce":
        c.softmax_ce(p(t["x"]), p(t["labels"]), case["rows"], case["cols"], grad_scale=1.0 / case["rows"], loss_row=p(o["loss_row"]),
                     loss_mean=p(o["loss_mean"]), dlogits=p(o["dx"]), argmax=p(o["argmax"]))
    else:
        prog, ins = PROGRAMS[case["program"]], [p(v) for v in t["in"]]
        c.eltwise_chain_fwd(prog, ins, p(o["y"]), case["n"], dtype=case["dtype"])
        c.eltwise_chain_bwd(prog, ins, p(t["seed"]), [p(v) for v in o["dx"]], case["n"], dtype=case["dtype"])
    return o


# ---- what a call cannot do without ----
def work(case):
    """Bytes: every input read once, every output written once.  flops: two per multiply-add of the matrix products, or the
    instructions of an elementwise program."""
    kind = case["kind"]
    if kind == "step":
        dims, batch = _dims(case), case["batch"]
        params = sum(a * b + b for a, b in zip(dims, dims[1:]))
        flops = sum(2 * batch * a * b * (3 if i else 2) for i, (a, b) in enumerate(zip(dims, dims[1:])))
        # parameters: read for the products, read and written by the update; adamw keeps two moments beside them.  The
        # activations of every layer are written by the forward pass and read by the backward pass.
        per_param = 12 + (16 if case["opt"] == "adamw" else 0)
        return {"bytes": per_param * params + 4 * batch * (dims[0] + 2 * sum(dims[1:])), "flops": flops}
    if kind in ("dense", "dense_bwd", "layer16"):
        m, k, n = case["m"], case["k"], case["n"]
        x, w, y = m * k, k * n, m * n
        if kind == "dense":
            return {"bytes": 4 * (x + w + y + n), "flops": 2 * m * k * n}
        if kind == "dense_bwd":
            return {"bytes": 4 * (2 * x + 2 * w + 2 * y + n), "flops": 4 * m * k * n}
        return {"bytes": 2 * (2 * x + 2 * w + 3 * y + 2 * n), "flops": 6 * m * k * n}
    if kind == "batched":
        t, m, k, n = (case[c] for c in "tmkn")
        return {"bytes": 4 * t * (2 * m * k + 2 * k * n + 2 * m * n), "flops": 6 * t * m * k * n}
    if kind == "softmax":
        return {"bytes": 4 * 4 * case["rows"] * case["cols"], "flops": 9 * case["rows"] * case["cols"]}
    if kind == "ce":
        return {"bytes": 2 * 4 * case["rows"] * case["cols"] + 12 * case["rows"], "flops": 6 * case["rows"] * case["cols"]}
    size = 4 if case["dtype"] == "f32" else 2
    return {"bytes": 6 * size * case["n"], "flops": 3 * len(PROGRAMS[case["program"]]) * case["n"]}


def tolerance(case):
    """About four times the error against 64 bits that was measured over the listed cases and a few drawn ones."""
    kind = case["kind"]
    if kind == "step":
        # An adamw step is lr * g / |g| at first: a gradient near zero moves its weight by up to 2 lr when its sign differs
        # (measured 4.5e-5 after one step of the largest network; several steps are compared).
        return {"rel": 2e-5 if case["opt"] == "sgd" else 1e-3, "max": 0.5}
    if kind in ("dense", "dense_bwd", "batched"):
        return {"rel": 8e-6}                    # f32 products as a split of two tensor-core terms: 1.3e-6 to 1.9e-6
    if kind == "layer16":
        # results, and the gradient of z, rounded to storage: 2.4e-3 in bf16, an eighth of that in f16
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 1.3e-3}
    if kind in ("softmax", "ce"):
        return {"rel": 1e-6, "differ": 1e-3}    # f32: 9e-8 at most; the predicted class of a row only changes at a tie
    return {"f32": {"rel": 1e-6}, "f16": {"rel": 2e-3}, "bf16": {"rel": 1.5e-2}}[case["dtype"]]   # 9.4e-8; 4.5e-4 in f16


# ---- the same outputs in 64 bits ----
_GELU_A, _GELU_B = 0.044715, math.sqrt(2.0 / math.pi)


def _act(act, z):
    if act == "gelu":
        return 0.5 * z * (1.0 + torch.tanh(_GELU_B * (z + _GELU_A * z ** 3)))
    return torch.relu(z) if act == "relu" else torch.tanh(z) if act == "tanh" else z


def _act_grad(act, saved):
    if act == "relu":
        return (saved > 0).double()
    if act == "tanh":
        return 1.0 - saved * saved
    th = torch.tanh(_GELU_B * (saved + _GELU_A * saved ** 3))
    return 0.5 * (1.0 + th) + 0.5 * saved * (1.0 - th * th) * _GELU_B * (1.0 + 3.0 * _GELU_A * saved ** 2)


def _exact_step(case, t):
    dims, act, n = _dims(case), case["act"], len(t["W"])
    f32 = lambda v: float(np.float32(v))   # noqa: E731
    W, b = [w.double() for w in t["W"]], [v.double() for v in t["b"]]
    h, hs, zs = t["x"].double(), [], []
    for l in range(n):
        hs.append(h)
        zs.append(h @ W[l] + b[l])
        h = _act(act, zs[l]) if l < n - 1 else zs[l]
    if case["loss"] == "ce":
        prediction = torch.softmax(h, -1)
        onehot = torch.nn.functional.one_hot(t["target"].long(), dims[-1]).double()
        loss, dz = -torch.log_softmax(h, -1) * onehot, prediction - onehot
    else:
        prediction = h
        loss, dz = (h - t["target"].double()) ** 2, 2.0 * (h - t["target"].double())
    new = {"W": [], "b": []}
    for l in range(n - 1, -1, -1):
        dW, db = hs[l].T @ dz, dz.sum(0)
        if l:
            dz = (dz @ W[l].T) * _act_grad(act, zs[l - 1] if act == "gelu" else hs[l])
        for name, p, g in (("W", W[l], dW), ("b", b[l], db)):
            if case["opt"] == "sgd":
                q = p - f32(SGD[1]) * g
            else:   # the first step: bias-corrected moments are the gradient itself
                _, lr, _, _, eps, wd = ADAMW
                q = p - f32(lr) * (g / (g.abs() + f32(eps)) + f32(wd) * p)
            new[name].insert(0, q)
    return {"prediction": prediction, "loss": loss, "loss_sum": loss.sum().reshape(1), **new}


def _exact_chain(case, t):
    x = [v.double().requires_grad_() for v in t["in"]]
    vals = []
    for op, a, b, imm in PROGRAMS[case["program"]]:
        if op == "input":
            v = x[a]
        elif op == "const":
            v = torch.full_like(x[0], imm)
        elif op in ("add", "sub", "mul", "div"):
            v = getattr(torch, op)(vals[a], vals[b])
        elif op in ("neg", "exp", "tanh"):
            v = getattr(torch, op)(vals[a])
        elif op == "elu":
            v = torch.where(vals[a] >= 0, vals[a], torch.exp(vals[a]) - 1.0)
        else:
            v = _act(op, vals[a])
        vals.append(v)
    grads = torch.autograd.grad(vals[-1], x, t["seed"].double())
    return {"y": vals[-1].detach(), "dx": [g for g in grads]}


def exact(case, seed):
    kind, t = case["kind"], _inputs(case, seed)
    if kind == "step":
        return _exact_step(case, t)
    if kind == "chain":
        return _exact_chain(case, t)
    d = {k: v.double() for k, v in t.items() if v.is_floating_point()}
    if kind == "dense":
        return {"y": _act(case["act"], d["x"] @ d["w"] + d["b"])}
    if kind in ("dense_bwd", "layer16"):
        out = {}
        saved = d.get("saved")
        if kind == "layer16":
            out["z"] = d["x"] @ d["w"] + d["b"]
            out["y"] = _act(case["act"], out["z"])
            saved = out["z"] if case["act"] == "gelu" else out["y"]
        dz = d["dy"] * _act_grad(case["act"], saved)
        return {**out, "dx": dz @ d["w"].T, "dw": d["x"].T @ dz, "db": dz.sum(0)}
    if kind == "batched":
        return {"y": d["a"] @ d["b"], "da": d["dy"] @ d["b"].transpose(1, 2), "db": d["a"].transpose(1, 2) @ d["dy"]}
    if kind == "softmax":
        y = torch.softmax(d["x"], -1)
        return {"y": y, "dx": y * (d["dy"] - (d["dy"] * y).sum(-1, keepdim=True))}
    logp = torch.log_softmax(d["x"], -1)
    labels = t["labels"].long()
    rows = torch.arange(case["rows"], device="cuda")
    loss = -logp[rows, labels]
    dx = torch.exp(logp)
    dx[rows, labels] -= 1.0
    return {"loss_row": loss, "loss_mean": loss.mean().reshape(1), "dx": dx / case["rows"], "argmax": None}
