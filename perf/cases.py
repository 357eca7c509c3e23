"""The work this runtime does for its users, as cases that can be timed and compared.

Everything goes through the public entry points: builtin programs on `DeviceExecutor` (what a compiled
graph becomes) and single builtins on `DeviceBuiltins`.  The families, and the range each stands for:

  builtins   the eight elementwise builtins called one by one on resident vectors, 2^12 ... 2^26 elements
  chain      the elementwise graph sigmoid((a + b) * c / d), 2^10 ... 2^25 elements
  logreg     a logistic-regression training step, batch 32 ... 8192, 13 ... 1024 features
  mlp        a training step of the 2-layer MLP, from a few hundred rows of a small ragged network to the
             65536 x 784-4096-10 step; as the graph compiler's builtin chain or with the fused builtins
  forward    inference with the same MLP on 1 ... 512 rows
  matmul     one fmatmul, all four transpose forms, dimensions 48 ... 8192, aligned and not (products with
             an unaligned dimension up to 2^34 multiply-adds: the large ones are layer-shaped)
  image      convolution -> ReLU -> pooling -> softmax of one single-channel image, 28^2 ... 2048^2 pixels

All tensors are float32, the only type the builtins take.
"""
import math

import torch

from __graft_entry__ import load_package

load_package()
from polarai_framework_b200.device_builtins import DeviceBuiltins, matmul_dims  # noqa: E402
from polarai_framework_b200.program import (DeviceExecutor, Program, elementwise_chain_program,  # noqa: E402
                                            fuse_program, logreg_program, mlp_program)

DEVICE = "cuda:0"


def listed():
    return [
        # single builtins on vectors that fit every cache: what one call costs
        {"name": "builtins_2pow16", "kind": "builtins", "n": 1 << 16},
        # the same calls as streams through HBM, the large end of the bandwidth sweep
        {"name": "builtins_2pow26", "kind": "builtins", "n": 1 << 26},
        # the small elementwise graph of the benchmark configurations
        {"name": "chain_2pow20", "kind": "chain", "n": 1 << 20},
        # the logistic-regression configuration, one launch per builtin as the graph compiler emits it
        {"name": "logreg_256x784", "kind": "logreg", "batch": 256, "n_in": 784, "fused": False},
        # the headline configuration: the full-batch step on one GPU
        {"name": "mlp_65536", "kind": "mlp", "batch": 65536, "n_in": 784, "n_hidden": 4096, "n_out": 10, "fused": True},
        # one GPU's share of that step when eight GPUs split the batch
        {"name": "mlp_8192", "kind": "mlp", "batch": 8192, "n_in": 784, "n_hidden": 4096, "n_out": 10, "fused": True},
        # a small network whose sizes are no multiples of anything, as the unfused builtin chain
        {"name": "mlp_ragged", "kind": "mlp", "batch": 999, "n_in": 301, "n_hidden": 514, "n_out": 7, "fused": False},
        # inference on a handful of rows
        {"name": "forward_16", "kind": "forward", "batch": 16, "n_in": 784, "n_hidden": 4096, "n_out": 10},
        # the matmul sweep: its largest and its smallest square
        {"name": "matmul_8192", "kind": "matmul", "tl": 0, "tr": 0, "m": 8192, "n": 8192, "k": 8192},
        {"name": "matmul_1024_tt", "kind": "matmul", "tl": 1, "tr": 1, "m": 1024, "n": 1024, "k": 1024},
        # a product with no aligned dimension
        {"name": "matmul_ragged_tf", "kind": "matmul", "tl": 1, "tr": 0, "m": 2001, "n": 1511, "k": 999},
        # the remaining operations of the catalogue on one picture
        {"name": "image_1024x768", "kind": "image", "h": 1024, "w": 768, "ksize": 5, "window": 2},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _dim(rng, lo, hi):
    """A matrix dimension: half of them multiples of 16, as layer widths usually are, half as they come."""
    v = _log(rng, lo, hi)
    return max(16, (v + 8) // 16 * 16) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["builtins", "chain", "logreg", "mlp", "forward", "matmul", "matmul", "image"])
    if kind == "builtins":
        return {"kind": kind, "n": _log(rng, 1 << 12, 1 << 26)}
    if kind == "chain":
        return {"kind": kind, "n": _log(rng, 1 << 10, 1 << 25)}
    if kind == "logreg":
        return {"kind": kind, "batch": _log(rng, 32, 8192), "n_in": _log(rng, 13, 1024), "fused": rng.random() < 0.5}
    if kind == "mlp":
        fused = rng.random() < 0.5
        if rng.random() < 0.5:                               # the benchmark's network, any batch
            return {"kind": kind, "batch": _dim(rng, 256, 65536 if fused else 32768), "n_in": 784, "n_hidden": 4096,
                    "n_out": 10, "fused": fused}
        return {"kind": kind, "batch": _dim(rng, 128, 8192), "n_in": _dim(rng, 16, 512),
                "n_hidden": _dim(rng, 64, 1024), "n_out": rng.randint(1, 16), "fused": fused}
    if kind == "forward":
        return {"kind": kind, "batch": _log(rng, 1, 512), "n_in": rng.choice([784, _dim(rng, 64, 1024)]),
                "n_hidden": rng.choice([4096, _dim(rng, 256, 4096)]), "n_out": 10}
    if kind == "matmul":
        tl, tr, dims = rng.randint(0, 1), rng.randint(0, 1), [_dim(rng, 48, 8192) for _ in range(3)]
        while any(d % 4 for d in dims) and math.prod(dims) > 1 << 34:
            i = dims.index(max(dims))
            dims[i] //= 2
        return {"kind": kind, "tl": tl, "tr": tr, "m": dims[0], "n": dims[1], "k": dims[2]}
    return {"kind": kind, "h": _log(rng, 28, 2048), "w": _log(rng, 28, 2048), "ksize": rng.choice([3, 5, 7]),
            "window": rng.choice([2, 3])}


# ---- inputs

def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _uniform(g, shape, lo, hi):
    return torch.empty(shape, device=DEVICE).uniform_(lo, hi, generator=g)


def _xavier(g, n_in, n_out):
    a = math.sqrt(6.0 / (n_in + n_out))
    return _uniform(g, (n_in, n_out), -a, a)


def _one_hot(g, batch, classes):
    if classes == 1:
        return torch.randint(0, 2, (batch, 1), device=DEVICE, generator=g).float()
    labels = torch.randint(0, classes, (batch,), device=DEVICE, generator=g)
    return torch.nn.functional.one_hot(labels, classes).float()


def _forward_program(batch, n_in, n_hidden, n_out):
    """The forward half of the 2-layer MLP: the activations of both layers."""
    p = Program("mlp_forward")
    p.tensor("X", batch, n_in), p.tensor("W1", n_in, n_hidden), p.tensor("W2", n_hidden, n_out)
    p.inputs = ["X", "W1", "W2"]
    p.tensor("Z1", batch, n_hidden), p.tensor("H", batch, n_hidden)
    p.tensor("Z2", batch, n_out), p.tensor("P", batch, n_out)
    p.op("fmatmul_f_f", "X", "W1", "Z1")
    p.op("fsigmoid", "Z1", "H")
    p.op("fmatmul_f_f", "H", "W2", "Z2")
    p.op("fsigmoid", "Z2", "P")
    p.outputs = ["H", "P"]
    return p


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "builtins":
        n = case["n"]
        s = {"case": case, "d": DeviceBuiltins(), "a": _uniform(g, n, -1, 1), "b": _uniform(g, n, -1, 1),
             "den": _uniform(g, n, 0.5, 2), "x": _uniform(g, n, -6, 6), "p": _uniform(g, n, 0.01, 0.99),
             "y": torch.randint(0, 2, (n,), device=DEVICE, generator=g).float(), "g": _uniform(g, 1, -1, 1)}
        s["fill"] = float(seed % 1009) / 8
        s["out"] = {k: torch.empty(n, device=DEVICE) for k in
                    ("fill", "copy", "add", "mul", "divide", "sigmoid", "logloss", "mulconcat")}
        return s
    if kind == "matmul":
        tl, tr, m, n, k = (case[x] for x in ("tl", "tr", "m", "n", "k"))
        left, right = _uniform(g, (k, m) if tl else (m, k), -1, 1), _uniform(g, (n, k) if tr else (k, n), -1, 1)
        m, n, k = matmul_dims(tl, tr, left.shape, right.shape)
        return {"case": case, "d": DeviceBuiltins(), "left": left, "right": right,
                "out": torch.empty((m, n), device=DEVICE)}
    if kind == "image":
        h, w, k, win = case["h"], case["w"], case["ksize"], case["window"]
        ch, cw = h - k + 1, w - k + 1
        ph, pw = (ch - win) // win + 1, (cw - win) // win + 1
        new = lambda *s: torch.empty(s, device=DEVICE)  # noqa: E731
        return {"case": case, "d": DeviceBuiltins(), "image": _uniform(g, (h, w), 0, 1),
                "kernel": _uniform(g, (k, k), -0.5, 0.5), "conv": new(ch, cw), "relu": new(ch, cw),
                "pool": new(ph, pw), "softmax": new(ph, pw)}
    if kind == "chain":
        ex = DeviceExecutor(elementwise_chain_program(case["n"]), DEVICE)
        ins = {t: _uniform(g, case["n"], -1, 1) for t in "abc"}
        ins["d"] = _uniform(g, case["n"], 0.5, 2)
        ex.set_inputs(**ins)
        return {"case": case, "ex": ex}
    if kind == "logreg":
        # the gradient is a sum over the batch; the rate is the usual one for its mean
        prog = logreg_program(case["batch"], case["n_in"], 0.1 / case["batch"])
        ex = DeviceExecutor(fuse_program(prog) if case["fused"] else prog, DEVICE)
        ex.set_inputs(X=torch.randn((case["batch"], case["n_in"]), device=DEVICE, generator=g),
                      W=torch.randn((case["n_in"], 1), device=DEVICE, generator=g) * 0.1,
                      Y=_one_hot(g, case["batch"], 1))
        return {"case": case, "ex": ex}
    b, i, h, o = (case[x] for x in ("batch", "n_in", "n_hidden", "n_out"))
    if kind == "mlp":
        prog = mlp_program(b, i, h, o, 0.1 / b)
        ex = DeviceExecutor(fuse_program(prog) if case["fused"] else prog, DEVICE)
        ex.set_inputs(X=torch.randn((b, i), device=DEVICE, generator=g), Y=_one_hot(g, b, o),
                      W1=_xavier(g, i, h), W2=_xavier(g, h, o))
    else:
        ex = DeviceExecutor(fuse_program(_forward_program(b, i, h, o)), DEVICE)
        ex.set_inputs(X=torch.randn((b, i), device=DEVICE, generator=g), W1=_xavier(g, i, h), W2=_xavier(g, h, o))
    return {"case": case, "ex": ex}


# ---- one pass

def run(state):
    if "ex" in state:                                        # a program: a training step, a graph, an inference
        ex = state["ex"]
        ex.run()
        return {name: ex.t[name] for name in ex.program.outputs}
    d, case = state["d"], state["case"]
    if case["kind"] == "matmul":
        return d.fmatmul(case["tl"], case["tr"], state["left"], state["right"], state["out"])
    if case["kind"] == "image":
        d.fconv2d(state["image"], state["kernel"], state["conv"])
        d.frelu(state["conv"], state["relu"])
        d.fpool(state["relu"], (case["window"],) * 2, (case["window"],) * 2, state["pool"])
        d.fsoftmax(state["pool"], state["softmax"])
        return {k: state[k] for k in ("conv", "relu", "pool", "softmax")}
    o = state["out"]
    d.ffill(state["fill"], o["fill"])
    d.fcopy(state["a"], o["copy"])
    d.fadd(state["a"], 0.34, state["b"], -0.21, o["add"])
    d.fmul(state["a"], state["b"], o["mul"])
    d.fdivide(state["a"], state["den"], o["divide"])
    d.fsigmoid(state["x"], o["sigmoid"])
    d.flogloss(state["p"], state["y"], o["logloss"])
    d.fmulconcat(state["g"], state["a"], o["mulconcat"])
    return o


# ---- what a pass cannot do without, and how closely two correct passes agree

def work(case):
    kind = case["kind"]
    if kind == "builtins":
        return {"bytes": 4 * 14 * case["n"], "flops": 0}     # a, b, den, x, p, y read, eight results written
    if kind == "chain":
        return {"bytes": 4 * 5 * case["n"], "flops": 0}
    if kind == "logreg":
        b, i = case["batch"], case["n_in"]
        return {"bytes": 4 * (b * i + 2 * b + 3 * i), "flops": 4 * b * i}
    if kind == "matmul":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4 * (m * k + k * n + m * n), "flops": 2 * m * n * k}
    if kind == "image":
        ch, cw = case["h"] - case["ksize"] + 1, case["w"] - case["ksize"] + 1
        pooled = ((ch - case["window"]) // case["window"] + 1) * ((cw - case["window"]) // case["window"] + 1)
        return {"bytes": 4 * (case["h"] * case["w"] + 2 * ch * cw + 2 * pooled),
                "flops": 2 * ch * cw * case["ksize"] ** 2}
    b, i, h, o = (case[x] for x in ("batch", "n_in", "n_hidden", "n_out"))
    if kind == "forward":
        return {"bytes": 4 * (b * i + i * h + h * o + b * h + b * o), "flops": 2 * b * (i * h + h * o)}
    return {"bytes": 4 * (b * i + 2 * b * o + 3 * (i * h + h * o)), "flops": 2 * b * (2 * i * h + 3 * h * o)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("builtins", "chain"):
        return {"rel": 1e-6, "max": 1e-5}                    # one rounded operation; the exponential and the logarithm
    if kind == "image":
        return {"rel": 1e-6, "max": 1e-5}                    # 9 to 49 products in a fixed order; the exponential
    # sums of k products in float32.  The tensor core's accumulator rounds toward zero, so the error of a
    # sum of zero-mean products grows with k (measured against float64: 2e-9 to 9e-9 of the result per term).
    k = {"matmul": lambda: case["k"], "logreg": lambda: max(case["batch"], case["n_in"])}.get(
        kind, lambda: max(case["batch"], case["n_in"], case["n_hidden"]))()
    return {"rel": max(1e-5, 1e-8 * k)}
