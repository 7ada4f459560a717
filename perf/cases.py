"""The work that programs on this back end do, as cases that can be timed and compared.

Two forms: one iteration of a training program's loop (`DeviceProgram.step_fed`, the input tensors already written), and
one call of a compiled function whose arguments stay on the device (`DeviceProgram.run`). A case is a dict of plain values:

  op "step"        a shipped training program, `program` names its file; forward, backward and optimizer update
  op "linear"      y[n, k] = x[n, d] @ W[d, k] + b[k]
  op "grad_w"      dW[d, k] = x[n, d]^T @ dy[n, k]       (the long reduction of a weight gradient)
  op "grad_x"      dx[n, d] = dy[n, k] @ W[d, k]^T       (the input gradient)
  op "softmax"     row softmax of [n, d]
  op "layer_norm"  layer_norm(x) * g + b of [n, d]
"""
import gzip
import json
import math
import os
import tempfile

import numpy as np
import torch

from anvil_lang_b200 import kir, pyapi
from anvil_lang_b200.backend import build
from anvil_lang_b200.program import DeviceProgram

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAMS = os.path.join(ROOT, "anvil_lang_b200", "programs")
GOLDEN = os.path.join(ROOT, "tests", "golden")

# program -> (batch, what the loop trains)
STEPS = {
    "c1_mlp_sgd": (64, "mlp"),
    "c3_mlp_adam": (256, "mlp"), "c3_mlp_adam.b128": (128, "mlp"), "c3_mlp_adam.b64": (64, "mlp"), "c3_mlp_adam.b32": (32, "mlp"),
    "c4_cnn_sgd": (128, "cnn"),
    "c5_transformer_t256.traj": (2, "gpt"),
    "c5_transformer": (64, "gpt"),
}
MAX_FLOPS = 2 * 16384 * 2048 * 2048        # of one drawn product


def listed():
    return [
        # the smallest configuration: a 60 us step that launches and latencies make up
        {"name": "mlp_sgd_step", "op": "step", "program": "c1_mlp_sgd"},
        # an MLP with Adam, whose products are small and whose optimizer state is most of the traffic
        {"name": "mlp_adam_step", "op": "step", "program": "c3_mlp_adam"},
        # convolutions as implicit products, pooling, SGD
        {"name": "cnn_sgd_step", "op": "step", "program": "c4_cnn_sgd"},
        # a small transformer (2 layers, D 128, 2 sequences of 256): many short launches, fused attention in both directions
        {"name": "small_transformer_step", "op": "step", "program": "c5_transformer_t256.traj"},
        # the benchmark's own step: 6 layers, D 512, 64 sequences of 256, Adam
        {"name": "transformer_step", "op": "step", "program": "c5_transformer"},
        # a linear layer called as a function, large and small, and with sizes that fill no tile
        {"name": "linear_large", "op": "linear", "n": 8192, "d": 1024, "k": 4096},
        {"name": "linear_small", "op": "linear", "n": 96, "d": 1024, "k": 256},
        {"name": "linear_ragged", "op": "linear", "n": 3001, "d": 1000, "k": 1503},
        # the two backward products of a linear layer at the transformer's sizes
        {"name": "grad_w", "op": "grad_w", "n": 16384, "d": 512, "k": 2048},
        {"name": "grad_x", "op": "grad_x", "n": 16384, "d": 512, "k": 2048},
        # row kernels called as functions
        {"name": "softmax_4096", "op": "softmax", "n": 4096, "d": 4096},
        {"name": "layer_norm_8192", "op": "layer_norm", "n": 8192, "d": 1024},
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm; half of them as programs round them (multiples of 8), half as they come."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return v if rng.random() < 0.5 or v < 16 else v // 8 * 8


def draw(rng):
    op = rng.choice(["linear"] * 3 + ["grad_w"] * 2 + ["grad_x"] * 2 + ["softmax"] * 2 + ["layer_norm"] * 2 + ["step"])
    if op == "step":
        return {"op": op, "program": rng.choice(["c3_mlp_adam.b128", "c3_mlp_adam.b64", "c3_mlp_adam.b32"])}
    if op in ("softmax", "layer_norm"):
        while True:
            n, d = _size(rng, 16, 16384), _size(rng, 16, 8192)
            if n * d <= 1 << 25:
                return {"op": op, "n": n, "d": d}
    while True:
        n, d, k = _size(rng, 32, 16384), _size(rng, 32, 4096), _size(rng, 16, 4096)
        if 2 * n * d * k <= MAX_FLOPS:
            return {"op": op, "n": n, "d": d, "k": k}


# ---------------------------------------------------------------------------------------------- programs

def _lowered(file, sizes):
    """A shipped lowered function at other sizes: the front end lowers [n, d] arguments of any size to the same kernels, so
    its extents and strides (and the 1 / d of a mean) are the only numbers that change."""
    with gzip.open(os.path.join(pyapi.LOWERED_DIR, file + ".kir.json.gz")) as f:
        meta = json.loads(f.read().decode())
    inv = {float(np.float32(1.0 / a)): float(np.float32(1.0 / b)) for a, b in sizes.items()}

    def sub(v):
        if isinstance(v, dict):
            return {key: sub(x) for key, x in v.items()}
        if isinstance(v, list):
            return [sub(x) for x in v]
        if isinstance(v, bool) or not isinstance(v, (int, float)):
            return v
        return sizes.get(v, v) if isinstance(v, int) else inv.get(v, v)

    text = meta["kir"]
    if any(a != b for a, b in sizes.items()):
        text = json.dumps(sub(json.loads(text)))
    prog = kir.loads(text)
    ids = {b.id: b for b in prog.buffers}
    return prog, [ids[i] for i in meta["inputs"]], [ids[i] for i in meta["outputs"]]


def _product(M, N, K, ta, tb):
    """C[m, n] = sum_k A * B; ta / tb: the operand is stored transposed."""
    A = kir.Buffer(1, "A", (K, M) if ta else (M, K), kir.F32, "input")
    B = kir.Buffer(2, "B", (N, K) if tb else (K, N), kir.F32, "input")
    C = kir.Buffer(3, "C", (M, N), kir.F32, "output")
    m, n, k = kir.Var(4, "m", M), kir.Var(5, "n", N), kir.Var(6, "k", K)

    def load(b, terms):
        return kir.E("load", kir.F32, buf=b, off=kir.Affine(0, terms))

    body = kir.E("bin", kir.F32, op="mul", a=[load(A, [(k, M), (m, 1)] if ta else [(m, K), (k, 1)]),
                                              load(B, [(n, K), (k, 1)] if tb else [(k, N), (n, 1)])])
    store = kir.Store(C, kir.Affine(0, [(m, N), (n, 1)]), kir.E("acc", kir.F32), False)
    kernel = kir.Kernel(7, "k7", "product", [m, n], [store], kir.Reduction([k], "sum", body))
    return kir.Program(kir.Block([kir.KernelStmt(kernel)]), [A, B, C], "product"), [A, B], [C]


def program(case):
    """(program, inputs, outputs) of a case; a training program's are found by name."""
    op = case["op"]
    if op == "step":
        for folder in (PROGRAMS, GOLDEN):
            path = os.path.join(folder, case["program"] + ".kir.json.gz")
            if os.path.exists(path):
                return kir.load(path), None, None
        raise FileNotFoundError(case["program"])
    n, d = case["n"], case["d"]
    if op == "linear":
        return _lowered("2004dbe945c335255d0b" if (n, d, case["k"]) == (8192, 1024, 4096) else "e4c699f26e56ac8eff53",
                        {8192: n, 1024: d, 4096: case["k"]} if (n, d, case["k"]) == (8192, 1024, 4096) else {96: n, 1024: d, 256: case["k"]})
    if op == "grad_w":
        return _product(d, case["k"], n, True, False)
    if op == "grad_x":
        return _product(n, d, case["k"], False, True)
    if op == "softmax":
        return _lowered("bfa409dc2ad04e39a996", {4096: 4096}) if (n, d) == (4096, 4096) else _lowered("dfeea9c2428fff98b48e", {64: n, 4096: d})
    if op == "layer_norm":
        return _lowered("6334341ef41e6fcc2f5c", {8192: n, 1024: d}) if (n, d) == (8192, 1024) else _lowered("b4ac1dc5899c161ef6e1", {128: n, 1024: d})
    raise ValueError(op)


# ---------------------------------------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _args(case, seed):
    """The arguments of a function call: activations of unit variance, weights of variance 1 / fan-in, gradients as a mean
    loss over n rows gives them (about 1 / n, rows of differing weight)."""
    g = _generator(seed)
    op, n, d, k = case["op"], case["n"], case["d"], case.get("k", 1)
    if op == "linear":
        return [_normal(g, n, d), _normal(g, d, k) / math.sqrt(d), _normal(g, k)]
    if op == "grad_w":
        return [_normal(g, n, d), _normal(g, n, k) * (_uniform(g, n, 1) / n)]
    if op == "grad_x":
        return [_normal(g, n, k) * (_uniform(g, n, 1) / n), _normal(g, d, k) / math.sqrt(d)]
    if op == "softmax":
        return [3.0 * _normal(g, n, d)]
    return [_normal(g, n, d) * 2.0 + 0.5, 1.0 + 0.1 * _normal(g, d), 0.1 * _normal(g, d)]


# (name, shape) of a training program's parameters, in the program's own order
def _parameters(prog):
    return [b for b in prog.roots() if b.kind == "param"]


def _initial(shapes, seed):
    """Parameters as the layers of the programs start: uniform +-1/sqrt(fan-in) for matrices and biases, ones and zeros for
    a layer norm's gain and bias, a small normal for the embeddings."""
    g = _generator(seed)
    out = {}
    for name, shape in shapes:
        last = name.rsplit(".", 1)[-1]
        if last == "g":
            out[name] = torch.ones(shape, device="cuda")
        elif ".ln" in name and last == "b":
            out[name] = torch.zeros(shape, device="cuda")
        elif last in ("E", "P"):
            out[name] = 0.02 * _normal(g, *shape)
        else:
            fan = math.prod(shape[1:]) if len(shape) == 4 else shape[0] if len(shape) == 2 else 512
            out[name] = (2.0 * _uniform(g, *shape) - 1.0) / math.sqrt(fan)
    return out


def _batch(case, seed):
    g = _generator(seed + (1 << 20))
    B, kind = STEPS[case["program"]]
    if kind == "gpt":
        return {"x": torch.randint(0, 256, (B, 257), generator=g, device="cuda", dtype=torch.int32)}
    x = _uniform(g, B, 784)
    return {"x": x.reshape(B, 1, 28, 28) if kind == "cnn" else x, "y": torch.randint(0, 10, (B,), generator=g, device="cuda", dtype=torch.int32)}


class _Arena:
    """A tensor of a compiled program as something torch can wrap without a copy; keeps the program alive."""

    def __init__(self, dp, b):
        self.dp = dp
        self.__cuda_array_interface__ = {"shape": tuple(b.shape), "typestr": "<i4" if b.dtype == kir.I32 else "<f4",
                                         "data": (dp.ptr(b), False), "version": 2, "strides": None}


def _view(dp, b):
    return torch.as_tensor(_Arena(dp, b), device="cuda")


def _writable_build():
    """Programs are compiled on first use; where the tree cannot be written, into a folder of this process."""
    if os.access(build.BUILD_DIR, os.W_OK):
        return
    folder = tempfile.mkdtemp(prefix="anvil_build_")
    for f in os.listdir(build.BUILD_DIR) if os.path.isdir(build.BUILD_DIR) else []:
        os.symlink(os.path.join(build.BUILD_DIR, f), os.path.join(folder, f))
    build.BUILD_DIR = folder


_stream = None


def _on_one_stream(dp):
    """All programs of this process run on one stream, as a host program that interleaves them would: each pass follows the
    one before it."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    dp.rtlib.anvil_rt_use_stream(dp.rt, _stream.cuda_stream)


def prepare(case, seed):
    _writable_build()
    prog, ins, outs = program(case)
    state = {"op": case["op"]}
    if case["op"] == "step":
        dp = DeviceProgram(prog, seed=0)
        _on_one_stream(dp)
        dp.prologue()
        dp.sync()
        params = _parameters(prog)
        start = _initial([(b.name, tuple(b.shape)) for b in params], seed)
        for b in params:
            _view(dp, b).copy_(start[b.name])
        feeds = {b.name: b for b in dp.gen.feed_bufs}
        for name, value in _batch(case, seed).items():
            _view(dp, feeds[name]).copy_(value.reshape(feeds[name].shape))
        by_name = {b.name: b for b in prog.roots() if b.kind == "state"}
        groups = {"param": params, "m": [by_name[b.name + ".m"] for b in params if b.name + ".m" in by_name],
                  "v": [by_name[b.name + ".v"] for b in params if b.name + ".m" in by_name]}
        state["groups"] = {g: [_view(dp, b) for b in bs] for g, bs in groups.items() if bs}
        state["loss"] = _view(dp, next(b for b in prog.roots() if b.name == "loss" and b.kind == ("var" if any(
            r.name == "loss" and r.kind == "var" for r in prog.roots()) else "temp")))
        state["names"] = [b.name for b in params]
        state["whole"] = len(params) <= 16
    else:
        dp = DeviceProgram(prog, seed=0, graphs=False)
        _on_one_stream(dp)
        for b, value in zip(ins, _args(case, seed)):
            _view(dp, b).copy_(value)
        state["out"] = [_view(dp, b) for b in outs]
    state["dp"] = dp
    torch.cuda.synchronize()
    return state


def run(state):
    dp = state["dp"]
    if state["op"] != "step":
        code, _ = dp.run()
        if code:
            raise RuntimeError(dp.error)
        return state["out"]
    dp.step_fed()
    out = {"loss": state["loss"]}
    if state["whole"]:
        for g, views in state["groups"].items():
            out[g] = dict(zip(state["names"], views))
    else:                      # a program with hundreds of tensors: each group as one flat tensor, in the program's order
        with torch.cuda.stream(_stream):
            for g, views in state["groups"].items():
                out[g] = torch.cat([v.reshape(-1) for v in views])
    return out


# ---------------------------------------------------------------------------------------------- work, tolerance

def _gpt(case):
    """(batch, layers, width) of a transformer program."""
    return (2, 2, 128) if case["program"] == "c5_transformer_t256.traj" else (STEPS[case["program"]][0], 6, 512)


def work(case):
    op = case["op"]
    if op == "step":
        B, kind = STEPS[case["program"]]
        if kind == "gpt":
            B, L, D = _gpt(case)
            tokens, weights = B * 256, L * 12 * D * D + 256 * D
            flops = 3 * 2 * tokens * weights + 3 * L * 2 * 2 * tokens * 256 * D
            # parameters and both moments read and written; per layer the activations that backward needs, written and read
            return {"bytes": 24 * (weights + 512 * D) + 2 * 4 * tokens * (L * 10 * D + 2 * D + 256), "flops": flops}
        if kind == "cnn":
            products = B * (26 * 26 * 9 * 32 + 11 * 11 * 288 * 64 + 1600 * 10)
            return {"bytes": 8 * (320 + 18496 + 16010) + 4 * B * (784 + 2 * 2 * (26 * 26 * 32 + 11 * 11 * 64)), "flops": 6 * products}
        weights = 784 * 128 + 1280 if case["program"] == "c1_mlp_sgd" else 784 * 1024 + 1024 * 1024 + 10240
        return {"bytes": (8 if case["program"] == "c1_mlp_sgd" else 24) * weights + 4 * B * 785, "flops": 6 * B * weights}
    n, d, k = case["n"], case["d"], case.get("k", 0)
    if op == "softmax":
        return {"bytes": 8 * n * d, "flops": 5 * n * d}
    if op == "layer_norm":
        return {"bytes": 8 * n * d + 8 * d, "flops": 8 * n * d}
    return {"bytes": 4 * (n * d + d * k + n * k + (k if op == "linear" else 0)), "flops": 2 * n * d * k}


def tolerance(case):
    """About four times the difference from 64 bits that the path shows. A product's error grows with the length of an
    accumulation chain (at most 4096: longer reductions are split): 1.9e-6 at 1024, 5.1e-6 at 2048, 9.9e-6 at 4096."""
    op = case["op"]
    if op == "step":
        # gradients of a whole step in f32 (a transformer's second moments are 2.7e-5 off); a ReLU or a pooling window at
        # its kink takes the other side on a last-bit change, and Adam divides a near-zero gradient by its own size
        return {"rel": 1e-3, "max": 0.2} if STEPS[case["program"]][1] != "gpt" else {"rel": 2e-4, "max": 0.2}
    if op in ("softmax", "layer_norm"):
        return {"rel": 1e-6, "max": 1e-5}
    rel = max(1e-5, 1e-8 * min(4096, {"linear": case["d"], "grad_w": case["n"], "grad_x": case["k"]}[op]))
    return {"rel": rel, "max": 20 * rel}


# ---------------------------------------------------------------------------------------------- 64 bits

def _shapes(case):
    _, kind = STEPS[case["program"]]
    if kind == "mlp":
        dims = [784, 128, 10] if case["program"] == "c1_mlp_sgd" else [784, 1024, 1024, 10]
        out = []
        for i, (a, b) in enumerate(zip(dims, dims[1:])):
            out += [("net.l%d.W" % (i + 1), (a, b)), ("net.l%d.b" % (i + 1), (b,))]
        return out
    if kind == "cnn":
        return [("net.c1.W", (32, 1, 3, 3)), ("net.c1.b", (32,)), ("net.c2.W", (64, 32, 3, 3)), ("net.c2.b", (64,)),
                ("net.fc.W", (1600, 10)), ("net.fc.b", (10,))]
    _, L, D = _gpt(case)
    out = [("net.E", (256, D)), ("net.P", (256, D))]
    for i in range(L):
        p = "net.layers.%d." % i
        out += [(p + "ln1.g", (D,)), (p + "ln1.b", (D,)), (p + "ln2.g", (D,)), (p + "ln2.b", (D,)), (p + "Wq", (D, D)), (p + "Wk", (D, D)),
                (p + "Wv", (D, D)), (p + "Wo", (D, D)), (p + "up.W", (D, 4 * D)), (p + "up.b", (4 * D,)), (p + "down.W", (4 * D, D)), (p + "down.b", (D,))]
    return out + [("net.lnf.g", (D,)), ("net.lnf.b", (D,)), ("net.out.W", (D, 256)), ("net.out.b", (256,))]


def _loss(case, p, batch):
    F = torch.nn.functional
    kind = STEPS[case["program"]][1]
    if kind == "mlp":
        h, last = batch["x"].double(), len(p) // 2
        for i in range(1, last + 1):
            h = h @ p["net.l%d.W" % i] + p["net.l%d.b" % i]
            h = torch.relu(h) if i < last else h
        return F.cross_entropy(h, batch["y"].long())
    if kind == "cnn":
        h = F.max_pool2d(torch.relu(F.conv2d(batch["x"].double(), p["net.c1.W"], p["net.c1.b"])), 2)
        h = F.max_pool2d(torch.relu(F.conv2d(h, p["net.c2.W"], p["net.c2.b"])), 2)
        return F.cross_entropy(h.flatten(1) @ p["net.fc.W"] + p["net.fc.b"], batch["y"].long())
    B, L, D = _gpt(case)
    H, T = D // 64, 256
    x = batch["x"].long()
    h = p["net.E"][x[:, :T]] + p["net.P"]
    mask = torch.triu(torch.ones(T, T, dtype=torch.bool, device=h.device), 1)

    def heads(t):
        return t.reshape(B, T, H, 64).transpose(1, 2)

    for i in range(L):
        q = "net.layers.%d." % i
        a = F.layer_norm(h, (D,), p[q + "ln1.g"], p[q + "ln1.b"], 1e-5)
        s = heads(a @ p[q + "Wq"]) @ heads(a @ p[q + "Wk"]).transpose(2, 3) / 8.0
        o = torch.softmax(s.masked_fill(mask, -math.inf), -1) @ heads(a @ p[q + "Wv"])
        h = h + o.transpose(1, 2).reshape(B, T, D) @ p[q + "Wo"]
        a = F.layer_norm(h, (D,), p[q + "ln2.g"], p[q + "ln2.b"], 1e-5)
        h = h + F.gelu(a @ p[q + "up.W"] + p[q + "up.b"], approximate="tanh") @ p[q + "down.W"] + p[q + "down.b"]
    logits = F.layer_norm(h, (D,), p["net.lnf.g"], p["net.lnf.b"], 1e-5) @ p["net.out.W"] + p["net.out.b"]
    return F.cross_entropy(logits.reshape(B * T, 256), x[:, 1:].reshape(-1))


def exact(case, seed):
    op = case["op"]
    if op != "step":
        a = [v.double() for v in _args(case, seed)]
        if op == "linear":
            return [a[0] @ a[1] + a[2]]
        if op == "grad_w":
            return [a[0].T @ a[1]]
        if op == "grad_x":
            return [a[0] @ a[1].T]
        if op == "softmax":
            return [torch.softmax(a[0], 1)]
        return [torch.nn.functional.layer_norm(a[0], (case["d"],), a[1], a[2], 1e-5)]
    shapes = _shapes(case)
    p = {name: v.double().requires_grad_() for name, v in _initial(shapes, seed).items()}
    loss = _loss(case, p, _batch(case, seed))
    grads = dict(zip(p, torch.autograd.grad(loss, list(p.values()))))
    out = {"loss": loss.detach(), "param": {}}
    if "sgd" in case["program"]:
        lr = 0.1 if case["program"] == "c1_mlp_sgd" else 0.05
        out["param"] = {name: (v - lr * grads[name]).detach() for name, v in p.items()}
        return out
    # the first Adam step: m = 0.1 g, v = 0.001 g^2, both divided by their bias corrections
    lr = 1e-3 if case["program"].startswith("c3") else 3e-4
    out["m"] = {name: 0.1 * g for name, g in grads.items()}
    out["v"] = {name: 0.001 * g * g for name, g in grads.items()}
    out["param"] = {name: (v - lr * grads[name] / (grads[name].abs() + 1e-8)).detach() for name, v in p.items()}
    if len(p) > 16:
        for g in ("param", "m", "v"):
            out[g] = torch.cat([v.reshape(-1) for v in out[g].values()])
    return out
