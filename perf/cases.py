"""The work this framework is used for, as cases that can be timed and compared.

A case is one pass of what a program built on the engine does over and over: a forward tape of one
of the three inference graphs, one layer on its own, one training step's share of a layer, a matrix
product, the pointwise part of a gated unit, a classifier's head. Inputs are drawn on the GPU from a
seed; everything a program keeps between passes (buffers, weights declared constant, a recorded
tape) is made in prepare(), and run() is the calls of one pass.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from gorgonia_b200 import Engine, tapes

ARENA_BYTES = 40 << 30
_engine = None


def engine():
    """One engine for the whole program, as gorgonia's tape machine has."""
    global _engine
    if _engine is None:
        _engine = _Tracked(arena_bytes=ARENA_BYTES)
        _engine.made = []
    return _engine


class _Tracked(Engine):
    """Remembers what it handed out, so that a state's buffers go back together."""

    def empty(self, shape, dtype=np.float32):
        t = super().empty(shape, dtype)
        self.made.append(t)
        return t


class _Buffers:
    """The device buffers (and the tape) of one state; they go back to the arena with it."""

    def __init__(self, e):
        self.e, self.tensors, self.tape = e, [], None

    def __enter__(self):
        self.e.made = self.tensors
        return self

    def __exit__(self, *exc):
        self.e.made = []

    def __del__(self):
        try:
            self.e.Signal()
            if self.tape is not None:
                self.tape.close()
            for t in self.tensors:
                t.free()
        except Exception:
            pass


class _Memory:
    def __init__(self, t, owner):
        kind = {"float32": "<f4", "float64": "<f8", "uint16": "<i2", "int64": "<i8", "int32": "<i4"}[t.dtype.name]
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": t.shape, "typestr": kind, "data": (t.ptr, False), "version": 3}


def view(t, owner):
    """A torch tensor over an engine tensor's memory."""
    v = torch.as_tensor(_Memory(t, owner), device="cuda")
    return v.view(torch.bfloat16) if getattr(t, "is_bf16", False) else v


def fill(t, values, owner):
    view(t, owner).copy_(values)


NUMPY = {torch.float32: np.float32, torch.float64: np.float64, torch.int64: np.int64}


def upload(e, values, owner):
    """An engine tensor with the values of a torch tensor."""
    if values.dtype == torch.bfloat16:
        t = e.empty(tuple(values.shape), np.uint16)
        t.is_bf16 = True
    else:
        t = e.empty(tuple(values.shape), NUMPY[values.dtype])
    fill(t, values, owner)
    return t


def _dt(case):
    return {"f32": torch.float32, "f64": torch.float64, "bf16": torch.bfloat16}[case.get("dtype", "f32")]


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------

def listed():
    return [
        # one batch through the small fully connected net: the call where latency and launches count
        {"name": "mlp_forward_256", "kind": "mlp", "batch": 256},
        # MNIST-sized convolutional net at its throughput batch
        {"name": "lenet_forward_8192", "kind": "lenet", "batch": 8192},
        # object detection, the largest of the three graphs at its throughput batch
        {"name": "yolo_forward_64", "kind": "yolo", "batch": 64},
        # one convolution of a detector on its own, bias and leaky rectifier folded in
        {"name": "conv_128_256", "kind": "conv", "batch": 16, "c": 128, "h": 26, "w": 26, "k": 256, "kernel": 3,
         "stride": 1, "pad": 1},
        # backward pass of a convolution, rectifier and max-pool at the training batch of the MNIST example
        {"name": "conv_train_100", "kind": "conv_train", "batch": 100, "c": 32, "h": 14, "w": 14, "k": 64},
        # dense layer, forward and both gradients, with sizes that no tile divides
        {"name": "dense_train_1000", "kind": "dense_train", "dtype": "f32", "batch": 1000, "n_in": 1152, "n_out": 625},
        # the same in gorgonia's default type
        {"name": "dense_train_f64_256", "kind": "dense_train", "dtype": "f64", "batch": 256, "n_in": 784, "n_out": 300},
        # square products, the sizes of the linear algebra sweep
        {"name": "matmul_f32_4096", "kind": "matmul", "dtype": "f32", "slices": 1, "m": 4096, "n": 4096, "k": 4096,
         "ta": False, "tb": False},
        {"name": "matmul_bf16_4096", "kind": "matmul", "dtype": "bf16", "slices": 1, "m": 4096, "n": 4096, "k": 4096,
         "ta": False, "tb": False},
        # the elementwise part of a gated unit on long vectors
        {"name": "gated_2p24", "kind": "gated", "dtype": "f32", "n": 1 << 24},
        # batch normalisation with scale, shift and dropout, forward and backward
        {"name": "norm_train_128", "kind": "norm_train", "batch": 128, "c": 64, "h": 28, "w": 28},
        # a classifier's last step on one small batch: bias, softmax, prediction, gradient
        {"name": "head_256", "kind": "head", "batch": 256, "classes": 10},
    ]


def _log(rng, lo, hi, step=1):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step
    return max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(["mlp", "lenet", "yolo", "conv", "conv", "conv_train", "dense_train", "dense_train", "matmul",
                       "matmul", "matmul", "gated", "gated", "norm_train", "head"])
    if kind in ("mlp", "lenet", "yolo"):
        lo, hi = {"mlp": (16, 4096), "lenet": (32, 8192), "yolo": (2, 48)}[kind]
        return {"kind": kind, "batch": _log(rng, lo, hi)}
    if kind == "conv":
        while True:
            kernel = rng.choice([1, 3, 3, 3, 5])
            hw = _log(rng, 7, 112)
            c = {"kind": kind, "batch": _log(rng, 1, 256), "c": rng.choice([3, 16, 24, 32, 64, 96, 128, 200, 256, 512]),
                 "h": hw, "w": hw + rng.choice([0, 0, 1, 5]), "k": rng.choice([16, 32, 50, 64, 125, 128, 256, 512]),
                 "kernel": kernel, "stride": rng.choice([1, 1, 1, 2]), "pad": kernel // 2}
            if work(c)["flops"] < 2e11 and work(c)["bytes"] < 2e9:
                return c
    if kind == "conv_train":
        hw = 2 * rng.randrange(3, 15)
        c = rng.choice([16, 32, 64, 128])
        return {"kind": kind, "batch": _log(rng, 16, min(512, (1 << 28) // (hw * hw * c * 9))), "c": c, "h": hw, "w": hw,
                "k": rng.choice([32, 64, 128])}
    if kind == "dense_train":
        dtype = rng.choice(["f32", "f32", "f64"])
        top = 4096 if dtype == "f32" else 1024
        return {"kind": kind, "dtype": dtype, "batch": _log(rng, 16, top), "n_in": _log(rng, 32, top),
                "n_out": _log(rng, 10, top)}
    if kind == "matmul":
        dtype = rng.choice(["f32", "f32", "bf16"])
        slices = rng.choice([1, 1, 1, _log(rng, 2, 64)])
        top, step = (5120 if slices == 1 else 1024), (8 if dtype == "bf16" else 1)
        ta, tb = rng.choice([(False, False), (False, False), (True, False), (False, True)])
        return {"kind": kind, "dtype": dtype, "slices": slices, "m": _log(rng, 96, top, step), "n": _log(rng, 96, top, step),
                "k": _log(rng, 96, top, step), "ta": ta, "tb": tb}
    if kind == "gated":
        return {"kind": kind, "dtype": rng.choice(["f32", "f32", "f64"]), "n": _log(rng, 1 << 10, 1 << 25)}
    if kind == "norm_train":
        hw = _log(rng, 4, 56)
        c = rng.choice([16, 32, 64, 100, 128, 256])
        return {"kind": kind, "batch": _log(rng, 8, max(8, min(2048, (1 << 24) // (hw * hw * c)))), "c": c, "h": hw, "w": hw}
    return {"kind": kind, "batch": _log(rng, 16, 65536), "classes": rng.choice([2, 10, 10, 37, 100, 1000])}


# ------------------------------------------------------------------------------------------
# inputs, shared by prepare() and exact()
# ------------------------------------------------------------------------------------------

MLP_DIMS = (784, 300, 100, 10)
LENET_CH = (1, 32, 64, 128)
YOLO_CH = (3, 16, 32, 64, 128, 256, 512, 1024, 1024, 125)
DROP, EPS, MOMENTUM = 0.3, 1e-5, 0.9


def inputs(case, seed):
    """The values of one case as torch tensors on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    kind, dt = case["kind"], _dt(case)

    def normal(*shape, scale=1.0):
        t = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64 if dt == torch.float64 else torch.float32)
        return t.mul_(scale) if scale != 1.0 else t

    def uniform(*shape):
        return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64 if dt == torch.float64 else torch.float32)

    def he(*shape):   # he-normal filters or Glorot-like dense weights, by fan-in
        fan = shape[1] * shape[2] * shape[3] if len(shape) == 4 else shape[0]
        return normal(*shape, scale=math.sqrt(2.0 / fan))

    b = case.get("batch")
    if kind == "mlp":
        return {"x": uniform(b, 784), "w": [he(MLP_DIMS[i], MLP_DIMS[i + 1]) for i in range(3)],
                "b": [normal(MLP_DIMS[i + 1], scale=0.1) for i in range(3)]}
    if kind == "lenet":
        return {"x": uniform(b, 1, 28, 28), "wc": [he(LENET_CH[i + 1], LENET_CH[i], 3, 3) for i in range(3)],
                "wd": [he(1152, 625), he(625, 10)]}
    if kind == "yolo":
        ks = [3] * 8 + [1]
        return {"x": uniform(b, 3, 416, 416), "w": [he(YOLO_CH[i + 1], YOLO_CH[i], ks[i], ks[i]) for i in range(9)],
                "b": [normal(YOLO_CH[i + 1], scale=0.1) for i in range(9)]}
    if kind == "conv":
        return {"x": F.leaky_relu(normal(b, case["c"], case["h"], case["w"]), 0.1),
                "w": he(case["k"], case["c"], case["kernel"], case["kernel"]), "b": normal(case["k"], scale=0.1)}
    if kind == "conv_train":
        c, h, w, k = case["c"], case["h"], case["w"], case["k"]
        act = F.relu(normal(b, k, h, w))
        return {"x": F.relu(normal(b, c, h, w)), "w": he(k, c, 3, 3), "on": (act > 0).to(torch.float32),
                "where": F.max_pool2d(act, 2, return_indices=True)[1], "dy": normal(b, k, h // 2, w // 2, scale=0.01)}
    if kind == "dense_train":
        return {"x": F.relu(normal(b, case["n_in"])), "w": he(case["n_in"], case["n_out"]),
                "b": normal(case["n_out"], scale=0.1), "dy": normal(b, case["n_out"], scale=0.01)}
    if kind == "matmul":
        s, m, n, k = case["slices"], case["m"], case["n"], case["k"]
        lead = (s,) if s > 1 else ()
        a = normal(*lead, *((k, m) if case["ta"] else (m, k)))
        return {"a": a.to(dt), "b": normal(*lead, *((n, k) if case["tb"] else (k, n)), scale=0.02).to(dt)}
    if kind == "gated":
        return {name: normal(case["n"]) for name in ("zi", "zf", "zg", "zo", "c")}
    if kind == "norm_train":
        shape = (b, case["c"], case["h"], case["w"])
        return {"x": normal(*shape, scale=2.0).add_(0.5), "gamma": uniform(case["c"]).add_(0.5), "beta": normal(case["c"]),
                "draws": uniform(*shape), "dy": normal(*shape, scale=0.01)}
    return {"h": normal(b, case["classes"]), "b": normal(case["classes"], scale=0.1),
            "g": normal(b, case["classes"], scale=1.0 / b)}


# ------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------

def prepare(case, seed):
    e = engine()
    v = inputs(case, seed)
    buf = _Buffers(e)
    with buf:
        st = _PREPARE[case["kind"]](e, case, v, buf)
    st["e"], st["buf"], st["kind"] = e, buf, case["kind"]
    st["views"] = {name: view(t, buf) for name, t in st["out"].items()}
    torch.cuda.synchronize()
    return st


def run(state):
    _RUN[state["kind"]](state["e"], state)
    return state["views"]


def _model(e, m, buf, out):
    torch.cuda.synchronize()
    m.record()
    buf.tape = m
    return {"m": m, "out": out}


def _prepare_mlp(e, case, v, buf):
    m = tapes.MLP(e, case["batch"])
    for i in range(3):
        fill(m.w[i], v["w"][i], buf)
        fill(m.b[i], v["b"][i], buf)
    fill(m.x, v["x"], buf)
    return _model(e, m, buf, {"logits": m.chain.layers[-1]["c"], "probabilities": m.out})


def _prepare_lenet(e, case, v, buf):
    m = tapes.LeNet(e, case["batch"])
    for i in range(3):
        fill(m.wc[i], v["wc"][i], buf)
    for i in range(2):
        fill(m.wd[i], v["wd"][i], buf)
    fill(m.x, v["x"], buf)
    return _model(e, m, buf, {"logits": m.dense.layers[-1]["c"], "probabilities": m.out})


def _prepare_yolo(e, case, v, buf):
    m = tapes.TinyYolo(e, case["batch"])
    for i in range(9):
        fill(m.w[i], v["w"][i], buf)
        fill(m.b[i], v["b"][i], buf)
    fill(m.x, v["x"], buf)
    return _model(e, m, buf, {"grid": m.out})


def _run_model(e, s):
    s["m"].replay()


def _conv_out(case):
    k, st, p = case["kernel"], case["stride"], case["pad"]
    return (case["h"] + 2 * p - k) // st + 1, (case["w"] + 2 * p - k) // st + 1


def _prepare_conv(e, case, v, buf):
    st = {n: upload(e, v[n], buf) for n in ("x", "w", "b")}
    e.constant(st["w"])
    st["out"] = {"y": e.empty((case["batch"], case["k"]) + _conv_out(case))}
    st["how"] = dict(pad=(case["pad"],) * 2, stride=(case["stride"],) * 2)
    return st


def _run_conv(e, s):
    e.Conv2d(s["x"], s["w"], s["out"]["y"], bias=s["b"], act="leaky", alpha=0.1, **s["how"])


def _prepare_conv_train(e, case, v, buf):
    b, c, h, w, k = (case[n] for n in ("batch", "c", "h", "w", "k"))
    st = {n: upload(e, v[n], buf) for n in ("x", "w", "on", "where", "dy")}
    st["w2"] = st["w"].reshape(k, c * 9)
    st["da"], st["rows"] = e.empty((b, k, h, w)), e.empty((b, h, w, k))
    st["col"], st["dcol"] = e.empty((b, h, w, c * 9)), e.empty((b, h, w, c * 9))
    st["rows2"] = st["rows"].reshape(b * h * w, k)
    st["col2"], st["dcol2"] = st["col"].reshape(b * h * w, c * 9), st["dcol"].reshape(b * h * w, c * 9)
    st["out"] = {"dw": e.empty((k, c * 9)), "dx": e.empty((b, c, h, w))}
    return st


def _run_conv_train(e, s):
    e.MaxPool2DDiff(s["dy"], s["where"], s["da"], (2, 2), (0, 0), (2, 2))
    e.Mul(s["da"], s["on"], unsafe=True)
    e.Transpose(s["da"], s["rows"], (0, 2, 3, 1))
    e.Im2Col(s["x"], s["col"], (3, 3), pad=(1, 1))
    e.MatMul(s["rows2"], s["col2"], s["out"]["dw"], transA=True)
    e.MatMul(s["rows2"], s["w2"], s["dcol2"])
    e.Col2Im(s["dcol"], s["out"]["dx"], (3, 3), pad=(1, 1))


def _prepare_dense_train(e, case, v, buf):
    st = {n: upload(e, v[n], buf) for n in ("x", "w", "b", "dy")}
    b, i, o, dt = case["batch"], case["n_in"], case["n_out"], st["x"].dtype
    st["out"] = {"y": e.empty((b, o), dt), "dx": e.empty((b, i), dt), "dw": e.empty((i, o), dt), "db": e.empty((1, o), dt)}
    return st


def _run_dense_train(e, s):
    o = s["out"]
    e.MatMul(s["x"], s["w"], o["y"], bias=s["b"])
    e.MatMul(s["dy"], s["w"], o["dx"], transB=True)
    e.MatMul(s["x"], s["dy"], o["dw"], transA=True)
    e.Reduce("sum", s["dy"], o["db"], 0)


def _prepare_matmul(e, case, v, buf):
    lead = (case["slices"],) if case["slices"] > 1 else ()
    return {"a": upload(e, v["a"], buf), "b": upload(e, v["b"], buf), "ta": case["ta"], "tb": case["tb"],
            "out": {"c": e.empty(lead + (case["m"], case["n"]))}}


def _run_matmul(e, s):
    e.MatMul(s["a"], s["b"], s["out"]["c"], transA=s["ta"], transB=s["tb"])


def _prepare_gated(e, case, v, buf):
    st = {n: upload(e, t, buf) for n, t in v.items()}
    st["out"] = {"c": e.empty((case["n"],), st["c"].dtype), "h": e.empty((case["n"],), st["c"].dtype)}
    return st


def _run_gated(e, s):
    o, z = s["out"], s["c"]
    e.made = []
    i, f, g, q = (e.empty(z.shape, z.dtype) for _ in range(4))
    e.Unary("sigmoid", s["zi"], reuse=i)
    e.Unary("sigmoid", s["zf"], reuse=f)
    e.Unary("tanh", s["zg"], reuse=g)
    e.Mul(f, s["c"], reuse=o["c"])
    e.Mul(i, g, unsafe=True)
    e.Add(o["c"], i, unsafe=True)
    e.Unary("sigmoid", s["zo"], reuse=q)
    e.Unary("tanh", o["c"], reuse=o["h"])
    e.Mul(o["h"], q, unsafe=True)
    for t in (i, f, g, q):
        t.free()
    e.made = []
    e.DoWork()


def _prepare_norm_train(e, case, v, buf):
    st = {n: upload(e, t, buf) for n, t in v.items()}
    c, shape = case["c"], st["x"].shape
    st["c"], st["s"] = c, case["h"] * case["w"]
    st["xn"], st["back"] = e.empty(shape), e.empty(shape)
    mean, var = e.empty(c), e.empty(c)
    st["running"] = (mean, var)
    fill(mean, torch.zeros(c, device="cuda"), buf)
    fill(var, torch.ones(c, device="cuda"), buf)
    st["out"] = {"y": e.empty(shape), "dx": e.empty(shape), "mean": e.empty(c), "var": e.empty(c)}
    return st


def _run_norm_train(e, s):
    o, (mean, var) = s["out"], s["running"]
    e.BatchNorm(s["x"], s["xn"], mean, var, o["mean"], o["var"], momentum=MOMENTUM, epsilon=EPS)
    e.BroadcastBinary("mul", s["xn"], s["gamma"], s["s"], s["c"], unsafe=True)
    e.BroadcastBinary("add", s["xn"], s["beta"], s["s"], s["c"], unsafe=True)
    e.Dropout(s["xn"], o["y"], DROP, uniforms=s["draws"])
    e.DropoutDiff(s["dy"], o["y"], s["back"], DROP)
    e.BroadcastBinary("mul", s["back"], s["gamma"], s["s"], s["c"], unsafe=True)
    e.BatchNormDiff(s["x"], s["back"], o["dx"], var, o["mean"], o["var"], epsilon=EPS)


def _prepare_head(e, case, v, buf):
    st = {n: upload(e, t, buf) for n, t in v.items()}
    b, n = case["batch"], case["classes"]
    st["z"] = e.empty((b, n))
    st["classes"] = n
    st["out"] = {"p": e.empty((b, n)), "dz": e.empty((b, n)), "db": e.empty((n,)), "best": e.empty((b,), np.int64)}
    return st


def _run_head(e, s):
    o = s["out"]
    e.BroadcastBinary("add", s["h"], s["b"], 1, s["classes"], reuse=s["z"])
    e.SoftMax(s["z"], o["p"])
    e.Argmax(s["z"], o["best"], 1)
    e.SoftMaxDiff(o["p"], s["g"], o["dz"])
    e.Reduce("sum", o["dz"], o["db"], 0)


_PREPARE = {"mlp": _prepare_mlp, "lenet": _prepare_lenet, "yolo": _prepare_yolo, "conv": _prepare_conv,
            "conv_train": _prepare_conv_train, "dense_train": _prepare_dense_train, "matmul": _prepare_matmul,
            "gated": _prepare_gated, "norm_train": _prepare_norm_train, "head": _prepare_head}
_RUN = {"mlp": _run_model, "lenet": _run_model, "yolo": _run_model, "conv": _run_conv, "conv_train": _run_conv_train,
        "dense_train": _run_dense_train, "matmul": _run_matmul, "gated": _run_gated, "norm_train": _run_norm_train,
        "head": _run_head}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without, and how exact its results are
# ------------------------------------------------------------------------------------------

def work(case):
    kind, b = case["kind"], case.get("batch", 1)
    size = {"f32": 4, "f64": 8, "bf16": 2}[case.get("dtype", "f32")]
    if kind == "mlp":
        w = sum(MLP_DIMS[i] * MLP_DIMS[i + 1] for i in range(3))
        return {"bytes": 4 * (b * (784 + 20) + w + sum(MLP_DIMS[1:])), "flops": 2 * b * w}
    if kind == "lenet":
        conv = 28 * 28 * 32 * 9 + 14 * 14 * 64 * 288 + 7 * 7 * 128 * 576
        dense = 1152 * 625 + 625 * 10
        return {"bytes": 4 * (b * (784 + 20) + 288 + 18432 + 73728 + dense), "flops": 2 * b * (conv + dense)}
    if kind == "yolo":
        s, flops, params = 416, 0, 0
        for i in range(9):
            p = YOLO_CH[i] * YOLO_CH[i + 1] * (1 if i == 8 else 9)
            flops += 2 * s * s * p
            params += p + YOLO_CH[i + 1]
            s //= 2 if i < 5 else 1
        return {"bytes": 4 * (b * (3 * 416 * 416 + 125 * 13 * 13) + params), "flops": b * flops}
    if kind == "conv":
        ho, wo = _conv_out(case)
        taps = case["c"] * case["kernel"] ** 2
        return {"bytes": 4 * (b * case["c"] * case["h"] * case["w"] + case["k"] * (taps + 1) + b * case["k"] * ho * wo),
                "flops": 2 * b * ho * wo * case["k"] * taps}
    if kind == "conv_train":
        c, k, hw = case["c"], case["k"], case["h"] * case["w"]
        return {"bytes": 4 * (b * hw * (2 * c + k) + 2 * k * c * 9) + b * k * (hw // 4) * 12, "flops": 4 * b * hw * k * c * 9}
    if kind == "dense_train":
        i, o = case["n_in"], case["n_out"]
        return {"bytes": size * (2 * b * i + 2 * b * o + 2 * i * o + 2 * o), "flops": 6 * b * i * o}
    if kind == "matmul":
        s, m, n, k = case["slices"], case["m"], case["n"], case["k"]
        return {"bytes": s * (size * (m * k + k * n) + 4 * m * n), "flops": 2 * s * m * n * k}
    if kind == "gated":
        return {"bytes": 7 * size * case["n"], "flops": 9 * case["n"]}
    if kind == "norm_train":
        n = b * case["c"] * case["h"] * case["w"]
        return {"bytes": 4 * (5 * n + 6 * case["c"]), "flops": 20 * n}
    n = b * case["classes"]
    return {"bytes": 4 * (4 * n + 2 * case["classes"]) + 8 * b, "flops": 12 * n}


def tolerance(case):
    kind, dtype = case["kind"], case.get("dtype", "f32")
    if dtype == "f64":
        return {"rel": 1e-13, "max": 1e-11}
    if kind in ("gated", "norm_train", "head"):
        return {"rel": 2e-6, "max": 1e-4, "differ": 1e-4}
    # sums of float32 products; through a whole net, or in one long chain of bfloat16 products (exact
    # themselves, summed in float32 by the tensor core), about 4e-6 is what shows
    return {"rel": 2e-5 if kind in ("mlp", "lenet", "yolo") or dtype == "bf16" else 1e-5, "max": 2e-4}


def exact(case, seed):
    """What run() returns, in 64 bits."""
    v = inputs(case, seed)
    up = lambda t: t.double() if t.is_floating_point() else t  # noqa: E731
    v = {n: [up(x) for x in t] if isinstance(t, list) else up(t) for n, t in v.items()}
    with torch.no_grad():
        return _EXACT[case["kind"]](case, v)


def _exact_mlp(case, v):
    a = v["x"]
    for i in range(3):
        a = a @ v["w"][i] + v["b"][i]
        a = F.relu(a) if i < 2 else a
    return {"logits": a, "probabilities": torch.softmax(a, 1)}


def _conv64(x, w, stride=1, pad=0, most=1 << 27):
    """Convolution as unfolded products, a few samples at a time."""
    k, c, r, s = w.shape
    ho, wo = (x.shape[2] + 2 * pad - r) // stride + 1, (x.shape[3] + 2 * pad - s) // stride + 1
    step = max(1, most // (c * r * s * ho * wo))
    out = [w.reshape(k, -1) @ F.unfold(x[i:i + step], (r, s), padding=pad, stride=stride) for i in range(0, len(x), step)]
    return torch.cat(out).reshape(len(x), k, ho, wo)


def _exact_lenet(case, v):
    a = v["x"]
    for w in v["wc"]:
        a = F.max_pool2d(F.relu(_conv64(a, w, pad=1)), 2)
    a = F.relu(a.reshape(len(a), -1) @ v["wd"][0]) @ v["wd"][1]
    return {"logits": a, "probabilities": torch.softmax(a, 1)}


def _exact_yolo(case, v):
    a = v["x"]
    for i in range(9):
        a = _conv64(a, v["w"][i], pad=1 if i < 8 else 0) + v["b"][i].reshape(1, -1, 1, 1)
        a = F.leaky_relu(a, 0.1) if i < 8 else a
        if i < 5:
            a = F.max_pool2d(a, 2)
        elif i == 5:    # explicit padding north 1, west 1 of gorgonia: windows start at the pixel itself
            a = F.max_pool2d(F.pad(a, (0, 1, 0, 1), value=-math.inf), 2, stride=1)
    return {"grid": a}


def _exact_conv(case, v):
    y = _conv64(v["x"], v["w"], case["stride"], case["pad"]) + v["b"].reshape(1, -1, 1, 1)
    return {"y": F.leaky_relu(y, 0.1)}


def _exact_conv_train(case, v):
    b, c, h, w, k = (case[n] for n in ("batch", "c", "h", "w", "k"))
    da = F.max_unpool2d(v["dy"], v["where"], 2, output_size=(h, w)) * v["on"]
    da = da.reshape(b, k, h * w)
    dw, dx = torch.zeros(k, c * 9, device="cuda", dtype=torch.float64), []
    for i in range(0, b, 32):
        col = F.unfold(v["x"][i:i + 32], 3, padding=1)
        dw += torch.einsum("bkp,bqp->kq", da[i:i + 32], col)
        dx.append(F.fold(v["w"].reshape(k, -1).t() @ da[i:i + 32], (h, w), 3, padding=1))
    return {"dw": dw, "dx": torch.cat(dx)}


def _exact_dense_train(case, v):
    return {"y": v["x"] @ v["w"] + v["b"], "dx": v["dy"] @ v["w"].t(), "dw": v["x"].t() @ v["dy"],
            "db": v["dy"].sum(0, keepdim=True)}


def _exact_matmul(case, v):
    a = v["a"].transpose(-1, -2) if case["ta"] else v["a"]
    b = v["b"].transpose(-1, -2) if case["tb"] else v["b"]
    return {"c": a @ b}


def _exact_gated(case, v):
    c = torch.sigmoid(v["zf"]) * v["c"] + torch.sigmoid(v["zi"]) * torch.tanh(v["zg"])
    return {"c": c, "h": torch.sigmoid(v["zo"]) * torch.tanh(c)}


def _exact_norm_train(case, v):
    x, col = v["x"], (1, -1, 1, 1)
    n = x.numel() // case["c"]
    mean = x.mean((0, 2, 3))
    dev = x - mean.reshape(col)
    var = dev.square().sum((0, 2, 3))
    inv = (1 / torch.sqrt(var / n + EPS)).reshape(col)
    keep = (v["draws"].float() < np.float32(1 - DROP)).double()
    y = (dev * inv * v["gamma"].reshape(col) + v["beta"].reshape(col)) / (1 - DROP) * keep
    g = v["dy"] / DROP * keep * v["gamma"].reshape(col)
    k = ((dev * g).sum((0, 2, 3)) / n).reshape(col) * inv.square()
    dx = (g - g.mean((0, 2, 3)).reshape(col) - dev * k) * inv
    return {"y": y, "dx": dx, "mean": mean, "var": var}


def _exact_head(case, v):
    p = torch.softmax(v["h"] + v["b"], 1)
    dz = p * (v["g"] - (v["g"] * p).sum(1, keepdim=True))
    return {"p": p, "dz": dz, "db": dz.sum(0), "best": None}


_EXACT = {"mlp": _exact_mlp, "lenet": _exact_lenet, "yolo": _exact_yolo, "conv": _exact_conv,
          "conv_train": _exact_conv_train, "dense_train": _exact_dense_train, "matmul": _exact_matmul,
          "gated": _exact_gated, "norm_train": _exact_norm_train, "head": _exact_head}
