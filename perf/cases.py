"""The work that programs written against this framework ask of it, as cases to be timed.

Every case goes through the public namespace (`nn.Conv2D`, `nn.leaky_relu`, `nn.backward`,
`nn.optimizer`, ...), in the default precision of the contractions (split FP16, fp32 level).
Ten kinds, each with a range that `draw` samples and that the listed cases stand for:

  serve    classifier inference, host images in, host logits out: one request of a few images
  infer    the same network over a batch that is already on the GPU
  train    one training step of the classifier (softmax cross-entropy, backward, optimizer)
  mlp      one training step of a small fully connected network: launch latency only
  dense    a Dense layer, forward and backward
  matmul   a (batched) matrix product, forward
  conv     a convolution layer with bias, forward, input gradient and kernel gradient
  affine   leaky_relu(x * g + b) per channel, forward and backward: element-wise traffic
  pool     max / average pooling, forward and backward
  reduce   sum / mean / max over some axes, forward and backward
"""
import functools

import numpy as np
import torch

import litenn_b200 as nn

CLASSES = 1000


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # one request with one image: what a server answers interactively
        {"name": "serve_1", "kind": "serve", "batch": 1, "size": 128, "width": 32},
        # one micro-batch of offline inference, the benchmark's own
        {"name": "infer_1024", "kind": "infer", "batch": 1024, "size": 128, "width": 32},
        # fine-tuning on a small ragged batch with the operators of the user guide, Adam
        {"name": "train_37_stock", "kind": "train", "batch": 37, "size": 60, "width": 32, "api": "stock", "opt": "adam"},
        # a full training step of the benchmark's network with the fused trainable blocks, SGD
        {"name": "train_512_block", "kind": "train", "batch": 512, "size": 128, "width": 32, "api": "block", "opt": "sgd"},
        # a small network on feature vectors: every kernel is a few microseconds
        {"name": "mlp_64", "kind": "mlp", "batch": 64, "features": 256, "hidden": 512, "layers": 3, "out": 10, "opt": "adam"},
        # the Dense configuration of the benchmark
        {"name": "dense_8192", "kind": "dense", "rows": 8192, "in": 1024, "out": 4096},
        # extents that no tile divides
        {"name": "matmul_odd", "kind": "matmul", "batch": 1, "m": 1003, "k": 777, "n": 1501},
        # the smallest convolution configuration of the benchmark
        {"name": "conv_8x16x32", "kind": "conv", "batch": 8, "ic": 16, "oc": 32, "size": 32, "k": 3, "stride": 1},
        # a strided stage of the benchmark
        {"name": "conv_256x128x56_s2", "kind": "conv", "batch": 256, "ic": 128, "oc": 256, "size": 56, "k": 3, "stride": 2},
        # per-channel scale, shift and activation over a large activation
        {"name": "affine_128x256x56", "kind": "affine", "batch": 128, "ch": 256, "size": 56},
        # the pooling configuration of the benchmark at a quarter of its batch
        {"name": "max_pool_64x128x112", "kind": "pool", "batch": 64, "ch": 128, "size": 112, "pool": 2, "op": "max"},
        # the reduction configuration of the benchmark: columns of a 256 x 512 x 1024 tensor
        {"name": "sum_256x512x1024_axis1", "kind": "reduce", "d0": 256, "d1": 512, "d2": 1024, "axes": "1", "op": "sum"},
    ]


def _log(rng, lo, hi):
    """A whole number whose logarithm is uniform between lo and hi."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["serve", "infer", "train", "mlp", "dense", "matmul", "conv", "affine", "pool", "reduce"])
    if kind == "serve":
        return {"kind": kind, "batch": _log(rng, 1, 64), "size": rng.randint(32, 128), "width": rng.choice([16, 24, 32])}
    if kind == "infer":
        return {"kind": kind, "batch": _log(rng, 8, 1024), "size": rng.randint(32, 128), "width": rng.choice([16, 24, 32])}
    if kind == "train":
        return {"kind": kind, "batch": _log(rng, 8, 512), "size": rng.randint(32, 128), "width": rng.choice([16, 24, 32]),
                "api": rng.choice(["stock", "block"]), "opt": rng.choice(["sgd", "momentum", "rmsprop", "adam"])}
    if kind == "mlp":
        return {"kind": kind, "batch": _log(rng, 8, 1024), "features": _log(rng, 16, 1024), "hidden": _log(rng, 32, 1024),
                "layers": rng.randint(2, 5), "out": _log(rng, 2, 1000), "opt": rng.choice(["sgd", "momentum", "rmsprop", "adam"])}
    if kind == "dense":
        return {"kind": kind, "rows": _log(rng, 16, 8192), "in": _log(rng, 32, 4096), "out": _log(rng, 16, 4096)}
    if kind == "matmul":
        batch = rng.choice([1, 1, _log(rng, 2, 16)])
        top = 4096 if batch == 1 else 1024
        return {"kind": kind, "batch": batch, "m": _log(rng, 32, top), "k": _log(rng, 32, top), "n": _log(rng, 32, top)}
    if kind == "conv":
        k = rng.choice([1, 3, 3, 3, 5])
        top = {1: 256, 3: 128, 5: 48}[k]
        return {"kind": kind, "batch": _log(rng, 1, 128), "ic": _log(rng, 8, top), "oc": _log(rng, 8, 2 * top),
                "size": _log(rng, 7, 56), "k": k, "stride": rng.choice([1, 1, 2])}
    if kind == "affine":
        return {"kind": kind, "batch": _log(rng, 1, 128), "ch": _log(rng, 8, 256), "size": rng.randint(7, 56)}
    if kind == "pool":
        return {"kind": kind, "batch": _log(rng, 1, 64), "ch": _log(rng, 8, 128), "size": rng.randint(14, 112),
                "pool": rng.choice([2, 2, 3]), "op": rng.choice(["max", "avg"])}
    return {"kind": kind, "d0": _log(rng, 4, 256), "d1": _log(rng, 8, 512), "d2": _log(rng, 16, 1024),
            "axes": rng.choice(["0", "1", "2", "all"]), "op": rng.choice(["sum", "mean", "max"])}


# ---------------------------------------------------------------------------------------------
# what the cases are made of
# ---------------------------------------------------------------------------------------------
class _Result(list):
    """The outputs of a pass as torch tensors over the framework's own buffers; keeps them alive."""
    owners = ()


class _Memory:
    def __init__(self, pointer, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (pointer, False), "version": 3}


@functools.lru_cache(maxsize=4096)
def _view(pointer, shape):
    return torch.as_tensor(_Memory(pointer, shape), device="cuda:0")


def _outputs(*tensors):
    r = _Result(_view(t._ptr(0), t.shape.shape) for t in tensors)
    r.owners = tensors
    return r


def _filled(shape, init):
    """A tensor with its values on the GPU (the random initializers draw from np.random)."""
    t = nn.Tensor(shape, init=init)
    t._ptr(0)
    return t


def _normal(shape, std=1.0):
    return _filled(shape, nn.initializer.RandomNormal(0.0, std))


def _uniform(shape, lo, hi):
    return _filled(shape, nn.initializer.RandomUniform(lo, hi))


def _one_hot(rng, batch, classes):
    t = np.zeros((batch, classes), np.float32)
    t[np.arange(batch), rng.integers(0, classes, batch)] = 1.0
    return nn.Tensor_from_value(t)


def _optimizer(name, tensors):
    if name == "sgd":
        return nn.optimizer.SGD(tensors, lr=1e-3)
    if name == "momentum":
        return nn.optimizer.SGD(tensors, momentum=0.9, lr=1e-3)
    if name == "rmsprop":
        return nn.optimizer.RMSprop(tensors, lr=1e-4)
    return nn.optimizer.Adam(tensors, lr=1e-4)


def _channels(width):
    return [3, width, 2 * width, 4 * width, 8 * width]


class Classifier(nn.Module):
    """Four 3x3 convolutions with leaky_relu, max-pooling after the first three, global mean and a
    Dense layer; `block` takes the fused trainable entry instead of three operators per block."""

    def __init__(self, width, block=False):
        self.block = block
        ch = _channels(width)
        self.convs = [nn.Conv2D(ch[i], ch[i + 1], 3, kernel_initializer=nn.initializer.HeNormal(),
                                bias_initializer=nn.initializer.RandomUniform(-0.1, 0.1)) for i in range(4)]
        self.dense = nn.Dense(ch[4], CLASSES, weight_initializer=nn.initializer.HeNormal(),
                              bias_initializer=nn.initializer.RandomUniform(-0.1, 0.1))

    def forward(self, x):
        for i, c in enumerate(self.convs):
            if self.block and i < 3:
                x = nn.conv2D_block(x, c.kernel, 1, 1, "same", bias_t=c.bias, activation="leaky_relu", alpha=0.1)
            elif self.block:
                x = nn.conv2D(x, c.kernel, 1, 1, "same", bias_t=c.bias, activation="leaky_relu", alpha=0.1)
            else:
                x = nn.leaky_relu(c(x), 0.1)
                if i < 3:
                    x = nn.max_pool2D(x)
        return self.dense(nn.flatten(nn.reduce_mean(x, (2, 3))))


class Perceptron(nn.Module):
    def __init__(self, features, hidden, layers, out):
        w = [features] + [hidden] * (layers - 1) + [out]
        self.layers = [nn.Dense(w[i], w[i + 1], weight_initializer=nn.initializer.HeNormal()) for i in range(layers)]

    def forward(self, x):
        for layer in self.layers[:-1]:
            x = nn.leaky_relu(layer(x), 0.1)
        return self.layers[-1](x)


def _touch(tensors):
    for t in tensors:
        t._ptr(0)


# ---------------------------------------------------------------------------------------------
# preparation: what a program holds before the call
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    np.random.seed(seed % (1 << 31))
    rng = np.random.default_rng(seed)
    kind, s = case["kind"], dict(case)
    if kind == "serve":
        s["net"] = Classifier(case["width"])
        _touch(s["net"].trainables())
        s["images"] = rng.random((case["batch"], 3, case["size"], case["size"]), np.float32)
    elif kind == "infer":
        s["net"] = Classifier(case["width"])
        _touch(s["net"].trainables())
        s["x"] = _uniform((case["batch"], 3, case["size"], case["size"]), 0.0, 1.0)
    elif kind in ("train", "mlp"):
        if kind == "train":
            s["net"] = Classifier(case["width"], case["api"] == "block")
            s["x"] = _uniform((case["batch"], 3, case["size"], case["size"]), 0.0, 1.0)
            s["t"] = _one_hot(rng, case["batch"], CLASSES)
        else:
            s["net"] = Perceptron(case["features"], case["hidden"], case["layers"], case["out"])
            s["x"] = _normal((case["batch"], case["features"]))
            s["t"] = _one_hot(rng, case["batch"], case["out"])
        s["params"] = s["net"].trainables()
        _touch(s["params"])
        s["opt"] = _optimizer(case["opt"], s["params"])
    elif kind == "dense":
        s["layer"] = nn.Dense(case["in"], case["out"], weight_initializer=nn.initializer.HeNormal(),
                              bias_initializer=nn.initializer.RandomUniform(-0.1, 0.1))
        s["x"] = _normal((case["rows"], case["in"]))
        s["dy"] = _normal((case["rows"], case["out"]), 0.1)
        s["leaves"] = [s["x"], s["layer"].weight, s["layer"].bias]
    elif kind == "matmul":
        lead = () if case["batch"] == 1 else (case["batch"],)
        s["a"] = _normal(lead + (case["m"], case["k"]))
        s["b"] = _normal(lead + (case["k"], case["n"]), case["k"] ** -0.5)
    elif kind == "conv":
        s["layer"] = nn.Conv2D(case["ic"], case["oc"], case["k"], case["stride"], kernel_initializer=nn.initializer.HeNormal(),
                               bias_initializer=nn.initializer.RandomUniform(-0.1, 0.1))
        s["x"] = _normal((case["batch"], case["ic"], case["size"], case["size"]))
        out = _conv_out(case)
        s["dy"] = _normal((case["batch"], case["oc"], out, out), 0.1)
        s["leaves"] = [s["x"], s["layer"].kernel, s["layer"].bias]
    elif kind == "affine":
        shape = (case["batch"], case["ch"], case["size"], case["size"])
        s["x"], s["dy"] = _normal(shape), _normal(shape, 0.1)
        s["g"] = _uniform((1, case["ch"], 1, 1), 0.5, 1.5)
        s["b"] = _uniform((1, case["ch"], 1, 1), -0.5, 0.5)
        s["leaves"] = [s["x"], s["g"], s["b"]]
    elif kind == "pool":
        out = -(-case["size"] // 2)
        s["x"] = _normal((case["batch"], case["ch"], case["size"], case["size"]))
        s["dy"] = _normal((case["batch"], case["ch"], out, out), 0.1)
        s["leaves"] = [s["x"]]
    else:
        s["x"] = _normal((case["d0"], case["d1"], case["d2"]))
        s["axes"] = None if case["axes"] == "all" else (int(case["axes"]),)
        s["dy"] = _normal([d for i, d in enumerate((case["d0"], case["d1"], case["d2"])) if s["axes"] is not None and i not in s["axes"]] or (1,), 0.1)
        s["leaves"] = [s["x"]]
    if "leaves" in s:
        _touch(s["leaves"])
        s["opt"] = nn.optimizer.SGD(s["leaves"])      # makes them trainable; these cases take no step
    nn.devices.wait()
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "serve":
        with nn.optimizer.freeze():
            return state["net"](nn.Tensor_from_value(state["images"])).np()
    if kind == "infer":
        with nn.optimizer.freeze():
            return _outputs(state["net"](state["x"]))
    if kind == "matmul":
        return _outputs(nn.matmul(state["a"], state["b"]))
    opt = state["opt"]
    opt.zero_grad()
    if kind in ("train", "mlp"):
        logits = state["net"](state["x"])
        loss = nn.categorical_crossentropy(nn.softmax(logits), state["t"]).mean()
        loss.backward()
        opt.step()
        return _outputs(loss, logits, *[p.get_grad() for p in state["params"]], *state["params"])
    x = state["x"]
    if kind in ("dense", "conv"):
        y = state["layer"](x)
    elif kind == "affine":
        y = nn.leaky_relu(x * state["g"] + state["b"], 0.1)
    elif kind == "pool":
        y = (nn.max_pool2D if state["op"] == "max" else nn.avg_pool2D)(x, state["pool"], 2)
    else:
        y = {"sum": nn.reduce_sum, "mean": nn.reduce_mean, "max": nn.reduce_max}[state["op"]](x, state["axes"])
    nn.backward({y: state["dy"]})
    return _outputs(y, *[t.get_grad() for t in state["leaves"]])


# ---------------------------------------------------------------------------------------------
# the work of a pass and how near another implementation comes
# ---------------------------------------------------------------------------------------------
def _conv_out(case):
    return (case["size"] - 1) // case["stride"] + 1


def _classifier_work(case):
    """(flops of one forward pass, those of the first convolution, parameters)"""
    ch, size, flops, first, params = _channels(case["width"]), case["size"], 0, 0, 0
    for i in range(4):
        f = 2 * case["batch"] * ch[i] * ch[i + 1] * 9 * size * size
        flops += f
        first = first or f
        params += ch[i] * ch[i + 1] * 9 + ch[i + 1]
        size = -(-size // 2) if i < 3 else size
    flops += 2 * case["batch"] * ch[4] * CLASSES
    return flops, first, params + (ch[4] + 1) * CLASSES


_STATE = {"sgd": 1, "momentum": 1, "rmsprop": 1, "adam": 2}     # tensors an optimizer keeps per parameter


def work(case):
    kind = case["kind"]
    if kind in ("serve", "infer", "train"):
        flops, first, params = _classifier_work(case)
        floats = case["batch"] * (3 * case["size"] ** 2 + CLASSES) + params
        if kind == "train":        # gradients written; parameters and optimizer state read and written
            floats += case["batch"] * CLASSES + params * (2 + 2 * _STATE[case["opt"]])
            flops = 3 * flops - first
        return {"bytes": 4 * floats, "flops": flops}
    if kind == "mlp":
        w = [case["features"]] + [case["hidden"]] * (case["layers"] - 1) + [case["out"]]
        pairs = list(zip(w[:-1], w[1:]))
        params = sum(a * b + b for a, b in pairs)
        macs = case["batch"] * sum(a * b for a, b in pairs)
        floats = case["batch"] * (case["features"] + 2 * case["out"]) + params * (3 + 2 * _STATE[case["opt"]])
        return {"bytes": 4 * floats, "flops": 2 * (3 * macs - case["batch"] * w[0] * w[1])}
    if kind == "dense":
        m, k, n = case["rows"], case["in"], case["out"]
        return {"bytes": 4 * (2 * m * k + 2 * m * n + 2 * k * n + 2 * n), "flops": 6 * m * k * n}
    if kind == "matmul":
        b, m, k, n = case["batch"], case["m"], case["k"], case["n"]
        return {"bytes": 4 * b * (m * k + k * n + m * n), "flops": 2 * b * m * k * n}
    if kind == "conv":
        out = _conv_out(case)
        x = case["batch"] * case["ic"] * case["size"] ** 2
        y = case["batch"] * case["oc"] * out ** 2
        taps = case["ic"] * case["k"] ** 2
        return {"bytes": 4 * (2 * x + 2 * y + 2 * case["oc"] * (taps + 1)), "flops": 6 * y * taps}
    if kind == "affine":
        x = case["batch"] * case["ch"] * case["size"] ** 2
        return {"bytes": 4 * (4 * x + 4 * case["ch"]), "flops": 10 * x}
    if kind == "pool":
        x = case["batch"] * case["ch"] * case["size"] ** 2
        y = case["batch"] * case["ch"] * (-(-case["size"] // 2)) ** 2
        return {"bytes": 4 * (2 * x + 2 * y), "flops": 2 * x}
    x = case["d0"] * case["d1"] * case["d2"]
    y = 1 if case["axes"] == "all" else x // case["d" + case["axes"]]
    return {"bytes": 4 * (2 * x + 2 * y), "flops": 2 * x}


def tolerance(case):
    """fp32 results: sums in another order differ by about 1e-5.  The gradients of a network also pass
    through leaky_relu and max-pooling.  A value nearer to zero (or to its neighbour) than the rounding
    of a 32-bit sum, about one in 10^6, may send its gradient the other way: one of the 10^4 to 10^5
    elements of a small layer's gradient, 1 / sqrt(4 * 10^4) of its norm."""
    if case["kind"] in ("pool", "reduce"):
        return {"rel": 2e-6, "max": 1e-4}
    if case["kind"] in ("train", "mlp"):
        return {"rel": 5e-3, "max": 0.2}
    return {"rel": 1e-5, "max": 1e-3}
