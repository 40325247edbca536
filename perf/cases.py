"""The workloads this framework's speed is judged by, through the entry points a user's program calls: single
convolution layers forward and backward, the bandwidth-bound layers around them, whole train steps (eager and as a
captured graph) and inference.

A case is a dict of plain values.  ``listed()`` names the fixed ones, ``draw(rng)`` gives another one of the same
ranges, ``prepare(case, seed)`` builds what a program holds before the call (layers, models, inputs on the GPU, made
from the seed), ``run(state)`` is one pass, ``work(case)`` the bytes and operations a pass cannot do without and
``tolerance(case)`` how far a correct implementation may be from another one."""
import math

import numpy as np
import torch

from aether_ml_b200 import layers as L
from aether_ml_b200.model import Accuracy_Categorical, Model

CLASSES = 10


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # The smallest network: a dense classifier on 28x28 images, one training step of the plain layer
        # list.  Its kernels take a few microseconds each, so the calls in between are what a user waits for.
        dict(name="mlp step", kind="step", net="mlp", widen=1, batch=128),
        # A training step of the two-block network on 28x28 single-channel images as a script without any option of
        # finalize() runs it: every layer by itself, one optimizer update per layer.
        dict(name="28x28 cnn step", kind="step", net="cnn28", widen=1, batch=256),
        # The three-block network on 32x32 colour images at the batch of the example script, the step captured once
        # and replayed (what Model.train does for flat models), block tails fused.
        dict(name="32x32 cnn graph step", kind="graph", net="cnn32", widen=1, batch=128),
        # The same network four times as wide at a batch of 4096: the largest training configuration.
        dict(name="wide cnn graph step", kind="graph", net="cnn32", widen=4, batch=4096),
        # Inference over a test set in batches, the last of them ragged.
        dict(name="32x32 cnn predict", kind="predict", net="cnn32", widen=1, batch=128, images=1000),
        # Normalisation, activation, spatial dropout and pooling between two convolutions as layers of their own,
        # forward and backward: bound by memory bandwidth.
        dict(name="block tail by layers", kind="tail", S=256, H=32, W=32, C=64, alpha=0.0, rate=0.1, pool="max", window=2),
        # A first layer: three input channels, where a pixel is twelve bytes and a window 27 products long.
        dict(name="conv 32x32 3-32", kind="conv", mode="bf16", S=128, H=32, W=32, Cin=3, Cout=32, f=3, s=1, pad="same"),
        # A deep layer on small images with many channels.
        dict(name="conv 8x8 256-256", kind="conv", mode="bf16", S=256, H=8, W=8, Cin=256, Cout=256, f=3, s=1, pad="same"),
        # The largest single layer.
        dict(name="conv 56x56 64-128", kind="conv", mode="bf16", S=256, H=56, W=56, Cin=64, Cout=128, f=3, s=1, pad="same"),
        # TF32 operands, chosen by users who want three decimal digits.
        dict(name="conv tf32 16x16 128-128", kind="conv", mode="tf32", S=256, H=16, W=16, Cin=128, Cout=128, f=3, s=1, pad="same"),
        # Downsampling by a strided convolution, at an image size and channel counts that fit no tile.
        dict(name="conv stride 2 57x45 48-72", kind="conv", mode="bf16", S=100, H=57, W=45, Cin=48, Cout=72, f=3, s=2, pad="same"),
        # Single precision all the way, as the arrays are.
        dict(name="conv fp32 28x28 32-64", kind="conv", mode="fp32", S=96, H=28, W=28, Cin=32, Cout=64, f=3, s=1, pad="same"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo, hi):
    c = _log_int(rng, lo, hi)
    how = rng.random()
    return max(16, c // 16 * 16) if how < 0.4 else max(4, c // 4 * 4) if how < 0.85 else c


# A drawn case stays below the largest listed one of its kind: operations, and bytes of inputs and outputs.
_MOST_CONV = {"tensor": 355e9, "strided": 15e9, "fp32": 8e9}
_MOST_BYTES = 1.3e9


def draw(rng):
    kind = rng.choices(("conv", "step", "graph", "predict", "tail"), (10, 4, 3, 2, 3))[0]
    while True:
        if kind == "conv":
            side = _log_int(rng, 7, 64)
            first = rng.random() < 0.2
            c = dict(kind=kind, mode=rng.choices(("bf16", "tf32", "fp32"), (5, 3, 2))[0], S=_log_int(rng, 4, 512), H=side,
                     W=max(7, side + rng.choice((0, 0, 0, -5, 1, 8))), Cin=rng.choice((1, 3)) if first else _channels(rng, 16, 256),
                     Cout=_channels(rng, 16, 256), f=rng.choices((1, 3, 5), (1, 7, 2))[0], s=2 if rng.random() < 0.2 else 1,
                     pad=rng.choice(("same", "same", "valid")))
            w = work(c)
            most = _MOST_CONV["fp32" if c["mode"] == "fp32" else "strided" if c["s"] > 1 or c["Cin"] % 4 or c["Cout"] % 4 else "tensor"]
            if w["flops"] <= most and w["bytes"] <= _MOST_BYTES:
                return c
        elif kind == "tail":
            pool = rng.choice(("max", "max", "average"))
            side = _log_int(rng, 7, 64)
            c = dict(kind=kind, S=_log_int(rng, 8, 1024), H=side, W=side + rng.choice((0, 0, 1)), C=_channels(rng, 8, 256),
                     alpha=rng.choice((0.0, 0.01)), rate=rng.choice((0.075, 0.1, 0.25)), pool=pool, window=rng.choice((2, 2, 3)))
            if work(c)["bytes"] <= _MOST_BYTES:
                return c
        else:
            net = rng.choices(("mlp", "cnn28", "cnn32"), (1, 2, 3))[0]
            c = dict(kind=kind, net=net, widen=rng.choice((1, 1, 2, 4)), batch=_log_int(rng, 16, 1024))
            if kind == "predict":
                c["images"] = _log_int(rng, 1, 8000)
            return c


# ------------------------------------------------------------------------------------------------ networks
def _network(net, widen, seed):
    """Layer lists of the repository's training configurations.  Parameters come from NumPy's generator, as the layers
    draw them; the dropout layers are seeded."""
    np.random.seed(seed % (1 << 31))
    m = Model()

    def spatial(rate):
        layer = L.Layer_Dropout_Spatial(rate)
        layer.seed = seed + 1
        m.add(layer)

    if net == "mlp":
        n = 128 * widen
        m.add(L.Flatten())
        m.add(L.Layer_Dense(784, n))
        m.add(L.ReLU())
        m.add(L.Layer_Dense(n, n))
        m.add(L.ReLU())
        m.add(L.Layer_Dense(n, CLASSES))
    elif net == "cnn28":
        c_in, hw = 1, 28
        for c_out in (32 * widen, 64 * widen):
            m.add(L.Conv_Layer((hw, hw, c_in), c_out, (3, 3), (1, 1), "same"))
            m.add(L.Batch_Norm(n_features=c_out))
            m.add(L.ReLU())
            m.add(L.Pooling((2, 2), (2, 2), "valid", "max"))
            c_in, hw = c_out, hw // 2
        m.add(L.Flatten())
        m.add(L.Layer_Dense(hw * hw * c_in, 128 * widen))
        m.add(L.ReLU())
        m.add(L.Layer_Dense(128 * widen, CLASSES))
    else:
        c_in, hw = 3, 32
        for c_out, rate in ((32 * widen, 0.075), (64 * widen, 0.1), (128 * widen, None)):
            m.add(L.Conv_Layer((hw, hw, c_in), c_out, (3, 3), (1, 1), "same"))
            m.add(L.Batch_Norm(n_features=c_out))
            m.add(L.ReLU())
            if rate:
                spatial(rate)
            m.add(L.Pooling((2, 2), (2, 2), "valid", "max"))
            c_in, hw = c_out, hw // 2
        m.add(L.Flatten())
        m.add(L.Layer_Dense(hw * hw * c_in, 256 * widen, weight_regularizer_l2=2e-5))
        m.add(L.Leaky_ReLU(0.01))
        m.add(L.Layer_Dropout(0.075, seed=seed + 2))
        m.add(L.Layer_Dense(256 * widen, CLASSES))
    m.add(L.SoftMax())
    m.set(loss=L.Loss_CategoricalCrossEntropy(label_smoothing=0.01),
          optimizer=L.Optimizer_Adam(learning_rate=1e-3, decay=5e-5), accuracy=Accuracy_Categorical())
    return m


def _image(net):
    return {"mlp": (28, 28, 1), "cnn28": (28, 28, 1), "cnn32": (32, 32, 3)}[net]


def _resume(m, g):
    """The state of a run that has been going for a while, as a checkpoint with the optimizer's state restores it:
    moments of plausible size, running statistics away from their initial values.  (From zero moments the first update
    is the sign of the gradient, whatever its size.)"""
    for layer in m.trainable_layers:
        for p, mom, cache in ((layer.weights, "weight_momentums", "weight_cache"), (layer.biases, "bias_momentums", "bias_cache")):
            a = torch.randn(p.shape, generator=g, device=p.device) * 1e-3
            b = torch.rand(p.shape, generator=g, device=p.device) * 1e-4 + 1e-6
            if hasattr(layer, cache):
                getattr(layer, mom).copy_(a)
                getattr(layer, cache).copy_(b)
            else:
                setattr(layer, mom, a)
                setattr(layer, cache, b)
        if isinstance(layer, L.Batch_Norm):
            n = layer.gamma.numel()
            layer.set_parameters(torch.rand(n, generator=g, device="cuda") + 0.5, torch.randn(n, generator=g, device="cuda") * 0.1,
                                 torch.randn(n, generator=g, device="cuda") * 0.1, torch.rand(n, generator=g, device="cuda") + 0.2)
    m.optimizer.iterations = 1000


# ------------------------------------------------------------------------------------------------ inputs and handles
def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind == "conv":
        np.random.seed(seed % (1 << 31))
        f = (case["f"], case["f"])
        layer = L.Conv_Layer((case["H"], case["W"], case["Cin"]), case["Cout"], f, (case["s"], case["s"]), case["pad"],
                             math_mode=case["mode"])
        layer.biases.copy_(torch.randn(case["Cout"], generator=g, device="cuda") * 0.1)
        shape = (case["S"], case["H"], case["W"], case["Cin"])
        if case["Cin"] <= 3:                        # images
            x = torch.rand(shape, generator=g, device="cuda")
        else:
            x = torch.randn(shape, generator=g, device="cuda")
        Ho, Wo = _conv_out(case)
        dy = torch.randn((case["S"], Ho, Wo, case["Cout"]), generator=g, device="cuda")
        return dict(kind=kind, layer=layer, x=x, dy=dy)
    if kind == "tail":
        np.random.seed(seed % (1 << 31))
        n, k = case["C"], case["window"]
        bn = L.Batch_Norm(n_features=n)
        bn.set_parameters(torch.rand(n, generator=g, device="cuda") + 0.5, torch.randn(n, generator=g, device="cuda") * 0.1,
                          torch.zeros(n, device="cuda"), torch.ones(n, device="cuda"))
        act = L.Leaky_ReLU(case["alpha"]) if case["alpha"] else L.ReLU()
        drop = L.Layer_Dropout_Spatial(case["rate"])
        pool = L.Pooling((k, k), (k, k), "valid", case["pool"])
        x = torch.randn((case["S"], case["H"], case["W"], n), generator=g, device="cuda")
        dy = torch.randn((case["S"], case["H"] // k, case["W"] // k, n), generator=g, device="cuda")
        return dict(kind=kind, layers=(bn, act, drop, pool), x=x, dy=dy)
    m = _network(case["net"], case["widen"], int(seed))
    rows = case.get("images", case["batch"])
    X = torch.rand((rows,) + _image(case["net"]), generator=g, device="cuda")
    y = torch.randint(0, CLASSES, (rows,), generator=g, device="cuda")
    if kind == "graph":
        m.finalize(flat=True, fuse=True, lean=True)
        _resume(m, g)
        m.capture_train_step(X, y)
    else:
        m.finalize()
        _resume(m, g)
    return dict(kind=kind, model=m, X=X, y=y, batch=case["batch"])


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "conv":
        layer = state["layer"]
        y = layer.forward(state["x"], training=True)
        dx = layer.backward(state["dy"])
        return y, dx, layer.dweights, layer.dbiases
    if kind == "tail":
        t = state["x"]
        for layer in state["layers"]:
            t = layer.forward(t, training=True)
        out, d = t, state["dy"]
        for layer in reversed(state["layers"]):
            d = layer.backward(d)
        bn = state["layers"][0]
        return out, d, bn.dweights, bn.dbiases, bn.running_mean, bn.running_var
    m = state["model"]
    if kind == "predict":
        return m.predict(state["X"], batch_size=state["batch"])
    if kind == "graph":
        out = m.train_step_graph(state["X"], state["y"])
        return out, m.flat_params, m.flat_grads, m.flat_m, m.flat_v, _running(m)
    out = m.train_step(state["X"], state["y"])
    return out, [_arrays(m, i) for i in range(len(m.trainable_layers))], _running(m)


def _arrays(m, i):
    """A layer's parameters, gradients and moments after the step.  The bias gradient of a convolution in front of a
    Batch_Norm is zero in exact arithmetic (the mean takes it out again), so what stands there is rounding alone."""
    layer = m.trainable_layers[i]
    follows = m.trainable_layers[i + 1] if i + 1 < len(m.trainable_layers) else None
    cancels = isinstance(layer, L.Conv_Layer) and isinstance(follows, L.Batch_Norm)
    return [layer.weights, layer.biases, layer.dweights, None if cancels else layer.dbiases, layer.weight_momentums,
            layer.weight_cache, layer.bias_momentums]


def _running(m):
    return [(layer.running_mean, layer.running_var) for layer in m.trainable_layers if isinstance(layer, L.Batch_Norm)]


# ------------------------------------------------------------------------------------------------ bytes and operations
def _conv_out(case):
    p = (case["f"] - 1) // 2 if case["pad"] == "same" else 0
    return tuple((n + 2 * p - case["f"]) // case["s"] + 1 for n in (case["H"], case["W"]))


def _net_work(net, widen):
    """(parameters, forward products of one image, those of its first layer)."""
    w = widen
    if net == "mlp":
        dims = [784, 128 * w, 128 * w, CLASSES]
        macs = [a * b for a, b in zip(dims, dims[1:])]
        return sum(a * b + b for a, b in zip(dims, dims[1:])), sum(macs), macs[0]
    c, hw, widths, dense = (1, 28, (32 * w, 64 * w), 128 * w) if net == "cnn28" else (3, 32, (32 * w, 64 * w, 128 * w), 256 * w)
    params, macs = 0, []
    for n in widths:
        params += 9 * c * n + n + 2 * n
        macs.append(hw * hw * 9 * c * n)
        c, hw = n, hw // 2
    for a, b in ((hw * hw * c, dense), (dense, CLASSES)):
        params += a * b + b
        macs.append(a * b)
    return params, sum(macs), macs[0]


def work(case):
    kind = case["kind"]
    if kind == "conv":
        Ho, Wo = _conv_out(case)
        ins, outs = case["S"] * case["H"] * case["W"] * case["Cin"], case["S"] * Ho * Wo * case["Cout"]
        w = case["f"] * case["f"] * case["Cin"] * case["Cout"] + case["Cout"]
        # read x, dy and the filter, write y, dx and the filter's gradient; three products of the same size
        return dict(bytes=4.0 * (2 * ins + 2 * outs + 2 * w), flops=6.0 * outs * case["f"] * case["f"] * case["Cin"])
    if kind == "tail":
        n, k = case["S"] * case["H"] * case["W"] * case["C"], case["window"]
        small = case["S"] * (case["H"] // k) * (case["W"] // k) * case["C"]
        return dict(bytes=4.0 * (2 * n + 2 * small), flops=16.0 * n)
    params, macs, first = _net_work(case["net"], case["widen"])
    pixels = math.prod(_image(case["net"]))
    if kind == "predict":
        return dict(bytes=4.0 * (case["images"] * (pixels + CLASSES) + params), flops=2.0 * case["images"] * macs)
    # the batch; parameters and two moments read and written, gradients written; nobody asks for the images' gradient
    return dict(bytes=4.0 * (case["batch"] * (pixels + CLASSES) + 7 * params), flops=2.0 * case["batch"] * (3 * macs - first))


# ------------------------------------------------------------------------------------------------ tolerances
def tolerance(case):
    kind = case["kind"]
    if kind == "conv":
        # relative error of the operands' rounding (8, 11 or 24 bits of mantissa), as the tests of each mode have it
        return {"rel": {"bf16": 1e-2, "tf32": 1e-3, "fp32": 1e-5}[case["mode"]]}
    if kind == "tail":
        if case["pool"] == "average":
            return {"rel": 1e-5}
        # Two cells of a window within a rounding of each other may change places: of 10 million values some, and each
        # moves a whole gradient from one cell to the next.
        return {"rel": 1e-3, "max": 0.99}
    # bf16 operands throughout; a pooling window's maximum may move as above
    return {"rel": 1e-2, "max": 0.99}
