"""A Dense layer and the (leaky) ReLU behind it in one launch each way against the same layers one by one: the forward pass
bit by bit (the same products and roundings), gradients up to the order of dB's sum (fp32, relative L2 <= 1e-6).  Row counts
around the 128-row tiles and the limit of the one-launch backward pass, channel counts with padded operand rows, a consumer
that takes the operand copy and one that does not, large batches that take CTA pairs, TF32 (no such epilogue)."""
import numpy as np
import pytest

from oracle import aether_oracle as O

pytestmark = pytest.mark.gpu


def network(n_in, n_mid, alpha, mode):
    from aether_ml_b200 import layers as L
    from aether_ml_b200.model import Accuracy_Categorical, Model
    np.random.seed(n_in + n_mid)
    m = Model()
    m.add(L.Layer_Dense(n_in, n_mid, math_mode=mode))
    m.add(L.Leaky_ReLU(alpha) if alpha else L.ReLU())
    m.add(L.Layer_Dense(n_mid, 64, math_mode=mode))
    m.add(L.ReLU())
    m.add(L.Layer_Dense(64, 10, math_mode=mode))
    m.add(L.SoftMax())
    m.set(loss=L.Loss_CategoricalCrossEntropy(), optimizer=L.Optimizer_Adam(), accuracy=Accuracy_Categorical())
    m.finalize()
    return m


@pytest.mark.parametrize("rows,n_in,n_mid,alpha,mode", [(1, 64, 64, 0.0, "bf16"), (31, 100, 32, 0.01, "bf16"), (128, 784, 128, 0.0, "bf16"),
                                                        (129, 48, 100, 0.3, "bf16"), (1000, 64, 260, 0.0, "bf16"), (1024, 32, 36, 0.0, "bf16"),
                                                        (1025, 128, 64, 0.01, "bf16"), (40000, 64, 128, 0.0, "bf16"), (200, 96, 64, 0.01, "tf32")])
def test_matches_layers(rows, n_in, n_mid, alpha, mode):
    import torch
    from aether_ml_b200 import _lib
    m = network(n_in, n_mid, alpha, mode)
    g = torch.Generator(device="cuda").manual_seed(rows)
    X = torch.randn((rows, n_in), generator=g, device="cuda")
    y = torch.randint(0, 10, (rows,), generator=g, device="cuda")
    n0 = _lib.launch_count()
    out = m.forward(X, training=True)
    m.backward(out, y)
    together = _lib.launch_count() - n0
    names = ("inputs", "output", "dinputs", "dweights", "dbiases")
    got = [{k: getattr(l, k).clone() for k in names if getattr(l, k, None) is not None} for l in m.layers]
    chains, m._chains, m._chain_ends = m._chains, {}, {}               # layer by layer
    n0 = _lib.launch_count()
    out = m.forward(X, training=True)
    m.backward(out, y)
    apart = _lib.launch_count() - n0
    assert len(chains) == 3 and (together < apart or mode == "tf32")         # two of these pairs, and the classifier head
    for l, have in zip(m.layers, got):
        for k, v in have.items():
            want = getattr(l, k)
            if k in ("inputs", "output"):
                assert torch.equal(v, want), (type(l).__name__, k)
            else:
                assert O.rel_l2(v.cpu().numpy(), want.cpu().numpy()) <= 1e-6, (type(l).__name__, k)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("rows,n_in,classes,kind", [(1, 128, 10, "int64"), (7, 132, 2, "int32"), (300, 256, 15, "soft"), (1000, 1024, 10, "int64"),
                                                    (33, 128, 16, "int64"), (20, 64, 10, "int32")])
def test_head_matches_layers(rows, n_in, classes, kind):
    """A classifier head with its SoftMax and the combined gradient in one launch each: the same operations, bit by bit
    (16 classes and 64 inputs are no heads and run layer by layer)."""
    import torch
    from aether_ml_b200 import _lib, layers as L
    from aether_ml_b200.model import Accuracy_Categorical, Model
    np.random.seed(classes)
    m = Model()
    m.add(L.Flatten())
    m.add(L.Layer_Dense(n_in, classes, weight_regularizer_l2=1e-3))
    m.add(L.SoftMax())
    m.set(loss=L.Loss_CategoricalCrossEntropy(label_smoothing=0.1), optimizer=L.Optimizer_Adam(), accuracy=Accuracy_Categorical())
    m.finalize()
    g = torch.Generator(device="cuda").manual_seed(rows)
    X = torch.randn((rows, n_in), generator=g, device="cuda") * 30
    if kind == "soft":
        y = torch.softmax(torch.randn((rows, classes), generator=g, device="cuda"), 1)
    else:
        y = torch.randint(0, classes, (rows,), generator=g, device="cuda", dtype=torch.int64 if kind == "int64" else torch.int32)
    n0 = _lib.launch_count()
    m.backward(m.forward(X, training=True), y)
    together = _lib.launch_count() - n0
    names = ("inputs", "output", "dinputs", "dweights", "dbiases")
    got = [{k: getattr(l, k).clone() for k in names if getattr(l, k, None) is not None} for l in m.layers]
    m._chains, m._chain_ends = {}, {}
    n0 = _lib.launch_count()
    m.backward(m.forward(X, training=True), y)
    assert _lib.launch_count() - n0 - together == (2 if n_in >= 128 and classes < 16 else 0)
    for l, have in zip(m.layers, got):
        for k, v in have.items():
            assert torch.equal(v, getattr(l, k)), (type(l).__name__, k)
