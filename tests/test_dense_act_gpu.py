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
    chains, m._chains, m._chain_ends = m._chains, {}, {}
    n0 = _lib.launch_count()
    out = m.forward(X, training=True)
    m.backward(out, y)
    apart = _lib.launch_count() - n0
    assert len(chains) == 2 and (together < apart or mode == "tf32")
    for l, have in zip(m.layers, got):
        for k, v in have.items():
            want = getattr(l, k)
            if k in ("inputs", "output"):
                assert torch.equal(v, want), (type(l).__name__, k)
            else:
                assert O.rel_l2(v.cpu().numpy(), want.cpu().numpy()) <= 1e-6, (type(l).__name__, k)
    assert _lib.device_status() == 0
