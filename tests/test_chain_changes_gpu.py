"""Arrays changed between the forward and the backward pass: the layers that run in one pass then give what they give one by
one, the activation's mask from its inputs as they were, Batch_Norm's gradient from its inputs as they are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["nothing", "bn.inputs", "act.inputs", "bn.gamma"])
@pytest.mark.parametrize("pool", [True, False])
def test_changed_between_the_passes(what, pool):
    import torch
    from aether_ml_b200 import layers as L
    from aether_ml_b200.model import Accuracy_Categorical, Model
    grads = []
    for apart in (False, True):
        np.random.seed(5)
        m = Model()
        m.add(L.Conv_Layer((8, 8, 16), 32, (3, 3), (1, 1), "same"))
        m.add(L.Batch_Norm(n_features=32))
        m.add(L.ReLU())
        if pool:
            m.add(L.Pooling())
        m.add(L.Flatten())
        m.add(L.Layer_Dense(512 if pool else 2048, 10))
        m.add(L.SoftMax())
        m.set(loss=L.Loss_CategoricalCrossEntropy(), optimizer=L.Optimizer_Adam(), accuracy=Accuracy_Categorical())
        m.finalize()
        if apart:
            m._chains, m._chain_ends = {}, {}
        g = torch.Generator(device="cuda").manual_seed(1)
        X, y = torch.randn((16, 8, 8, 16), generator=g, device="cuda"), torch.randint(0, 10, (16,), generator=g, device="cuda")
        out = m.forward(X, training=True)
        bn, act = m.layers[1], m.layers[2]
        change = torch.randn(bn.inputs.shape, generator=g, device="cuda")
        if what == "bn.inputs":
            bn.inputs.copy_(change)
        elif what == "act.inputs":
            act.inputs.copy_(change)
        elif what == "bn.gamma":
            bn.gamma.mul_(-0.5)
        m.backward(out, y)
        grads.append([act.dinputs, bn.dinputs, bn.dweights, bn.dbiases, m.layers[0].dweights])
    for a, b in zip(*grads):
        assert float((a - b).norm() / b.norm()) <= 1e-5            # (fp32 sums in another order; bf16 operands of equal arrays)
