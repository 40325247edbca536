"""Inference over several batches at once stays within its bound of memory, workspaces included, gives the workspaces back when
the call ends, and leaves layers whose backward pass is right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def network():
    from aether_ml_b200 import layers as L
    from aether_ml_b200.model import Accuracy_Categorical, Model
    np.random.seed(5)
    m = Model()
    m.add(L.Conv_Layer((16, 16, 3), 16, (3, 3), (1, 1), "same"))
    m.add(L.Batch_Norm(n_features=16))
    m.add(L.ReLU())
    m.add(L.Pooling((2, 2), (2, 2), "valid", "max"))
    m.add(L.Conv_Layer((8, 8, 16), 32, (3, 3), (1, 1), "same"))
    m.add(L.Batch_Norm(n_features=32))
    m.add(L.ReLU())
    m.add(L.Flatten())
    m.add(L.Layer_Dense(8 * 8 * 32, 64))
    m.add(L.ReLU())
    m.add(L.Layer_Dense(64, 10))
    m.add(L.SoftMax())
    m.set(loss=L.Loss_CategoricalCrossEntropy(), optimizer=L.Optimizer_Adam(), accuracy=Accuracy_Categorical())
    m.finalize()
    return m


@pytest.mark.parametrize("trained", [True, False])          # what the layers have seen before: three steps, or one batch
@pytest.mark.parametrize("call", ["predict", "evaluate"])
def test_workspaces_are_given_back(call, trained):
    import torch
    m = network()
    g = torch.Generator(device="cuda").manual_seed(3)
    X, y = torch.rand((200, 16, 16, 3), generator=g, device="cuda"), torch.randint(0, 10, (200,), generator=g, device="cuda")
    if trained:
        for k in range(3):
            m.train_step(X[8 * k:8 * k + 8], y[8 * k:8 * k + 8])
    else:
        m.forward(X[:8], training=False)
    held = m._workspaces()
    assert m._pass_samples(X, 8, 192) == 192
    for _ in range(2):
        m.predict(X, batch_size=8) if call == "predict" else m.evaluate(X, y, batch_size=8)
        assert all(w.buf is buf for _, w, buf, _ in held if buf is not None)
    # the layers stand as the last batch left them: a backward pass of theirs is that of a fresh forward pass
    for l in (m.layers[4], m.layers[8]):
        junk = [torch.full((1 << 22,), float("nan"), device="cuda") for _ in range(8)]       # over the memory that was given back
        del junk
        dy = torch.randn(l.output.shape, generator=g, device="cuda")
        dx = l.backward(dy).clone()
        grads = l.dweights.clone(), l.dbiases.clone()
        l.forward(l.inputs.clone(), training=True)
        assert torch.equal(l.backward(dy), dx) and torch.equal(l.dweights, grads[0]) and torch.equal(l.dbiases, grads[1])


@pytest.mark.parametrize("limit", [1, 300_000, 3_000_000, 20_000_000])
def test_the_bound_counts_workspaces(limit):
    import torch
    m = network()
    m.INFERENCE_PASS_BYTES = limit
    X = torch.rand((300, 16, 16, 3), device="cuda")
    n = m._pass_samples(X, 7, 294)
    assert n % 7 == 0 and 7 <= n <= 294
    per_sample, working = m._output_bytes((16, 16, 3))
    assert len(working) == 4 and (n == 7 or n * per_sample + sum(l._plan((n, *s) if s else n).ws_bytes for l, s in working) <= limit)
    want = torch.vstack([m.forward(X[k:k + 7], training=False) for k in range(0, 300, 7)])
    got = m.predict(X, batch_size=7)
    assert float((got - want).norm() / want.norm()) <= 1e-4         # (fp32 sums of bf16 products in tiles of another size)
