"""Captured train steps: operand copies of the weights and the parameters' gradients on a second stream inside the graph.  Replays give the bits
of eager steps, whatever the layers: fused and lean block tails, single layers, regularizers, odd batches, weights replaced and an
inference in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(net, options):
    from aether_ml_b200 import layers as L
    from aether_ml_b200.model import Accuracy_Categorical, Model
    np.random.seed(3)
    m = Model()
    if net == "cnn":
        c, hw = 3, 20
        for n in (16, 64, 72):
            for l in (L.Conv_Layer((hw, hw, c), n, (3, 3), (1, 1), "same"), L.Batch_Norm(n_features=n), L.ReLU()):
                m.add(l)
            if n < 72:
                m.add(L.Pooling((2, 2), (2, 2), "valid", "max"))
                hw //= 2
            c = n
        m.add(L.Flatten())
        sizes = (hw * hw * c, 192, 100)
    else:
        m.add(L.Flatten())
        sizes = (20 * 20 * 3, 128, 136)
    for a, b in zip(sizes, sizes[1:]):
        m.add(L.Layer_Dense(a, b, weight_regularizer_l2=1e-3, bias_regularizer_l2=1e-3, weight_regularizer_l1=1e-4))
        m.add(L.Leaky_ReLU(0.01))
    m.add(L.Layer_Dense(sizes[-1], 10))
    m.add(L.SoftMax())
    m.set(loss=L.Loss_CategoricalCrossEntropy(), optimizer=L.Optimizer_Adam(learning_rate=1e-3, decay=1e-4), accuracy=Accuracy_Categorical())
    m.finalize(flat=True, **options)
    return m


@pytest.mark.parametrize("net,options,batch", [("cnn", dict(fuse=True, lean=True), 37), ("cnn", dict(fuse=True), 128), ("cnn", {}, 64), ("mlp", {}, 1), ("mlp", {}, 300)])
def test_replays_are_the_eager_steps(net, options, batch):
    import torch
    from aether_ml_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(batch)
    X = [torch.rand((batch, 20, 20, 3), generator=g, device="cuda") for _ in range(4)]
    y = [torch.randint(0, 10, (batch,), generator=g, device="cuda") for _ in range(4)]
    eager, graph = _model(net, options), _model(net, options)
    eager.enable_device_step()
    graph.capture_train_step(X[0], y[0])
    for k in range(4):
        if k == 2:                                          # other weights, and a pass over another batch in between
            for m in (eager, graph):
                m.flat_params.mul_(1.001)
                m.predict(X[0][: batch // 2 + 1])
        a, b = eager.train_step(X[k], y[k]).clone(), graph.train_step_graph(X[k], y[k])
        assert torch.equal(a, b), k
        for name in ("flat_grads", "flat_params", "flat_m", "flat_v"):
            assert torch.equal(getattr(eager, name), getattr(graph, name)), (k, name)
    assert all(l.__dict__.get("_branch") is None and not l._weights_fixed for l in graph.layers if hasattr(l, "_weights_fixed"))
    graph.release_graphs()
    assert _lib.device_status() == 0
