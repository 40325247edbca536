"""Captured train steps: operand copies of the weights and the parameters' gradients on a second stream inside the graph.  Replays give the bits
of eager steps, whatever the layers: fused and lean block tails, single layers, regularizers, odd batches, weights replaced and an
inference in between.  Methods of the caller's that use weights or gradients find them where they run: such a model has no second stream."""
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


@pytest.mark.parametrize("own", ["layer subclass", "patched layer", "model subclass", "patched model", "other layer"])
@pytest.mark.parametrize("net", ["cnn", "mlp"])
def test_methods_of_the_caller(net, own, monkeypatch):
    import torch
    from aether_ml_b200 import _lib, layers as L
    from aether_ml_b200.model import Model

    def clip(layer):
        layer.dweights.clamp_(-1e-3, 1e-3)

    def build():
        m = _model(net, {})
        dense = [l for l in m.layers if type(l) is L.Layer_Dense][1]
        layer = m.layers[4] if net == "cnn" and own != "other layer" else dense
        if own == "layer subclass":
            class Clipped(type(layer)):
                def backward(self, dvalues, **kwargs):
                    out = super().backward(dvalues, **kwargs)
                    clip(self)
                    return out
            layer.__class__ = Clipped
        elif own == "patched layer":
            inner = layer.backward
            layer.backward = lambda d, **kwargs: (inner(d, **kwargs), clip(layer))[0]
        elif own == "model subclass":
            class Clipping(Model):
                def backward(self, output, y):
                    super().backward(output, y)
                    for l in self.trainable_layers:
                        clip(l)
            m.__class__ = Clipping
        elif own == "patched model":
            back = m.backward
            m.backward = lambda output, y: (back(output, y), clip(layer))[0]
        else:
            class Looking(L.Leaky_ReLU):
                def backward(self, dvalues):
                    clip(self.next)
                    return super().backward(dvalues)
            layer.prev.__class__ = Looking
        m.finalize()                                        # (what runs in one pass is decided anew)
        return m
    monkeypatch.setattr(L._Branch, "fork", lambda *a: pytest.fail("on a second stream"))
    g = torch.Generator(device="cuda").manual_seed(9)
    X = [torch.rand((48, 20, 20, 3), generator=g, device="cuda") for _ in range(3)]
    y = [torch.randint(0, 10, (48,), generator=g, device="cuda") for _ in range(3)]
    eager, graph = build(), build()
    eager.enable_device_step()
    graph.capture_train_step(X[0], y[0])
    for k in range(3):
        a, b = eager.train_step(X[k], y[k]).clone(), graph.train_step_graph(X[k], y[k])
        assert torch.equal(a, b) and torch.equal(eager.flat_grads, graph.flat_grads) and torch.equal(eager.flat_params, graph.flat_params)
    graph.release_graphs()
    assert _lib.device_status() == 0
