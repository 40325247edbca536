"""A model runs its layers along `prev` and `next`, also where a caller has wired them otherwise after finalize: a layer that is
skipped in the middle of what would run in one pass (Batch_Norm .. Pooling, Dense and activation, classifier head).  The
wired model is compared with the layers called by hand, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def network(kinds):
    from aether_ml_b200 import layers as L
    from aether_ml_b200.model import Accuracy_Categorical, Model
    np.random.seed(5)
    make = dict(conv=lambda: L.Conv_Layer((8, 8, 16), 16, (3, 3), (1, 1), "same"), bn=lambda: L.Batch_Norm(n_features=16), relu=L.ReLU,
                leaky=lambda: L.Leaky_ReLU(0.1), pool=L.Pooling, flat=L.Flatten, dense=lambda: L.Layer_Dense(256, 256), head=lambda: L.Layer_Dense(256, 10),
                softmax=L.SoftMax)
    m = Model()
    for k in kinds.split():
        m.add(make[k]())
    m.set(loss=L.Loss_CategoricalCrossEntropy(), optimizer=L.Optimizer_Adam(), accuracy=Accuracy_Categorical())
    m.finalize()
    return m


@pytest.mark.parametrize("kinds,skip", [("conv bn relu pool flat head softmax", 1), ("conv bn relu pool flat head softmax", 2),
                                        ("conv bn leaky relu pool flat head softmax", 3), ("flat dense relu dense leaky head softmax", 2),
                                        ("flat dense relu dense leaky head softmax", 4), ("flat dense relu head softmax", 2)])
def test_a_skipped_layer(kinds, skip):
    import torch
    m = network(kinds)
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn((32, 8, 8, 16) if kinds.startswith("conv") else (32, 16, 16, 1), generator=g, device="cuda")
    y = torch.randint(0, 10, (32,), generator=g, device="cuda")
    ls = m.layers
    ls[skip + 1].prev, ls[skip - 1].next = ls[skip - 1], ls[skip + 1]
    out = m.forward(X, training=True)
    m.backward(out, y)
    got = [(l.output.clone(), [d.clone() for d in (getattr(l, "dweights", None), getattr(l, "dbiases", None)) if d is not None])
           for k, l in enumerate(ls) if k != skip]
    rest = [l for k, l in enumerate(ls) if k != skip]
    t = X
    for l in rest:
        t = l.forward(t, True)
    m.softmax_classifier_output.backward(t, y, training=True)
    d = m.softmax_classifier_output.dinputs
    for l in reversed(rest[:-1]):
        l.backward(d)
        d = l.dinputs
    for (o, grads), l in zip(got, rest):
        assert torch.equal(o, l.output), type(l).__name__
        for a, b in zip(grads, (getattr(l, "dweights", None), getattr(l, "dbiases", None))):
            assert float((a - b).norm()) <= 1e-6 * float(b.norm()) + 1e-7, type(l).__name__       # (dB's order differs, fp32)


def _inference_network(kinds):
    """`network` with a head that fits what the Flatten in front of it reads."""
    from aether_ml_b200 import layers as L
    m = network(kinds)
    m.layers[kinds.split().index("head")].__dict__.update(L.Layer_Dense(8 * 8 * 16, 10).__dict__)
    m.finalize()
    return m


def _batch_by_batch(m, X, batch):
    import torch
    return torch.vstack([m.forward(X[k:k + batch], training=False).clone() for k in range(0, len(X), batch)])


@pytest.mark.parametrize("source", [0, 1, 2])
def test_inference_of_several_batches_with_a_layer_that_reads_an_earlier_one(source):
    """The Flatten reads the output of the convolution, the Batch_Norm or the activation, past the layers that would have run in one pass."""
    import torch
    m = _inference_network("conv bn relu pool flat head softmax")
    m.layers[4].prev = m.layers[source]
    X = torch.randn((90, 8, 8, 16), generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    assert torch.equal(m.predict(X, batch_size=16), _batch_by_batch(m, X, 16))


def test_inference_of_several_batches_with_a_layer_of_the_callers():
    """It keeps a convolution's output as its own input, whatever it is handed."""
    import torch
    from aether_ml_b200 import layers as L
    m = _inference_network("conv bn relu pool flat head softmax")

    class Skip(L.Flatten):
        def forward(self, inputs, training):
            return super().forward(self.source.output, training)
    m.layers[4].__class__ = Skip
    m.layers[4].source = m.layers[0]
    m.finalize()
    X = torch.randn((90, 8, 8, 16), generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
    assert torch.equal(m.predict(X, batch_size=16), _batch_by_batch(m, X, 16))
    del m.layers[4].source
    m.layers[4].__class__ = L.Flatten                       # the same with a patched instance
    inner, conv = m.layers[4].forward, m.layers[0]
    m.layers[4].forward = lambda inputs, training: inner(conv.output, training)
    m.finalize()
    assert torch.equal(m.predict(X, batch_size=16), _batch_by_batch(m, X, 16))
