"""What an inference over several batches leaves behind, without a device."""
import numpy as np
import pytest


class Layer:
    _weights_fixed = False


@pytest.fixture
def model(monkeypatch):
    """A model whose passes are recorded: (number of samples, keyword arguments, whether the layer took its weights as fixed)."""
    from aether_ml_b200.model import Model
    passes = []

    def forward(self, X, training, **kw):
        passes.append((len(X), kw, self.layers[0]._weights_fixed))
        return X
    monkeypatch.setattr(Model, "forward", forward)
    m = Model()
    m.layers = [Layer()]
    return m, passes


def test_weights_are_fixed_during_a_pass_only(model):
    """A loop over the passes that is left in the middle (a wrong label, an interrupt: the traceback keeps the loop alive) must
    not leave the layers believing that their weights cannot change."""
    m, passes = model
    loop = m._inference(np.zeros((10, 3)), 2)
    for _ in range(3):
        next(loop)
        assert not m.layers[0]._weights_fixed
    assert [fixed for _, _, fixed in passes] == [False, True, True]
    list(loop)
    assert not m.layers[0]._weights_fixed and len(passes) == 5


@pytest.mark.parametrize("how", ["subclass", "instance"])
@pytest.mark.parametrize("images,batch,sizes", [(10, 2, [2] * 5), (7, 3, [3, 3, 1]), (5, None, [5])])
def test_a_forward_of_the_callers_own(how, images, batch, sizes):
    """It is called with the batches the caller asked for and the arguments it has always had."""
    from aether_ml_b200.model import Model
    seen = []

    def forward(self, X, training):
        seen.append((len(X), training))
        return X
    if how == "subclass":
        m = type("Own", (Model,), {"forward": forward})()
    else:
        m = Model()
        m.forward = lambda X, training: forward(m, X, training)
    m.layers = [Layer()]
    X = np.arange(3.0 * images).reshape(images, 3)
    out = [o for _, o in m._inference(X, batch)]
    assert seen == [(n, False) for n in sizes] and np.array_equal(np.vstack(out), X)


def test_a_forward_that_reuses_its_output():
    """predict keeps what each pass returned, also when the next pass writes into the same array."""
    import torch
    from aether_ml_b200.layers import SoftMax
    from aether_ml_b200.model import Model
    buffer = torch.empty(2, 3)
    m = Model()
    m.layers = [SoftMax()]
    m.forward = lambda X, training: buffer.copy_(torch.as_tensor(X))
    X = np.arange(18.0).reshape(6, 3)
    assert np.array_equal(m.predict(X, batch_size=2).numpy(), X)
