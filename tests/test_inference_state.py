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
