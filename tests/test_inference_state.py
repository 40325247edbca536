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


@pytest.mark.parametrize("room", [8, 6, 5, 2])
def test_several_batches_without_the_memory(monkeypatch, room):
    """A pass over several batches that runs out of memory is done batch by batch, from memory that the pass does not hold."""
    import torch
    from aether_ml_b200.layers import _Workspace
    from aether_ml_b200.model import Model
    seen = []

    def forward(self, X, training, keep=True):
        seen.append((len(X), self.layers[0]._weights_fixed, keep))
        self.layers[0].output = X
        self.layers[0]._ws.buf, self.layers[0]._ws.size = object(), len(X)
        if len(X) > room:
            raise torch.OutOfMemoryError("no room")
        return X
    monkeypatch.setattr(Model, "forward", forward)
    monkeypatch.setattr(Model, "_pass_samples", lambda self, X, batch, most: 6)
    m = Model()
    m.layers = [Layer()]
    m.input_layer = Layer()
    ws = m.layers[0]._ws = _Workspace()
    buf = ws.buf = object()
    X = np.arange(21.0).reshape(21, 1)
    outs = []
    held = m._workspaces()
    for sl, out in m._inference(X, 2, held):
        assert np.array_equal(out, X[sl])
        outs.append(out)
    m._restore_workspaces(held)
    assert np.array_equal(np.vstack(outs), X) and ws.buf is buf
    assert not m.layers[0]._weights_fixed
    if room >= 6:
        assert [n for n, _, _ in seen] == [6, 6, 6, 2, 1] and [f for _, f, _ in seen] == [False] + [True] * 4
    else:
        assert [n for n, _, _ in seen] == [6] + [2] * 10 + [1] and [f for _, f, _ in seen] == [False, False] + [True] * 10
    assert [k for _, _, k in seen] == [False] * (len(seen) - 1) + [True]


def test_one_batch_without_the_memory(monkeypatch):
    """The caller's own batch size not fitting is the caller's to know."""
    import torch
    from aether_ml_b200.model import Model

    def forward(self, X, training, keep=True):
        raise torch.OutOfMemoryError("no room")
    monkeypatch.setattr(Model, "forward", forward)
    monkeypatch.setattr(Model, "_pass_samples", lambda self, X, batch, most: batch)
    m = Model()
    m.layers = [Layer()]
    with pytest.raises(torch.OutOfMemoryError):
        list(m._inference(np.zeros((9, 1)), 2))
