"""Which way a model updates its layers: Optimizer_Adam takes all of them in one launch; a subclass or an instance that
updates in its own way is asked for every layer."""
import pytest


class Layer:
    pass


@pytest.fixture
def updated(monkeypatch):
    """(model, list of what was called), without a device."""
    from aether_ml_b200.layers import Optimizer_Adam
    from aether_ml_b200.model import Model
    calls = []
    monkeypatch.setattr(Optimizer_Adam, "update_layers", lambda self, layers: calls.append(("all", len(layers))))
    monkeypatch.setattr(Optimizer_Adam, "_ensure_state", staticmethod(lambda layer: None))
    monkeypatch.setattr(Optimizer_Adam, "_step", lambda self, *a: calls.append(("adam", a[0])))
    m = Model()
    m.trainable_layers = [Layer(), Layer()]
    for k, l in enumerate(m.trainable_layers):
        for n in ("weights", "dweights", "weight_momentums", "weight_cache", "biases", "dbiases", "bias_momentums", "bias_cache"):
            setattr(l, n, "%s%d" % (n, k))
    return m, calls


EACH = ["weights0", "biases0", "weights1", "biases1"]


def test_itself(updated):
    from aether_ml_b200.layers import Optimizer_Adam
    m, calls = updated
    m.optimizer = Optimizer_Adam()
    m._apply_optimizer()
    assert calls == [("all", 2)] and m.optimizer.iterations == 1


@pytest.mark.parametrize("how", ["subclass step", "subclass update", "instance step", "instance update", "subclass as it is"])
def test_own_way(updated, how):
    from aether_ml_b200.layers import Optimizer_Adam
    m, calls = updated
    if how.startswith("subclass"):
        def _step(self, p, *a):
            calls.append(("own", p))

        def update_parameters(self, layer):
            calls.append(("own", layer))
        body = {"subclass step": {"_step": _step}, "subclass update": {"update_parameters": update_parameters}, "subclass as it is": {}}[how]
        m.optimizer = type("Own", (Optimizer_Adam,), body)()
    else:
        m.optimizer = Optimizer_Adam()
        setattr(m.optimizer, "_step" if how.endswith("step") else "update_parameters", lambda *a: calls.append(("own", a[0])))
    m._apply_optimizer()
    want = list(m.trainable_layers) if how.endswith("update") else EACH
    assert calls == ([("all", 2)] if how == "subclass as it is" else [("own", k) for k in want])
