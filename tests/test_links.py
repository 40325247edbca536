"""Who owns whom: a model's layers do not own their neighbours (a dropped model frees its memory at once), a layer that a caller
links by hand owns what it was given, as any attribute does."""
import gc
import weakref

import pytest


@pytest.fixture
def no_collector():
    gc.collect()
    gc.disable()
    yield
    gc.enable()


def test_links_set_by_hand(no_collector):
    from aether_ml_b200.layers import Layer_Dropout, Leaky_ReLU, ReLU
    first = ReLU()
    first.next = Leaky_ReLU(0.1)
    first.next.next = Layer_Dropout(0.5)
    assert isinstance(first.next, Leaky_ReLU) and isinstance(first.next.next, Layer_Dropout)
    first.prev = "input"
    assert first.prev == "input" and not hasattr(first.next, "prev")
    first.next = None
    assert first.next is None


def test_links_of_a_model(no_collector):
    from aether_ml_b200.layers import Flatten, Loss_CategoricalCrossEntropy, Optimizer_Adam, ReLU, SoftMax
    from aether_ml_b200.model import Accuracy_Categorical, Model
    m = Model()
    for l in (Flatten(), ReLU(), SoftMax()):
        m.add(l)
    m.set(loss=Loss_CategoricalCrossEntropy(), optimizer=Optimizer_Adam(), accuracy=Accuracy_Categorical())
    m.finalize()
    a, b, c = m.layers
    assert a.prev is m.input_layer and a.next is b and b.prev is a and b.next is c and c.next is m.loss
    refs = [weakref.ref(l) for l in (a, b, c)]
    del a, b, c, l, m
    assert all(r() is None for r in refs)
