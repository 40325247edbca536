"""The (leaky) ReLU's way back by the bits its forward pass kept: the same numbers as from the inputs, at sizes around the groups of 128 values, with
zeros, signed zeros, infinities and NaN; inputs replaced or changed in between are read again, and none are kept of arrays whose changes nobody counts."""
import pytest

pytestmark = pytest.mark.gpu


def _values(n, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(n, generator=g, device="cuda")
    special = torch.tensor([0.0, -0.0, float("inf"), -float("inf"), float("nan"), 1e-45, -1e-45], device="cuda")
    at = torch.randint(0, n, (min(n, 700),), generator=g, device="cuda")
    x[at] = special[torch.arange(len(at), device="cuda") % 7]
    return x


@pytest.mark.parametrize("n", [4, 124, 128, 132, 1020, 4096, 4100, 1184 * 256 * 4, 1184 * 256 * 4 + 4, (1 << 22) + 60])
@pytest.mark.parametrize("alpha", [0.0, 0.01])
def test_bits_give_the_same_gradient(n, alpha):
    import torch
    from aether_ml_b200 import layers as L
    x, dy = _values(n, n), _values(n, n + 1)
    layer, plain = (L.Leaky_ReLU(alpha) if alpha else L.ReLU() for _ in range(2))
    layer.MASK_FROM = 1
    y, want = layer.forward(x, True), plain.forward(x, False)
    assert layer._mask is not None and plain._mask is None
    assert torch.equal(y.view(torch.int32), want.view(torch.int32))
    assert torch.equal(layer.backward(dy).view(torch.int32), plain.backward(dy).view(torch.int32))
    assert torch.equal(plain.dinputs.view(torch.int32), torch.where(x < 0, alpha * dy, dy).view(torch.int32))


def test_changed_inputs_are_read_again():
    import torch
    from aether_ml_b200 import layers as L
    layer = L.ReLU()
    layer.MASK_FROM = 1
    x, dy = torch.randn(512, device="cuda"), torch.randn(512, device="cuda")
    layer.forward(x, True)
    x.neg_()
    assert torch.equal(layer.backward(dy), torch.where(x < 0, torch.zeros_like(dy), dy))
    layer.forward(x, True)
    layer.inputs = other = torch.randn(512, device="cuda")
    assert torch.equal(layer.backward(dy), torch.where(other < 0, torch.zeros_like(dy), dy))
    layer.forward(x, True)
    layer.forward(other, False)                             # an inference pass keeps none
    assert layer._mask is None and torch.equal(layer.backward(dy), torch.where(other < 0, torch.zeros_like(dy), dy))


class Foreign:
    """An array of another library: torch learns its address, and of changes nothing."""

    def __init__(self, t):
        self.t = t
        self.__cuda_array_interface__ = dict(t.__cuda_array_interface__)


@pytest.mark.parametrize("wrapped", [False, True])
def test_changes_of_an_array_that_another_library_owns(wrapped):
    import torch
    from aether_ml_b200 import layers as L
    layer = L.Leaky_ReLU(0.25)
    layer.MASK_FROM = 1
    memory, dy = torch.randn(4096, device="cuda"), torch.randn(4096, device="cuda")
    x = Foreign(memory)
    layer.forward(torch.as_tensor(x, device="cuda") if wrapped else x, True)
    memory.neg_()                                           # the owner's kernel, behind torch's back
    assert torch.equal(layer.backward(dy), torch.where(memory < 0, 0.25 * dy, dy))


def test_inputs_of_inference_mode():
    import torch
    from aether_ml_b200 import layers as L
    layer = L.ReLU()
    layer.MASK_FROM = 1
    dy = torch.randn(4096, device="cuda")
    with torch.inference_mode():
        x = torch.randn(4096, device="cuda")
        y = layer.forward(x, True)
        assert torch.equal(y, x.clamp(min=0))
        x.neg_()
        assert torch.equal(layer.backward(dy), torch.where(x < 0, torch.zeros_like(dy), dy))
