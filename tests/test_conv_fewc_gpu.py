"""dX of layers with one to four input channels: filter rows in one pass (3 and 5) and one by one, strides whose pixel
classes see no tap, image heights around the strips of four rows, output channels around the eight lanes' 32, rows of dy
that are no multiple of 16 bytes.  fp32 sums: relative L2 <= 1e-5 against the float64 oracle."""
import numpy as np
import pytest

from oracle import aether_oracle as O

pytestmark = pytest.mark.gpu

# (S, H, W, Cin, Cout, f, stride, pad)
SHAPES = [(2, 7, 9, 1, 16, 3, (1, 1), "same"), (3, 8, 5, 2, 36, 3, (1, 1), "valid"), (2, 9, 33, 3, 32, 3, (1, 1), "same"),
          (1, 5, 5, 4, 260, 5, (1, 1), "same"), (2, 12, 6, 3, 33, 5, (1, 1), "valid"), (5, 4, 4, 3, 31, 3, (1, 1), "same"),
          (1, 1, 1, 3, 8, 1, (1, 1), "same"), (2, 11, 13, 3, 20, 3, (2, 2), "same"), (2, 11, 13, 2, 7, 3, (4, 3), "same"),
          (2, 9, 9, 1, 24, 2, (1, 1), "valid"), (1, 15, 14, 4, 12, 7, (2, 1), "same")]


@pytest.mark.parametrize("shape", SHAPES)
def test_dx_of_first_layers(shape):
    import torch
    from aether_ml_b200 import layers
    S, H, W, Cin, Cout, f, st, pad = shape
    rng = np.random.default_rng(S + 7 * Cout)
    x = rng.standard_normal((S, H, W, Cin)).astype(np.float32)
    layer = layers.Conv_Layer((H, W, Cin), Cout, (f, f), st, pad, math_mode="fp32")
    w = layer.filter_weights.cpu().numpy()
    y = layer.forward(x, True)
    dy = rng.standard_normal(tuple(y.shape)).astype(np.float32)
    dx = layer.backward(dy)
    torch.cuda.synchronize()
    want, _, _ = O.conv_backward(x.astype(np.float64), w.astype(np.float64), dy.astype(np.float64), st, pad)
    assert O.rel_l2(dx.cpu().numpy(), want) <= 1e-5


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,st", [(3, 9, 11, 3, 32, (3, 1), (1, 1)), (2, 13, 12, 1, 36, (3, 5), (1, 1)), (2, 11, 10, 4, 33, (5, 3), (1, 1)), (4, 10, 21, 2, 16, (3, 3), (1, 2)),
                                                 (1, 17, 9, 3, 260, (5, 5), (1, 3)), (2, 8, 15, 1, 7, (5, 2), (1, 1)), (2, 9, 9, 3, 24, (3, 3), (2, 1)), (3, 28, 28, 1, 1, (3, 3), (1, 1))])
def test_dx_of_filters_that_are_not_square(S, H, W, Cin, Cout, f, st):
    """Filters of three and five rows at row stride 1, whatever their width and the columns' stride: their rows in one pass."""
    import torch
    from aether_ml_b200 import layers
    rng = np.random.default_rng(S + 7 * Cout)
    x = rng.standard_normal((S, H, W, Cin)).astype(np.float32)
    layer = layers.Conv_Layer((H, W, Cin), Cout, f, st, "valid", math_mode="fp32")
    y = layer.forward(x, True)
    dy = rng.standard_normal(tuple(y.shape)).astype(np.float32)
    dx = layer.backward(dy)
    torch.cuda.synchronize()
    want, _, _ = O.conv_backward(x.astype(np.float64), layer.filter_weights.cpu().numpy().astype(np.float64), dy.astype(np.float64), st, "valid")
    assert O.rel_l2(dx.cpu().numpy(), want) <= 1e-5
