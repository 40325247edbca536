"""The tiled fp32 convolution kernels at the sizes where their tiles end: channel counts around the column tiles (16, 32,
64, 128) and the row tiles of the filter gradient, scalar and 16-byte loads, strides whose pixel classes differ in size or
see no tap at all, enough pixels for the 128-row tiles.  fp32 sums: relative L2 <= 1e-5 against the float64 oracle."""
import numpy as np
import pytest

from oracle import aether_oracle as O

pytestmark = pytest.mark.gpu

# (S, H, W, Cin, Cout, f, stride, pad)
SHAPES = [(3, 13, 11, 16, 17, 3, (2, 2), "same"), (2, 12, 15, 33, 31, 3, (3, 2), "valid"), (2, 9, 10, 65, 130, 3, (1, 2), "same"),
          (4, 10, 10, 20, 36, 1, (2, 2), "same"), (2, 11, 9, 128, 64, 5, (2, 3), "same"), (1, 5, 5, 129, 127, 3, (4, 4), "same"),
          (50, 33, 31, 16, 32, 3, (1, 1), "same"), (50, 33, 31, 12, 15, 3, (2, 1), "same"), (40, 32, 33, 8, 128, 3, (1, 1), "valid"),
          (44, 30, 31, 4, 64, 1, (1, 1), "same"), (1, 1, 1, 300, 90, 1, (1, 1), "valid"), (7, 6, 6, 3, 5, 5, (3, 3), "valid")]


@pytest.mark.parametrize("shape", SHAPES)
def test_tile_edges(shape):
    import torch
    from aether_ml_b200 import layers
    S, H, W, Cin, Cout, f, st, pad = shape
    rng = np.random.default_rng(S + 7 * Cin)
    x = rng.standard_normal((S, H, W, Cin)).astype(np.float32)
    layer = layers.Conv_Layer((H, W, Cin), Cout, (f, f), st, pad, math_mode="fp32")
    w = layer.filter_weights.cpu().numpy()
    b = rng.standard_normal(Cout).astype(np.float32)
    layer.set_parameters(w, b)
    y = layer.forward(x, True)
    dy = rng.standard_normal(tuple(y.shape)).astype(np.float32)
    dx = layer.backward(dy)
    torch.cuda.synchronize()
    yo = O.conv_forward(x.astype(np.float64), w.astype(np.float64), b, st, pad)
    dxo, dwo, dbo = O.conv_backward(x.astype(np.float64), w.astype(np.float64), dy.astype(np.float64), st, pad)
    for got, want in ((y, yo), (dx, dxo), (layer.dweights, dwo), (layer.dbiases, dbo)):
        assert O.rel_l2(got.cpu().numpy(), want) <= 1e-5


# Reductions cut into pieces: all tiles of a small layer, the tiles behind the full rounds of a larger one (whole rows of tiles:
# 56 and 20 of 500 + 20), scalar and 16-byte rows, the classes of a strided layer's dX, pieces of unequal length.
SPLIT = [(3, 9, 8, 130, 77, 3, (1, 1), "same"), (2, 7, 9, 256, 64, 3, (1, 1), "valid"), (5, 11, 10, 96, 52, 3, (2, 2), "same"),
         (40, 40, 40, 64, 48, 3, (1, 1), "same"), (4, 8, 8, 200, 33, 5, (1, 1), "same"), (1, 6, 5, 260, 24, 1, (1, 1), "valid")]


@pytest.mark.parametrize("shape", SPLIT)
def test_split_reductions(shape):
    test_tile_edges(shape)
