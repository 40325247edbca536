"""Single-precision convolutions on the tensor cores (operands as sums of three bf16 numbers) at the sizes where their tiles end:
channel counts around the 64-channel rows and the 16-column tiles, no multiples of 4, strides whose pixel phases and classes
differ in size or see no tap, tiles that span images.  The bound is that of the FMA kernels they replace: an fp32 sum of K
products in any order is within K * 2^-24 of the exact one relative to the sum of magnitudes, for random signs within
sqrt(K) * 2^-24 of the result: 3e-6 for the longest reduction here (K = 2304 taps times channels); measured 3e-7."""
import numpy as np
import pytest

from oracle import aether_oracle as O

pytestmark = pytest.mark.gpu

# (S, H, W, Cin, Cout, f, stride, pad, mode)
SHAPES = [(9, 19, 17, 65, 130, 3, (1, 1), "same", "fp32"), (60, 15, 13, 37, 71, 3, (1, 1), "valid", "bf16"), (40, 21, 18, 72, 48, 3, (2, 2), "same", "bf16"),
          (61, 8, 8, 128, 33, 3, (1, 1), "same", "fp32"), (30, 23, 20, 64, 64, 5, (3, 2), "valid", "tf32"), (70, 30, 31, 96, 32, 1, (1, 1), "same", "fp32"),
          (120, 12, 11, 100, 129, 1, (2, 2), "same", "fp32"), (60, 20, 21, 16, 50, 5, (1, 1), "same", "fp32"), (40, 33, 20, 90, 17, 3, (2, 1), "valid", "bf16"), (16, 7, 7, 256, 256, 3, (1, 1), "same", "fp32"), (90, 9, 10, 32, 144, 3, (1, 4), "same", "tf32")]


def _layer(shape, x, b):
    from aether_ml_b200 import layers
    S, H, W, Cin, Cout, f, st, pad, mode = shape
    layer = layers.Conv_Layer((H, W, Cin), Cout, (f, f), st, pad, math_mode=mode)
    w = layer.filter_weights.cpu().numpy()
    layer.set_parameters(w, b)
    return layer, w


@pytest.mark.parametrize("shape", SHAPES)
def test_against_float64(shape):
    S, H, W, Cin, Cout, f, st, pad, mode = shape
    rng = np.random.default_rng(S + Cin)
    x = rng.standard_normal((S, H, W, Cin)).astype(np.float32)
    b = rng.standard_normal(Cout).astype(np.float32)
    layer, w = _layer(shape, x, b)
    y = layer.forward(x, True)
    dy = rng.standard_normal(tuple(y.shape)).astype(np.float32)
    dx = layer.backward(dy)
    yo = O.conv_forward(x.astype(np.float64), w.astype(np.float64), b, st, pad)
    dxo, dwo, dbo = O.conv_backward(x.astype(np.float64), w.astype(np.float64), dy.astype(np.float64), st, pad)
    for got, want in ((y, yo), (dx, dxo), (layer.dweights, dwo), (layer.dbiases, dbo)):
        assert O.rel_l2(got.cpu().numpy(), want) <= 3e-6


def test_values_without_remainders():
    """Infinite, NaN and very large operands: their parts are not numbers, the outputs are those of fp32 sums."""
    shape = SHAPES[1]
    S, H, W, Cin, Cout, f, st, pad, mode = shape
    rng = np.random.default_rng(5)
    x = rng.standard_normal((S, H, W, Cin)).astype(np.float32)
    x[0, 3, 4, 5], x[1, 2, 2, 0], x[2, 7, 7, 36], x[3, 0, 0, 1] = np.inf, -np.inf, np.nan, np.float32(3.4e38)
    b = rng.standard_normal(Cout).astype(np.float32)
    layer, w = _layer(shape, x, b)
    w *= np.float32(1e-3)                                    # (3.4e38 stays in range)
    w[0, 0, 5, 3] = 0.0                                      # 0 * inf
    layer.set_parameters(w, b)
    y = layer.forward(x, True)
    dy = rng.standard_normal(tuple(y.shape)).astype(np.float32) * np.float32(1e-3)       # (nor does its product with dy overflow)
    dy[4, 1, 1, 7] = np.inf
    dx = layer.backward(dy)
    with np.errstate(all="ignore"):
        yo = O.conv_forward(x.astype(np.float64), w.astype(np.float64), b, st, pad)
        dxo, dwo, dbo = O.conv_backward(x.astype(np.float64), w.astype(np.float64), dy.astype(np.float64), st, pad)
    for got, want in ((y, yo), (dx, dxo), (layer.dweights, dwo), (layer.dbiases, dbo)):
        got = got.cpu().numpy()
        assert (np.isnan(got) == np.isnan(want)).all() and (np.isposinf(got) == np.isposinf(want)).all() and (np.isneginf(got) == np.isneginf(want)).all()
        small = np.isfinite(want) & (np.abs(want) < 1e30)
        big = np.isfinite(want) & ~small
        assert O.rel_l2(got[small], want[small]) <= 3e-6
        assert np.allclose(got[big].astype(np.float64), want[big].astype(np.float64), rtol=3e-6)
