"""bf16 convolutions of at most 32 input channels on rows of 32 channels: one and two steps of 16, the last of them partial, more
and fewer taps than a stage holds, column tiles of 32 to 128, images that share a tile; the statistics of the epilogue.  bf16
operands: relative L2 <= 1e-2, as the other tests of that mode have it."""
import numpy as np
import pytest

from oracle import aether_oracle as O

pytestmark = pytest.mark.gpu

# (S, H, W, Cin, Cout, f, pad)
SHAPES = [(9, 8, 8, 32, 64, 3, "same"), (5, 7, 9, 16, 32, 5, "same"), (40, 16, 16, 20, 128, 3, "same"), (3, 11, 6, 28, 36, 3, "valid"), (70, 6, 5, 32, 96, 1, "same")]


@pytest.mark.parametrize("shape", SHAPES)
def test_against_oracle(shape):
    from aether_ml_b200 import layers
    S, H, W, Cin, Cout, f, pad = shape
    rng = np.random.default_rng(S)
    x = rng.standard_normal((S, H, W, Cin)).astype(np.float32)
    conv = layers.Conv_Layer((H, W, Cin), Cout, (f, f), (1, 1), pad, math_mode="bf16")
    w = conv.filter_weights.cpu().numpy()
    b = rng.standard_normal(Cout).astype(np.float32)
    conv.set_parameters(w, b)
    y = conv.forward(x, True).cpu().numpy()
    dy = rng.standard_normal(y.shape).astype(np.float32)
    dx = conv.backward(dy).cpu().numpy()
    dxo, dwo, dbo = O.conv_backward(x, w, dy, (1, 1), pad)
    for got, want in ((y, O.conv_forward(x, w, b, (1, 1), pad)), (dx, dxo), (conv.dweights.cpu().numpy(), dwo), (conv.dbiases.cpu().numpy(), dbo)):
        assert O.rel_l2(got, want) <= 1e-2
    # the statistics that go with the output describe that output
    conv.emit_bn_stats = True
    y2 = conv.forward(x, True)
    mean, var = y.reshape(-1, Cout).mean(0), y.reshape(-1, Cout).var(0)
    assert (conv.bn_partials is not None) == (conv._plan(tuple(x.shape)).stats_blocks > 0)
    if conv.bn_partials is not None:
        stats, blocks, _ = conv.bn_partials
        p = stats.view(dtype=__import__("torch").float32)[:blocks * 3 * Cout].cpu().numpy().reshape(blocks, 3, Cout).astype(np.float64)
        n = p[:, 0].sum(0)
        m = (p[:, 0] * p[:, 1]).sum(0) / n
        v = (p[:, 2] + p[:, 0] * p[:, 1] ** 2).sum(0) / n - m * m
        assert np.allclose(m, mean, atol=1e-4) and np.allclose(v, var, rtol=1e-3)
    assert np.array_equal(y2.cpu().numpy(), y)
