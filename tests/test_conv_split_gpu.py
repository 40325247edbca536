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

# Pointwise layers that are large enough (rows of channels to the next 8 instead of whole tile rows), strided and not; a filter gradient of
# 162 tiles and 39 stages each, so that 14 CTAs have a second one and all a second epoch; a column tile of 128 with 50 stages.
MORE = [(6, 43, 43, 88, 188, 1, (1, 1), "same", "fp32"), (200, 23, 21, 300, 331, 1, (2, 1), "same", "bf16"), (50, 7, 7, 384, 384, 3, (1, 1), "same", "fp32"),
        (24, 28, 28, 128, 128, 5, (1, 1), "same", "fp32")]


def _split(shape):
    """Whether the library takes these kernels for the shape (then forward calls use a part of the workspace only)."""
    from aether_ml_b200 import _lib
    S, H, W, Cin, Cout, f, st, pad, mode = shape
    P = (f - 1) // 2 if pad == "same" else 0
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, *st, P, P, _lib.MATH_MODES[mode])
    return _lib.lib().aether_conv2d_fwd_workspace_bytes(d) < _lib.lib().aether_conv2d_workspace_bytes(d)


def _reference(shape, x, w, b, dy):
    """y, dX, dW and dB in float64 for arrays on the device."""
    import torch
    S, H, W, Cin, Cout, f, st, pad, mode = shape
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    y = torch.nn.functional.conv2d(xd.permute(0, 3, 1, 2), wd.permute(3, 2, 0, 1), stride=st, padding=(f - 1) // 2 if pad == "same" else 0).permute(0, 2, 3, 1)
    y.backward(dy.double())
    return y.detach() + b.double(), xd.grad, wd.grad, dy.double().sum((0, 1, 2))


def _off(got, want):
    return float((got.double() - want).norm() / want.norm())


def _random(shape, seed, scale=(1.0, 1.0, 1.0), positive=False):
    """A layer and x, dy for it, from N(0, 1) times `scale` of x, w and dy; all positive if asked for."""
    import torch
    from aether_ml_b200 import layers
    S, H, W, Cin, Cout, f, st, pad, mode = shape
    np.random.seed(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    layer = layers.Conv_Layer((H, W, Cin), Cout, (f, f), st, pad, math_mode=mode)
    make = lambda t, k: (t.abs() if positive else t) * k
    layer.filter_weights.copy_(make(layer.filter_weights, scale[1]))
    x = make(torch.randn((S, H, W, Cin), generator=g, device="cuda"), scale[0])
    _, Ho, Wo = layer._extent(H, W)
    dy = make(torch.randn((S, Ho, Wo, Cout), generator=g, device="cuda"), scale[2])
    return layer, x, dy


def _pass(layer, x, dy):
    y = layer.forward(x, True)
    return y, layer.backward(dy), layer.dweights, layer.dbiases


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


def test_routes():
    """What the other tests here are about is what runs (two pointwise shapes of the list are too small for it)."""
    assert [_split(s) for s in SHAPES] == [s[5] > 1 for s in SHAPES] and all(_split(s) for s in MORE)


@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("shape", MORE + [SHAPES[0], SHAPES[2], SHAPES[7]])
def test_large_and_one_sided(shape, positive):
    """Sums of one sign, too: those that the tensor cores truncate lose in one direction there.  A stage's sum is at most four truncations of 2^-24
    off, the at most 50 stages are added with rounding: below 54 * 2^-24 = 3.2e-6 at worst; measured 2.5e-7."""
    layer, x, dy = _random(shape, 3, positive=positive)
    for got, want in zip(_pass(layer, x, dy), _reference(shape, x, layer.filter_weights, layer.biases, dy)):
        assert _off(got, want) <= 3.2e-6


@pytest.mark.parametrize("scale", [(2.0**-118, 1.0, 1.0), (1.0, 2.0**-116, 1.0), (1.0, 1.0, 2.0**-121), (2.0**-124, 2.0**20, 2.0**-80), (2.0**90, 2.0**-60, 2.0**-90)])
@pytest.mark.parametrize("shape", [SHAPES[0], SHAPES[2]])
def test_small_operands(shape, scale):
    """Operands of which bf16 cannot hold the last bits, alone and beside others of ordinary size: 24 bits of each count.  (Outputs near the end of
    the range are rounded to 2^-149.)"""
    layer, x, dy = _random(shape, 4, scale)
    x[1], dy[1] = x[1] * 2.0**8, dy[1] * 2.0**8
    for got, want in zip(_pass(layer, x, dy), _reference(shape, x, layer.filter_weights, layer.biases, dy)):
        assert float((got.double() - want).norm()) <= 3e-6 * float(want.norm()) + 2.0**-149 * want.numel()**0.5


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


# strided layers of odd channel counts, with rows of 32 channels, without padding; several column tiles; 5x5 taps
@pytest.mark.parametrize("shape", [SHAPES[2], SHAPES[10], SHAPES[8], SHAPES[4], SHAPES[0], SHAPES[7]])
@pytest.mark.parametrize("where", ["x and dy", "filter", "sums", "overflow"])
def test_not_finite_anywhere(shape, where):
    """Infinite, NaN, very large operands and sums that overflow in x, the filter and dy, which reach some outputs: those are what
    fp32 sums are (padding is zeros: 0 * inf), the others are as exact as ever."""
    from aether_ml_b200 import _lib
    assert _split(shape)
    S, H, W, Cin, Cout, f, st, pad, mode = shape
    layer, x, dy = _random(shape, 5)
    w = layer.filter_weights
    if where == "x and dy":
        x[0, 3, 4, 5], x[1, 2, 2, 0], x[2, 5, 5, 1], x[3, 0, 0, 2] = float("inf"), -float("inf"), float("nan"), 3.4e38
        dy[1, 1, 1, 7], dy[5, 0, 1, 2] = float("inf"), float("nan")
        w *= 1e-3                                            # (3.4e38 stays in range, with dy, too)
        dy *= 1e-3
    elif where == "filter":
        w[0, 0, 3, 2], w[-1, -1, 6, 9], w[0, -1, 7, 4] = float("inf"), float("nan"), -float("inf")
    elif where == "sums":
        x *= 2.0**60                                         # sums of 2^95 and more, finite ones
        w *= 2.0**40
        dy *= 2.0**30
    else:
        w *= 2.0**10                                         # sums of 2^110, and some that overflow (of one sign: in any order)
        w[..., 3] = w[..., 3].abs() * 2.0**20
        x[0], dy[1] = x[0].abs() * 2.0**100, dy[1].abs() * 2.0**100
    got = [t.cpu().numpy() for t in _pass(layer, x, dy)]
    X, DY, Wt = (t.cpu().numpy().astype(np.float64) for t in (x, dy, w))
    with np.errstate(all="ignore"):
        want = [O.conv_forward(X, Wt, np.zeros(Cout), st, pad), *O.conv_backward(X, Wt, DY, st, pad)]
        want = [np.where(np.abs(t) > 3.5e38, np.sign(t) * np.inf, t) for t in want]
        X, DY, Wt = np.abs(X), np.abs(DY), np.abs(Wt)
        sizes = [O.conv_forward(X, Wt, np.zeros(Cout), st, pad), *O.conv_backward(X, Wt, DY, st, pad)]
        for a, b, size in zip(got, want, sizes):
            sure = ~(np.abs(b) > 3e38) | np.isinf(b)         # (in between the order of the sum decides)
            a, b, size = a[sure], b[sure], size[sure]
            assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b))
            fine = np.isfinite(b)
            assert (np.abs(a[fine] - b[fine]) <= 3e-6 * size[fine]).all()
    assert _lib.device_status() == 0


def test_time_of_values_that_are_not_finite():
    """A diverged network's arrays are NaN or infinite throughout.  Such a pass may take longer than one of finite values, but not by orders of
    magnitude: NaN ends a sum early, infinite ones of one sign go all the way."""
    import torch
    shape = (96, 28, 28, 32, 64, 3, (1, 1), "same", "fp32")
    times = []
    for value, positive in ((1.0, True), (float("nan"), False), (float("inf"), False), (float("inf"), True)):
        layer, x, dy = _random(shape, 6, positive=positive)
        x.mul_(value)
        dy.mul_(value)
        for _ in range(3):
            _pass(layer, x, dy)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            _pass(layer, x, dy)
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) / 5)
    assert max(times[1:3]) < 15 * times[0] and times[3] < 50 * times[0], times          # (measured 6 and 23 times)


def test_less_memory(monkeypatch):
    """Inference asks for the part of the workspace that forward calls use; without the memory for a workspace the layer runs as it can."""
    import torch
    from aether_ml_b200 import layers
    shape = SHAPES[2]
    layer, x, dy = _random(shape, 8)
    p = layer._plan(tuple(x.shape))
    want = _reference(shape, x, layer.filter_weights, layer.biases, dy)
    y = layer.forward(x, False)
    assert layer._ws.size == p.fwd_ws_bytes < p.ws_bytes and _off(y, want[0]) <= 3e-6
    grads = layer.backward(dy), layer.dweights, layer.dbiases
    assert layer._ws.size == p.ws_bytes
    again = _pass(layer, x, dy)
    assert all(torch.equal(a, b) for a, b in zip((y, *grads), again))

    def no_room(self, nbytes):
        if nbytes > p.least_ws_bytes():
            raise torch.OutOfMemoryError("no room")
        return grow(self, nbytes)
    grow = layers._Workspace._grow
    monkeypatch.setattr(layers._Workspace, "_grow", no_room)
    small, _, _ = _random(shape, 8)
    for got, w in zip(_pass(small, x, dy), want):
        assert _off(got, w) <= 3e-6
    assert small._ws.size == p.least_ws_bytes() < p.fwd_ws_bytes


def test_outputs_come_before_scratch():
    """A process that may take 700 MiB more: a layer's outputs (2 x 196) fit beside the least workspace, not beside the 592 it would rather have."""
    import torch
    from aether_ml_b200 import layers
    np.random.seed(1)
    layer = layers.Conv_Layer((112, 112, 64), 64, (3, 3), (1, 1), "same", math_mode="fp32")
    x = torch.randn((64, 112, 112, 64), device="cuda")
    dy = torch.randn(x.shape, device="cuda")
    p = layer._plan(tuple(x.shape))
    assert p.least_ws_bytes() < 200 << 20 < p.fwd_ws_bytes < 500 << 20 < p.ws_bytes
    torch.cuda.empty_cache()
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (700 << 20)) / torch.cuda.get_device_properties(0).total_memory)
        y = layer.forward(x, True)
        dx = layer.backward(dy)
        assert layer._ws.size == p.least_ws_bytes()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    rich, _, _ = _random((64, 112, 112, 64, 64, 3, (1, 1), "same", "fp32"), 1)
    rich.filter_weights.copy_(layer.filter_weights)
    for a, b in zip((y, dx, layer.dweights), _pass(rich, x, dy)):
        assert _off(a, b.double()) <= 3e-6
    assert rich._ws.size == p.ws_bytes
    del rich, x, dy, y, dx
    torch.cuda.empty_cache()
