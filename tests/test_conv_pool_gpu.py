"""Inference of a convolution with the Batch_Norm, activation and 2x2 max pooling behind it in one launch, against the convolution and the pass over its
output: where both run the same kernel on the same tiles' order of sums the bits are the same, else the convolutions' outputs differ in the order of fp32
sums of n products, 2 * n * 2^-23 of the sum of absolute values, which the affine map scales and the maximum passes on."""
import numpy as np
import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu

# (S, H, W, Cin, Cout, f, pad): first layers (tap tables and not, channels to the next 32, several chunks) and per-tap shapes (boxes of 8 and 16 columns, cut
# off at the image, several images, narrow rows, wide and overhanging column tiles); first layers of so many channels that only two or three accumulators are there
# for a CTA's tiles, of which it takes five and more, and ones with as many tiles of four accumulators
SHAPES = [(5, 32, 32, 3, 32, 3, 1), (3, 28, 28, 1, 64, 3, 1), (2, 10, 12, 3, 20, 3, 1), (2, 9, 11, 4, 128, 2, 0), (1, 6, 6, 1, 256, 7, 1), (300, 32, 32, 3, 96, 3, 1),
          (7, 16, 16, 32, 64, 3, 1), (9, 8, 8, 64, 128, 3, 1), (3, 14, 14, 32, 64, 3, 1), (2, 20, 24, 64, 40, 3, 1), (5, 4, 6, 16, 192, 3, 1), (200, 8, 8, 128, 256, 3, 1),
          (11, 2, 2, 68, 100, 1, 0), (3, 18, 34, 96, 160, 5, 2), (90, 16, 16, 64, 128, 3, 1),
          (100, 32, 32, 3, 160, 3, 1), (100, 32, 32, 3, 192, 3, 1), (200, 28, 28, 1, 256, 3, 1), (130, 30, 30, 4, 132, 3, 1), (120, 32, 32, 2, 200, 5, 2), (110, 32, 32, 3, 128, 3, 1)]


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,pad", SHAPES)
@pytest.mark.parametrize("alpha", [0.0, 0.1])
def test_one_launch_against_two(S, H, W, Cin, Cout, f, pad, alpha):
    import torch
    lib = _lib.lib()
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, 1, 1, pad, pad, _lib.MATH_MODES["bf16"])
    assert lib.aether_conv2d_pool_supported(d)
    Ho, Wo = H + 2 * pad - f + 1, W + 2 * pad - f + 1
    g = torch.Generator(device="cuda").manual_seed(S + Cout)
    R = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    bf = lambda t: t.bfloat16().float()                      # representable: the copies round nothing
    x, w, b = bf(R(S, H, W, Cin)), bf(R(f, f, Cin, Cout)), R(Cout)
    gamma, beta, mean, var = R(Cout), R(Cout), R(Cout), R(Cout).abs() + 0.1
    n = max(lib.aether_conv2d_workspace_bytes(d), 16)
    ws, ws2 = (torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(2))
    bws = torch.empty(lib.aether_bn_workspace_bytes(S * Ho * Wo, Cout), dtype=torch.uint8, device="cuda")
    ld = (Cout + 63) // 64 * 64
    y = torch.empty((S, Ho, Wo, Cout), device="cuda")
    pooled, one = (torch.full((S, Ho // 2, Wo // 2, Cout), float("nan"), device="cuda") for _ in range(2))
    copy, copy_one = (torch.full((S * (Ho // 2) * (Wo // 2) + 1, ld), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    P, st = (lambda t: t.data_ptr()), torch.cuda.current_stream().cuda_stream
    assert lib.aether_conv2d_fwd(d, P(x), P(w), P(b), P(y), P(ws), n, st) == 0
    assert lib.aether_chain_fwd(P(y), None, 0, P(gamma), P(beta), P(mean), P(var), None, None, None, None, None, P(pooled), None, S, Ho, Wo, Cout, 2, 2, 1e-5, 0.9,
                                alpha, None, 0, P(copy), ld, P(bws), bws.numel(), st) == 0
    for _ in range(2):
        assert lib.aether_conv2d_pool_fwd(d, P(x), P(w), P(b), P(gamma), P(beta), P(mean), P(var), 1e-5, alpha, P(one), P(copy_one), ld, P(ws2), n, 0, st) == 0
    again = torch.full_like(one, float("nan"))
    assert lib.aether_conv2d_pool_fwd(d, P(x), P(w), P(b), P(gamma), P(beta), P(mean), P(var), 1e-5, alpha, P(again), None, 0, P(ws2), n, 0, st) == 0
    assert torch.equal(one, again)
    if Cin <= 4:
        assert torch.equal(one, pooled) and torch.equal(copy_one, copy)
    size = torch.nn.functional.conv2d(x.double().abs().permute(0, 3, 1, 2), w.double().abs().permute(3, 2, 0, 1), padding=pad).permute(0, 2, 3, 1)
    worst = torch.nn.functional.max_pool2d(size.permute(0, 3, 1, 2), 2).permute(0, 2, 3, 1) * (gamma / torch.sqrt(var + 1e-5)).abs()
    assert bool(((one.double() - pooled.double()).abs() <= 2 * f * f * Cin * 2.0**-23 * worst + 1e-6 * pooled.double().abs()).all())
    rows = copy_one[:-1].reshape(S, Ho // 2, Wo // 2, ld)
    assert torch.equal(rows[..., :Cout], one.bfloat16()) and bool((rows[..., Cout:] == 0).all())
    assert bool((copy_one[-1] == 7).all())                   # nothing behind the last window
    assert _lib.device_status() == 0


@pytest.mark.parametrize("S,H,W,Cin,Cout", [(9, 12, 14, 3, 32), (40, 16, 16, 1, 192), (20, 16, 16, 32, 64), (9, 10, 10, 64, 132)])
def test_values_that_are_not_finite(S, H, W, Cin, Cout):
    """Infinities and NaN in the images and in the filter: in the same places as from the convolution and the pass behind it, with the signs."""
    import torch
    lib = _lib.lib()
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, 3, 3, 1, 1, 1, 1, _lib.MATH_MODES["bf16"])
    g = torch.Generator(device="cuda").manual_seed(Cout)
    R = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    x, w, b, gamma, beta, mean, var = R(S, H, W, Cin), R(3, 3, Cin, Cout), R(Cout), R(Cout), R(Cout), R(Cout), R(Cout).abs() + 0.1
    x[0, 2, 3, 0], x[1, H - 1, W - 1, Cin - 1], x[2, 0, 0, 0], x[S - 1, 5, 6, 0] = float("inf"), -float("inf"), float("nan"), float("inf")
    w[1, 1, 0, Cout - 1], w[0, 2, Cin - 1, 1] = float("inf"), float("nan")
    n = max(lib.aether_conv2d_workspace_bytes(d), 16)
    ws, ws2 = (torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(2))
    bws = torch.empty(lib.aether_bn_workspace_bytes(S * H * W, Cout), dtype=torch.uint8, device="cuda")
    y, two, one = torch.empty((S, H, W, Cout), device="cuda"), torch.empty((S, H // 2, W // 2, Cout), device="cuda"), torch.empty((S, H // 2, W // 2, Cout), device="cuda")
    P, st = (lambda t: t.data_ptr()), torch.cuda.current_stream().cuda_stream
    assert lib.aether_conv2d_fwd(d, P(x), P(w), P(b), P(y), P(ws), n, st) == 0
    assert lib.aether_chain_fwd(P(y), None, 0, P(gamma), P(beta), P(mean), P(var), None, None, None, None, None, P(two), None, S, H, W, Cout, 2, 2, 1e-5, 0.9, 0.1, None, 0, None, 0, P(bws),
                                bws.numel(), st) == 0
    assert lib.aether_conv2d_pool_fwd(d, P(x), P(w), P(b), P(gamma), P(beta), P(mean), P(var), 1e-5, 0.1, P(one), None, 0, P(ws2), n, 0, st) == 0
    assert bool(two.isnan().any()) and bool(two.isinf().any()) and bool(two[3, :, :, 2:Cout - 1].isfinite().all())
    finite = two.isfinite()
    assert torch.equal(one.isnan(), two.isnan()) and torch.equal(one.nan_to_num(0.0)[~finite], two.nan_to_num(0.0)[~finite])
    assert float((one - two)[finite].norm() / two[finite].norm()) <= 9 * Cin * 2.0**-23
    assert _lib.device_status() == 0


def test_refused_where_the_epilogue_does_not_fit():
    lib = _lib.lib()
    for S, H, W, Cin, Cout, f, s, pad, mode in [(2, 7, 8, 64, 64, 3, 1, 1, "bf16"), (2, 8, 7, 3, 32, 3, 1, 1, "bf16"), (2, 8, 8, 64, 64, 3, 1, 1, "tf32"), (2, 8, 8, 64, 64, 3, 2, 1, "bf16"), (2, 8, 8, 64, 1028, 1, 1, 0, "bf16")]:
        d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, s, s, pad, pad, _lib.MATH_MODES[mode])
        assert not lib.aether_conv2d_pool_supported(d)


def test_taken_where_it_is_faster():
    """Boxes of windows fill little of 10- and 18-pixel rows; what a whole prediction runs follows from it."""
    lib = _lib.lib()
    for S, H, W, Cin, Cout, f, mode, want in [(896, 16, 16, 32, 64, 3, "bf16", 1), (512, 8, 8, 256, 512, 3, "bf16", 1), (300, 14, 14, 32, 64, 3, "bf16", 1), (900, 32, 32, 3, 192, 3, "bf16", 1), (900, 18, 18, 16, 16, 3, "bf16", 0),
                                              (900, 10, 10, 512, 1024, 3, "bf16", 0), (128, 10, 10, 256, 256, 3, "bf16", 0), (900, 4, 4, 256, 256, 3, "bf16", 0), (896, 16, 16, 32, 64, 3, "tf32", 0), (9, 7, 8, 64, 64, 3, "bf16", 0)]:
        d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, 1, 1, f // 2, f // 2, _lib.MATH_MODES[mode])
        assert lib.aether_conv2d_pool_faster(d) == want, (S, H, W, Cin, Cout)


@pytest.mark.parametrize("hw,channels,batch,images", [(32, (32, 64, 128), 128, 1000), (28, (32, 64), 50, 230), (12, (20, 48), 16, 90), (32, (192, 32), 64, 400), (20, (32, 64, 32), 60, 900)])
def test_predictions_are_those_of_single_batches(hw, channels, batch, images):
    """Several batches in one pass (convolutions go on to their pooled outputs) and batch by batch with every layer's arrays."""
    import torch
    from aether_ml_b200 import layers as L
    from aether_ml_b200.model import Accuracy_Categorical, Model
    np.random.seed(1)
    m, c, n = Model(), 3, hw
    for k in channels:
        for l in (L.Conv_Layer((n, n, c), k, (3, 3), (1, 1), "same"), L.Batch_Norm(n_features=k), L.Leaky_ReLU(0.1), L.Layer_Dropout_Spatial(0.2), L.Pooling((2, 2), (2, 2), "valid", "max")):
            m.add(l)
        c, n = k, n // 2
    for l in (L.Flatten(), L.Layer_Dense(n * n * c, 64), L.ReLU(), L.Layer_Dense(64, 10), L.SoftMax()):
        m.add(l)
    m.set(loss=L.Loss_CategoricalCrossEntropy(), optimizer=L.Optimizer_Adam(), accuracy=Accuracy_Categorical())
    m.finalize()
    g = torch.Generator(device="cuda").manual_seed(3)
    for l in m.layers:
        if isinstance(l, L.Batch_Norm):
            l.set_parameters(torch.rand(l.gamma.numel(), generator=g, device="cuda") + 0.5, torch.randn(l.gamma.numel(), generator=g, device="cuda") * 0.1,
                             torch.randn(l.gamma.numel(), generator=g, device="cuda") * 0.1, torch.rand(l.gamma.numel(), generator=g, device="cuda") + 0.2)
    X = torch.rand((images, hw, hw, 3), generator=g, device="cuda")
    single = torch.vstack([m.forward(X[k:k + batch], training=False).clone() for k in range(0, images, batch)])
    n0 = _lib.launch_count()
    joined = m.predict(X, batch_size=batch)
    launches = _lib.launch_count() - n0
    # bf16 operands of the layers behind round what differs in the last bit of the ones in front: 2^-9 of a value, through two or three layers
    assert float((joined.double() - single.double()).norm() / single.double().norm()) <= 5e-3
    conv = m.layers[0]
    assert conv.output.shape[0] == images - (images - 1) // batch * batch and torch.equal(conv.inputs, X[(images - 1) // batch * batch:])
    original = L.Conv_Layer.forward
    try:                                                     # a convolution of the caller's own runs by itself
        conv.forward = lambda inputs, training: original(conv, inputs, training)
        n0 = _lib.launch_count()
        again = m.predict(X, batch_size=batch)
        assert _lib.launch_count() - n0 > launches
    finally:
        del conv.forward
    assert float((again.double() - joined.double()).norm() / joined.double().norm()) <= 5e-3
    assert _lib.device_status() == 0
