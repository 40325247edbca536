"""The tiled fp32 convolution kernels where 32-bit quantities end: more pixel classes of a strided dX than a grid takes along one
axis, and tiles whose samples lie more than 2^31 pixels apart.  fp32 sums: relative L2 <= 1e-5 against float64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,st", [(2, 301, 262, 5, 6, 3, (300, 260)), (3, 300, 520, 2, 16, 3, (299, 259)), (1, 270, 300, 8, 4, 5, (256, 257))])
def test_many_pixel_classes(S, H, W, Cin, Cout, f, st):
    import torch
    from aether_ml_b200 import layers
    np.random.seed(1)
    g = torch.Generator(device="cuda").manual_seed(2)
    layer = layers.Conv_Layer((H, W, Cin), Cout, (f, f), st, "same", math_mode="fp32")
    x = torch.randn((S, H, W, Cin), generator=g, device="cuda")
    y = layer.forward(x, True)
    dy = torch.randn(y.shape, generator=g, device="cuda")
    dx = layer.backward(dy)
    xd, wd = x.double().requires_grad_(), layer.filter_weights.double().requires_grad_()
    p = (f - 1) // 2
    want = torch.nn.functional.conv2d(xd.permute(0, 3, 1, 2), wd.permute(3, 2, 0, 1), stride=st, padding=p).permute(0, 2, 3, 1)
    want.backward(dy.double())
    assert st[0] * st[1] > 65535
    for a, b in ((y, want.detach()), (dx, xd.grad), (layer.dweights, wd.grad)):
        assert a.shape == b.shape and float((a.double() - b).norm() / b.norm()) <= 1e-5


def test_samples_far_apart():
    """128 samples of 4130 x 4130 pixels in one tile, one output pixel each: the last begins 2.17e9 pixels behind the first."""
    import torch
    from aether_ml_b200 import layers
    np.random.seed(1)
    S, n, f = 128, 4130, 9
    if torch.cuda.mem_get_info()[0] < 20 << 30:
        pytest.skip("needs 9 GB of inputs")
    layer = layers.Conv_Layer((n, n, 1), 4, (f, f), (n, n), "valid", math_mode="fp32")
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.full((S, n, n, 1), float("nan"), device="cuda")            # (nothing but the windows is read)
    x[:, :f, :f] = torch.randn((S, f, f, 1), generator=g, device="cuda")
    y = layer.forward(x, True)
    dy = torch.randn(y.shape, generator=g, device="cuda")
    layer.backward(dy, need_dinputs=False)
    cols, w, gd = x[:, :f, :f].double().reshape(S, f * f), layer.filter_weights.double().reshape(f * f, 4), dy.double().reshape(S, 4)
    for a, b in ((y, cols @ w), (layer.dweights, cols.T @ gd), (layer.dbiases, gd.sum(0))):
        assert float((a.double().reshape(b.shape) - b).norm() / b.norm()) <= 1e-5
    del x, layer
    torch.cuda.empty_cache()
