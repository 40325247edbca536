"""First layers in single precision, forward and filter gradient: rows in one and several pieces, pieces of fewer pixels than the filter is wide, more pieces than
the GPU takes at once, channel counts of whole and of ragged groups of four, all numbers of input channels (filter rows together and by themselves),
paddings other than "same", a row stride.  Forward: sums of K products and the bias, within K + 2 roundings of 2^-24 of the sum of absolute values; dW
and dB: sums over P pixels in any order, within P roundings, of which a tree of partial sums of at most 4096 makes 4096."""
import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu

# (S, H, W, Cin, Cout, f, sH, padH, padW)
SHAPES = [(128, 32, 32, 3, 32, 3, 1, 1, 1), (7, 13, 11, 3, 20, 3, 1, 0, 0), (40, 9, 70, 1, 16, 3, 1, 1, 1), (3, 30, 31, 1, 208, 3, 1, 1, 1), (90, 28, 28, 2, 50, 3, 1, 1, 1),
          (5, 17, 19, 4, 33, 3, 2, 1, 1), (20, 24, 29, 1, 80, 5, 1, 2, 2), (6, 21, 23, 3, 28, 5, 1, 0, 0), (4, 15, 18, 2, 37, 5, 1, 4, 3), (3, 12, 40, 4, 17, 5, 3, 2, 2),
          (200, 7, 7, 3, 64, 5, 1, 0, 0), (1, 3, 3, 3, 4, 3, 1, 0, 0), (2, 5, 6, 1, 1, 5, 1, 2, 2), (300, 20, 20, 3, 3, 3, 1, 2, 0), (2, 64, 64, 3, 256, 3, 1, 1, 1),
          # (the filter gradient goes the other way)
          (30, 16, 18, 4, 256, 5, 1, 2, 2), (40, 20, 21, 2, 54, 5, 1, 2, 2), (30, 28, 28, 4, 128, 5, 1, 2, 2)]


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,sH,ph,pw", SHAPES)
def test_first_layers_in_single_precision(S, H, W, Cin, Cout, f, sH, ph, pw):
    import torch
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(S + Cout)
    Ho, Wo = (H + 2 * ph - f) // sH + 1, W + 2 * pw - f + 1
    new = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    x, w, b, dy = new(S, H, W, Cin), new(f, f, Cin, Cout), new(Cout), new(S, Ho, Wo, Cout)
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, sH, 1, ph, pw, _lib.MATH_MODES["fp32"])
    n = lib.aether_conv2d_workspace_bytes(d)
    ws = torch.empty(n + 16, dtype=torch.uint8, device="cuda")
    y, dw, db = (torch.full(t.shape, float("nan"), device="cuda") for t in (dy, w, b))
    stream = torch.cuda.current_stream().cuda_stream

    def both(x, w, b, dy):
        xd, wd = x.double().permute(0, 3, 1, 2), w.double().permute(3, 2, 0, 1).contiguous().requires_grad_(True)
        out = torch.nn.functional.conv2d(xd, wd, b.double(), stride=(sH, 1), padding=(ph, pw))
        out.backward(dy.double().permute(0, 3, 1, 2))
        return out.detach().permute(0, 2, 3, 1), wd.grad.permute(2, 3, 1, 0), dy.double().sum((0, 1, 2))

    for _ in range(2):
        assert lib.aether_conv2d_fwd(d, x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), ws.data_ptr(), n, stream) == 0
        assert lib.aether_conv2d_bwd(d, x.data_ptr(), dy.data_ptr(), w.data_ptr(), None, dw.data_ptr(), db.data_ptr(), ws.data_ptr(), n, 0, stream) == 0
        rounds = (f * f * Cin + 2, min(S * Ho * Wo, 4096) + 12, min(S * Ho * Wo, 4096) + 12)
        for got, want, most, r in zip((y, dw, db), both(x, w, b, dy), both(x.abs(), w.abs(), b.abs(), dy.abs()), rounds):
            assert bool(((got.double() - want).abs() <= r * 2.0 ** -24 * most + 1e-30).all())
    assert lib.aether_device_status() == 0


@pytest.mark.parametrize("S,H,W,Cin,Cout,f", [(6, 13, 17, 3, 20, 3), (3, 20, 33, 1, 16, 5), (4, 11, 12, 4, 33, 3), (5, 9, 30, 2, 7, 3)])
def test_values_that_are_not_finite(S, H, W, Cin, Cout, f):
    """Infinities and NaN in the images reach the pixels whose windows hold them and the filter values that they meet, at the images' edges, too."""
    import torch
    lib, p = _lib.lib(), f // 2
    g = torch.Generator(device="cuda").manual_seed(S + Cout)
    new = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    x, w, b, dy = new(S, H, W, Cin), new(f, f, Cin, Cout), new(Cout), new(S, H, W, Cout)
    x[0, 0, 0, 0], x[1, H - 1, W - 1, Cin - 1], x[2, 4, 5, 0] = float("inf"), float("nan"), -float("inf")
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, 1, 1, p, p, _lib.MATH_MODES["fp32"])
    n = lib.aether_conv2d_workspace_bytes(d)
    ws = torch.empty(n + 16, dtype=torch.uint8, device="cuda")
    y, dw, db = torch.empty_like(dy), torch.empty_like(w), torch.empty_like(b)
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.aether_conv2d_fwd(d, x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), ws.data_ptr(), n, stream) == 0
    assert lib.aether_conv2d_bwd(d, x.data_ptr(), dy.data_ptr(), w.data_ptr(), None, dw.data_ptr(), db.data_ptr(), ws.data_ptr(), n, 0, stream) == 0
    pads = torch.nn.functional.pad(x.double(), (0, 0, p, p, p, p))
    taps = [[pads[:, i:i + H, j:j + W] for j in range(f)] for i in range(f)]
    want = b.double() + sum(taps[i][j] @ w[i, j].double() for i in range(f) for j in range(f))
    grad = torch.stack([torch.stack([taps[i][j].reshape(-1, Cin).T @ dy.double().reshape(-1, Cout) for j in range(f)]) for i in range(f)])
    for got, exact in ((y, want), (dw, grad)):
        finite = exact.isfinite()
        assert torch.equal(got.isnan(), exact.isnan()) and torch.equal(got.isposinf(), exact.isposinf()) and torch.equal(got.isneginf(), exact.isneginf()) and not bool(finite.all())
        if bool(finite.any()):
            assert float((got.double() - exact)[finite].norm() / exact[finite].norm()) <= 1e-5
    assert bool(want[:, :, :, 0].isfinite().any()) and _lib.device_status() == 0
