"""dX of first layers at stride 1 with 3x3 and 5x5 filters, tile by tile: strips of 4 and 8 rows, tiles of 8, 16 and 32 columns, strips of several images in
a tile, one and several chunks of channels, more tiles than blocks (the two stages' barriers change phase), few output channels (two groups of columns),
paddings other than "same".  fp32 sums of n products in any order: within n roundings of 2^-24 of the sum of absolute values."""
import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu

# (S, H, W, Cin, Cout, f, padH, padW)
SHAPES = [(128, 32, 32, 3, 32, 3, 1, 1), (600, 17, 33, 1, 64, 3, 1, 1), (330, 16, 40, 3, 36, 3, 1, 1), (700, 7, 7, 3, 100, 3, 1, 1), (701, 9, 14, 2, 12, 3, 1, 1),
          (64, 28, 28, 4, 32, 3, 0, 0), (90, 33, 31, 3, 72, 5, 2, 2), (200, 20, 28, 1, 16, 5, 2, 2), (130, 30, 64, 3, 16, 5, 0, 0), (40, 8, 8, 4, 128, 5, 2, 2),
          (3, 70, 41, 3, 33, 3, 1, 1), (150, 20, 21, 4, 61, 5, 2, 2), (20, 11, 13, 3, 24, 3, 2, 0), (9, 12, 10, 1, 32, 5, 4, 5), (1, 3, 3, 3, 4, 3, 0, 0), (200, 28, 28, 4, 20, 5, 2, 2)]


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,ph,pw", SHAPES)
def test_dx_of_first_layers_by_tiles(S, H, W, Cin, Cout, f, ph, pw):
    import torch
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(S + Cout)
    Ho, Wo = H + 2 * ph - f + 1, W + 2 * pw - f + 1
    dy, w = torch.randn((S, Ho, Wo, Cout), generator=g, device="cuda"), torch.randn((f, f, Cin, Cout), generator=g, device="cuda")
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, 1, 1, ph, pw, 0)
    ws = torch.empty(lib.aether_conv2d_workspace_bytes(d) + 16, dtype=torch.uint8, device="cuda")
    dx = torch.full((S, H, W, Cin), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(2):
        assert lib.aether_conv2d_bwd(d, None, dy.data_ptr(), w.data_ptr(), dx.data_ptr(), None, None, ws.data_ptr(), ws.numel(), 0, stream) == 0

    def gather(a, b):                                       # in float64: dy padded by what a tap can reach, a product per tap
        pad = torch.nn.functional.pad(a, (0, 0, f, f + pw, f, f + ph))
        out = torch.zeros((S, H, W, Cin), dtype=torch.float64, device="cuda")
        for i in range(f):
            for j in range(f):
                r, c = ph - i + f, pw - j + f
                out += pad[:, r:r + H, c:c + W] @ b[i, j].T
        return out
    want, size = gather(dy.double(), w.double()), gather(dy.double().abs(), w.double().abs())
    assert bool(((dx.double() - want).abs() <= f * f * Cout * 2.0**-24 * size + 1e-30).all())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("S,H,W,Cin,Cout,f", [(128, 32, 32, 3, 32, 3), (330, 16, 40, 3, 36, 3), (64, 9, 14, 2, 12, 3), (90, 33, 31, 3, 72, 5), (9, 10, 13, 1, 33, 3), (30, 20, 28, 1, 16, 5), (70, 7, 7, 4, 100, 3)])
def test_filter_values_that_are_not_finite(S, H, W, Cin, Cout, f):
    """An infinite or NaN filter value reaches the pixels that its tap reaches: those whose column of dy lies in the image."""
    import torch
    lib, pad = _lib.lib(), f // 2
    g = torch.Generator(device="cuda").manual_seed(S)
    dy, w = torch.randn((S, H, W, Cout), generator=g, device="cuda"), torch.randn((f, f, Cin, Cout), generator=g, device="cuda")
    w[pad, 0, 0, Cout // 2] = float("inf")                   # (the middle row: its rows of dy are in the image everywhere)
    if Cin > 1:
        w[pad, f - 1, Cin - 1, Cout - 1] = float("nan")
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, 1, 1, pad, pad, 0)
    ws = torch.empty(lib.aether_conv2d_workspace_bytes(d) + 16, dtype=torch.uint8, device="cuda")
    dx = torch.zeros((S, H, W, Cin), device="cuda")
    assert lib.aether_conv2d_bwd(d, None, dy.data_ptr(), w.data_ptr(), dx.data_ptr(), None, None, ws.data_ptr(), ws.numel(), 0, torch.cuda.current_stream().cuda_stream) == 0

    def gather(a, b):
        rows = torch.nn.functional.pad(a, (0, 0, 0, 0, f, f))
        out = torch.zeros((S, H, W, Cin), dtype=torch.float64, device="cuda")
        for i in range(f):
            for j in range(f):
                lo, hi = max(0, j - pad), min(W, W + j - pad)            # columns that see column wo = column + pad - j of dy
                out[:, :, lo:hi] += rows[:, pad - i + f:pad - i + f + H, lo + pad - j:hi + pad - j] @ b[i, j].T
        return out
    want = gather(dy.double(), w.double())
    size = gather(dy.double().abs(), w.double().abs().nan_to_num(0.0, 0.0))
    finite = want.isfinite()
    assert torch.equal(dx.isfinite(), finite) and torch.equal(dx.isnan(), want.isnan()) and torch.equal(dx.isposinf(), want.isposinf())
    assert bool(finite[:, :, W - pad:, 0].all()) and not bool(finite[:, :, :W - pad, 0].any())
    assert Cin == 1 or (bool(finite[:, :, :pad, Cin - 1].all()) and not bool(finite[:, :, pad:, Cin - 1].any()))
    assert bool(((dx.double() - want)[finite].abs() <= f * f * Cout * 2.0**-24 * size[finite]).all())
    assert _lib.device_status() == 0
