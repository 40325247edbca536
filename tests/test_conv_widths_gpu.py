"""Column tiles of 96 and 192 channels in the per-tap kernel: full, overhanging the last channels (whose filter tile reads on into the next tap), two of
them, with bias and statistics, few and many tiles (pairs of CTAs), against float64 on operands that the mode represents.  Forward and dX sum n
products in fp32, which tcgen05 truncates: n * 2^-23 of the sum of absolute values."""
import ctypes

import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu

SHAPES = [(100, 8, 8, 192, 192, 3, "bf16"), (256, 8, 8, 160, 180, 3, "bf16"), (700, 8, 8, 64, 192, 3, "bf16"), (9, 7, 7, 32, 132, 3, "bf16"), (1500, 6, 6, 192, 192, 3, "bf16"),
          (100, 9, 9, 160, 96, 3, "tf32"), (60, 11, 10, 96, 224, 3, "tf32"), (400, 8, 8, 92, 192, 3, "tf32"), (30, 10, 10, 224, 160, 5, "tf32"), (900, 8, 8, 192, 64, 1, "tf32"), (3, 6, 5, 68, 132, 3, "tf32")]


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,mode", SHAPES)
def test_forward_and_dx(S, H, W, Cin, Cout, f, mode):
    import torch
    lib, pad = _lib.lib(), (f - 1) // 2
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, 1, 1, pad, pad, _lib.MATH_MODES[mode])
    g = torch.Generator(device="cuda").manual_seed(S + Cout)
    bits = 16 if mode == "bf16" else 13                      # of mantissa that the mode drops
    cut = lambda t: (t.view(torch.int32) & ~((1 << bits) - 1)).view(torch.float32)
    x, dy = (cut(torch.randn((S, H, W, c), generator=g, device="cuda")) for c in (Cin, Cout))
    w, b = cut(torch.randn((f, f, Cin, Cout), generator=g, device="cuda")), torch.randn((Cout,), generator=g, device="cuda")
    n = lib.aether_conv2d_workspace_bytes(ctypes.byref(d))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    y, y2, dx = torch.full_like(dy, float("nan")), torch.full_like(dy, float("nan")), torch.full_like(x, float("nan"))
    stream = torch.cuda.current_stream().cuda_stream
    P = lambda t: t.data_ptr()
    assert lib.aether_conv2d_fwd(d, P(x), P(w), P(b), P(y), P(ws), n, stream) == 0
    assert lib.aether_conv2d_bwd(d, None, P(dy), P(w), P(dx), None, None, P(ws), n, 2, stream) == 0
    blocks = lib.aether_conv2d_bnstats_blocks(d)
    assert blocks > 0
    part = torch.full((blocks, 3, Cout), float("nan"), device="cuda")
    assert lib.aether_conv2d_fwd_bnstats(d, P(x), P(w), P(b), P(y2), P(part), part.numel() * 4, P(ws), n, stream) == 0
    assert torch.equal(y, y2)

    def taps(a, m, sign):                                   # a: (S, H, W, C) in float64; m: (f, f, C, N)
        pads = torch.nn.functional.pad(a, (0, 0, pad, pad, pad, pad))
        out = 0
        for i in range(f):
            for j in range(f):
                r, c = (i, j) if sign > 0 else (2 * pad - i, 2 * pad - j)
                out = out + pads[:, r:r + H, c:c + W] @ m[i, j]
        return out
    wd = w.double()
    want, size = taps(x.double(), wd, 1) + b.double(), taps(x.double().abs(), wd.abs(), 1) + b.double().abs()
    assert bool(((y.double() - want).abs() <= f * f * Cin * 2.0**-23 * size).all())
    back, size = taps(dy.double(), wd.transpose(2, 3), -1), taps(dy.double().abs(), wd.abs().transpose(2, 3), -1)
    assert bool(((dx.double() - back).abs() <= f * f * Cout * 2.0**-23 * size).all())
    p = part.double()
    count = p[:, 0].sum(0)
    assert bool((count == S * H * W).all())
    mean = (p[:, 0] * p[:, 1]).sum(0) / count
    m2 = (p[:, 2] + p[:, 0] * (p[:, 1] - mean) ** 2).sum(0)
    yd = y.double().reshape(-1, Cout)
    # a partial's mean and squares are rounded to 24 bits, its sums have S * H * W terms: 1e-5 of the deviation is a hundred times that
    assert bool(((mean - yd.mean(0)).abs() <= 1e-5 * yd.std(0)).all()) and bool(((m2 / count / yd.var(0, unbiased=False) - 1).abs() <= 1e-4).all())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,mode", [(20, 13, 13, 64, 64, 3, "bf16"), (40, 15, 15, 64, 128, 3, "bf16"), (30, 16, 16, 32, 64, 3, "bf16"), (12, 31, 31, 128, 64, 3, "bf16"), (9, 44, 44, 32, 128, 3, "bf16"),
                                                   (33, 16, 16, 28, 64, 3, "tf32"), (9, 44, 44, 64, 64, 3, "tf32"), (25, 16, 14, 64, 96, 5, "bf16"), (20, 19, 19, 64, 192, 3, "bf16"),
                                                   # (rounds enough for the kernel that keeps a window, the others above run tap by tap)
                                                   (700, 13, 13, 64, 64, 3, "bf16"), (500, 16, 16, 64, 128, 3, "bf16"), (100, 44, 44, 64, 64, 3, "bf16"), (700, 16, 16, 28, 64, 3, "tf32"), (500, 13, 13, 32, 64, 3, "tf32"),
                                                   (600, 16, 14, 64, 96, 5, "bf16")])
def test_images_that_fill_little_of_a_strip(S, H, W, Cin, Cout, f, mode):
    test_forward_and_dx(S, H, W, Cin, Cout, f, mode)
