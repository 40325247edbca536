"""Filter gradients at the image heights where strips are divided differently (13 to 24 rows, and heights that no strip divides) and with one group of
rows per pair of CTAs (256 output channels; TF32: one, two and four, channels that fill no row of 128 bytes), against float64 on operands rounded as the kernels round them.  Sums of n fp32 products in
any order are within n roundings of the sum of absolute values, of which tcgen05 truncates each: n * 2^-23."""
import ctypes

import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,mode", [(300, 16, 16, 64, 64, 3, "bf16"), (200, 13, 13, 64, 128, 3, "bf16"), (150, 15, 14, 128, 128, 3, "bf16"), (120, 18, 18, 96, 160, 3, "bf16"),
                                                   (90, 24, 24, 32, 64, 5, "bf16"), (60, 23, 21, 128, 64, 3, "bf16"), (100, 17, 30, 64, 64, 3, "bf16"), (200, 13, 13, 128, 256, 3, "bf16"),
                                                   (100, 25, 24, 128, 256, 3, "bf16"), (256, 8, 8, 256, 256, 3, "bf16"), (64, 9, 9, 256, 256, 5, "bf16"), (128, 16, 16, 128, 128, 3, "tf32"),
                                                   (200, 13, 13, 96, 116, 3, "tf32"), (100, 16, 16, 148, 236, 3, "tf32"), (40, 20, 20, 64, 500, 5, "tf32"), (60, 13, 13, 292, 236, 5, "tf32")])
def test_filter_gradient(S, H, W, Cin, Cout, f, mode):
    import torch
    lib, pad = _lib.lib(), (f - 1) // 2
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, 1, 1, pad, pad, _lib.MATH_MODES[mode])
    g = torch.Generator(device="cuda").manual_seed(S + H)
    bits = 16 if mode == "bf16" else 13                      # of mantissa that the mode drops
    cut = lambda t: (t.view(torch.int32) & ~((1 << bits) - 1)).view(torch.float32)        # representable: nothing is rounded
    x, dy = (cut(torch.randn((S, H, W, c), generator=g, device="cuda")) for c in (Cin, Cout))
    w = torch.zeros((f, f, Cin, Cout), device="cuda")
    n = lib.aether_conv2d_workspace_bytes(ctypes.byref(d))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    dw, db = torch.full_like(w, float("nan")), torch.full((Cout,), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.aether_conv2d_bwd(d, x.data_ptr(), dy.data_ptr(), w.data_ptr(), None, dw.data_ptr(), db.data_ptr(), ws.data_ptr(), n, 0, stream) == 0

    def product(a, b):                                      # in float64, a tap at a time
        pads = torch.nn.functional.pad(a, (0, 0, pad, pad, pad, pad))
        cols = b.reshape(-1, Cout)
        return torch.stack([torch.stack([pads[:, i:i + H, j:j + W].reshape(-1, Cin).T @ cols for j in range(f)]) for i in range(f)])
    want, size = product(x.double(), dy.double()), product(x.double().abs(), dy.double().abs())
    assert bool(((dw.double() - want).abs() <= S * H * W * 2.0**-23 * size).all())
    assert float((dw.double() - want).norm() / want.norm()) <= 1e-4          # (truncation of random signs: 1e-6 to 2e-5 measured)
    assert _lib.device_status() == 0
