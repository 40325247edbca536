"""Filter gradients of single-precision layers whose units have 128 channels of dy: the second 64 of a tile partly filled, full and with a tile behind
them, strided, one and several units per CTA.  Sums of n fp32 products in any order: within n roundings of 2^-24 of the sum of absolute values."""
import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,H,W,Cin,Cout,f,s", [(100, 57, 45, 48, 72, 3, 2), (30, 40, 41, 61, 99, 3, 1), (40, 33, 32, 64, 128, 3, 1), (100, 12, 13, 200, 250, 3, 1),
                                                (40, 28, 28, 32, 65, 5, 1), (50, 14, 14, 256, 256, 3, 1)])
def test_filter_gradient(S, H, W, Cin, Cout, f, s):
    import torch
    lib, pad = _lib.lib(), (f - 1) // 2
    Ho, Wo = (H + 2 * pad - f) // s + 1, (W + 2 * pad - f) // s + 1
    d = _lib.AetherConvDesc(S, H, W, Cin, Cout, f, f, s, s, pad, pad, _lib.MATH_MODES["fp32"])
    g = torch.Generator(device="cuda").manual_seed(S + Cout)
    x, dy = torch.randn((S, H, W, Cin), generator=g, device="cuda"), torch.randn((S, Ho, Wo, Cout), generator=g, device="cuda")
    w = torch.zeros((f, f, Cin, Cout), device="cuda")
    n = lib.aether_conv2d_workspace_bytes(d)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    dw, db = torch.full_like(w, float("nan")), torch.full((Cout,), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.aether_conv2d_bwd(d, x.data_ptr(), dy.data_ptr(), w.data_ptr(), None, dw.data_ptr(), db.data_ptr(), ws.data_ptr(), n, 0, stream) == 0

    def product(a, b):                                      # in float64, a tap at a time
        pads = torch.nn.functional.pad(a, (0, 0, pad, pad + s, pad, pad + s))
        cols = b.reshape(-1, Cout)
        return torch.stack([torch.stack([pads[:, i:i + Ho * s:s, j:j + Wo * s:s].reshape(-1, Cin).T @ cols for j in range(f)]) for i in range(f)])
    want, size = product(x.double(), dy.double()), product(x.double().abs(), dy.double().abs())
    assert bool(((dw.double() - want).abs() <= S * Ho * Wo * 2.0**-24 * size).all())
    assert float((dw.double() - want).norm() / want.norm()) <= 3e-6          # (signs are random; measured 1e-7 to 2e-7)
    assert bool(((db.double() - dy.double().sum((0, 1, 2))).abs() <= S * Ho * Wo * 2.0**-24 * dy.double().abs().sum((0, 1, 2))).all())
    assert _lib.device_status() == 0
