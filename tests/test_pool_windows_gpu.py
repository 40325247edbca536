"""Pooling and the per-channel passes where no row of channels is a whole number of 16-byte pieces and no whole number of windows covers the image: windows of 2,
3 and other sizes, ragged at the right, at the bottom and at both, max and average, against PyTorch in float64.  Max and the cells outside every window are exact;
averages are within fH * fW + 1 roundings of 2^-24, the channel passes within 3 of their terms' absolute values."""
import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [4, 5, 61, 128, 1])
@pytest.mark.parametrize("S,H,W,fH,fW", [(3, 9, 10, 2, 2), (2, 11, 10, 3, 3), (2, 12, 14, 3, 3), (5, 8, 8, 2, 2), (2, 10, 13, 4, 3), (1, 3, 3, 3, 3), (2, 7, 15, 1, 2),
                                           # large windows: few of them cell by cell, many window by window
                                           (3, 29, 30, 14, 9), (1, 60, 51, 15, 17), (40, 41, 50, 4, 3), (64, 43, 50, 14, 9), (96, 33, 31, 8, 8)])
@pytest.mark.parametrize("kind", ["max", "average"])
def test_windows_that_leave_cells_over(C, S, H, W, fH, fW, kind):
    import torch
    import torch.nn.functional as F
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(C + H)
    Ho, Wo = H // fH, W // fW
    x, dy = torch.randn((S, H, W, C), generator=g, device="cuda"), torch.randn((S, Ho, Wo, C), generator=g, device="cuda")
    y, dx = torch.full_like(dy, float("nan")), torch.full_like(x, float("nan"))
    arg = torch.zeros((S, Ho, Wo, C), dtype=torch.uint8, device="cuda")
    code = _lib.POOL_MAX if kind == "max" else _lib.POOL_AVG
    st = torch.cuda.current_stream().cuda_stream
    assert lib.aether_pool_fwd(x.data_ptr(), y.data_ptr(), arg.data_ptr(), S, H, W, C, fH, fW, fH, fW, code, st) == 0
    assert lib.aether_pool_bwd(dy.data_ptr(), arg.data_ptr(), dx.data_ptr(), S, H, W, C, fH, fW, fH, fW, code, st) == 0
    x, y, dx, dy = x.cpu(), y.cpu(), dx.cpu(), dy.cpu()
    xd = x.double().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    out = (F.max_pool2d if kind == "max" else F.avg_pool2d)(xd, (fH, fW))
    out.backward(dy.double().permute(0, 3, 1, 2))
    tol = 0.0 if kind == "max" else (fH * fW + 1) * 2.0 ** -24
    scale = F.avg_pool2d(xd.detach().abs(), (fH, fW)).permute(0, 2, 3, 1)
    assert bool(((y.double() - out.detach().permute(0, 2, 3, 1)).abs() <= tol * scale).all())
    want = xd.grad.permute(0, 2, 3, 1)
    assert bool(((dx.double() - want).abs() <= tol * want.abs()).all())


@pytest.mark.parametrize("rows,C,shift", [(1000, 61, 0), (1001, 3, 0), (77, 1, 0), (512, 30, 0), (333, 7, 1), (255, 3, 0), (256, 3, 0), (769, 1, 0), (20, 5, 0)])
def test_channel_passes_of_ragged_rows(rows, C, shift):
    """shift: arrays that begin between two 16-byte boundaries."""
    import torch
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(rows)
    n = rows * C
    new = lambda: torch.randn(n + shift, generator=g, device="cuda")[shift:]
    x, dy = new(), new()
    y, dx = torch.full_like(new(), float("nan")), torch.full((n + shift,), float("nan"), device="cuda")[shift:]
    scale = torch.randn(C, generator=g, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert lib.aether_channel_scale(x.data_ptr(), scale.data_ptr(), y.data_ptr(), n, C, st) == 0
    assert torch.equal(y.view(rows, C), x.view(rows, C) * scale)
    if shift:
        return
    gamma, beta, mean = (torch.randn(C, generator=g, device="cuda") for _ in range(3))
    var = torch.rand(C, generator=g, device="cuda") + 0.5
    ws = torch.empty(lib.aether_bn_workspace_bytes(rows, C), dtype=torch.uint8, device="cuda")
    dg, db = torch.empty_like(gamma), torch.empty_like(beta)
    assert lib.aether_bn_bwd(x.data_ptr(), dy.data_ptr(), gamma.data_ptr(), mean.data_ptr(), var.data_ptr(), dx.data_ptr(), dg.data_ptr(), db.data_ptr(),
                             rows, C, 1e-5, ws.data_ptr(), ws.numel(), st) == 0
    X, D, G = x.view(rows, C).double(), dy.view(rows, C).double(), gamma.double()
    inv = (var.double() + 1e-5) ** -0.5
    hat = (X - mean.double()) * inv
    parts = (D, -D.mean(0), -hat * (D * hat).mean(0))
    want = G * inv * sum(parts)
    # (the third term's coefficients are those of x and of 1, whose products cancel in hat; the means are sums of `rows` fp32 terms in partial sums of at most 64)
    size = (G * inv).abs() * (D.abs() + D.abs().mean(0) + (X.abs() + mean.double().abs()) * inv * (D * hat).abs().mean(0))
    assert bool(((dx.view(rows, C).double() - want).abs() <= 72 * 2.0 ** -24 * size).all())
