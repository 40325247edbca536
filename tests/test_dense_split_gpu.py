"""Dense layers of few tiles, whose K chunks two, four or eight CTAs share: K that divides evenly and not, rows and columns that overhang a tile, one tile, with
and without the activation, against float64 on operands that bf16 represents.  The same bits with and without it, and on a second call.  Sums of K products in
fp32, which tcgen05 truncates: (K + 8) * 2^-23 of the sum of absolute values."""
import ctypes

import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,K,N", [(100, 3136, 128), (256, 2048, 256), (300, 1800, 320), (500, 2600, 416), (1, 5000, 32), (129, 1028, 36), (40, 1024, 64), (128, 960, 512), (512, 3136, 128), (480, 4096, 128), (512, 2112, 256), (500, 3000, 512)])
def test_dense_forward(rows, K, N):
    import torch
    lib = _lib.lib()
    d = _lib.AetherConvDesc(rows, 1, 1, K, N, 1, 1, 1, 1, 0, 0, _lib.MATH_MODES["bf16"])
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w, b = torch.randn((rows, K), generator=g, device="cuda").bfloat16().float(), torch.randn((K, N), generator=g, device="cuda").bfloat16().float(), torch.randn((N,), generator=g, device="cuda")
    n = lib.aether_conv2d_workspace_bytes(ctypes.byref(d))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    stream, P = torch.cuda.current_stream().cuda_stream, lambda t: t.data_ptr()
    want, size = x.double() @ w.double() + b.double(), x.double().abs() @ w.double().abs() + b.double().abs()
    outs = []
    for _ in range(2):
        y, y2, act = (torch.full((rows, N), float("nan"), device="cuda") for _ in range(3))
        assert lib.aether_conv2d_fwd(ctypes.byref(d), P(x), P(w), P(b), P(y), P(ws), n, stream) == 0
        assert lib.aether_conv2d_act_fwd(ctypes.byref(d), P(x), P(w), P(b), P(y2), P(act), 0.125, None, 0, P(ws), n, 0, stream) == 0
        assert torch.equal(y, y2) and torch.equal(act, torch.where(y > 0, y, 0.125 * y))
        assert bool(((y.double() - want).abs() <= (K + 8) * 2.0**-23 * size).all())
        outs.append(y)
    assert torch.equal(*outs) and _lib.device_status() == 0


def test_values_that_are_not_finite():
    """An infinity and a NaN in two CTAs' parts of K: in the rows that hold them, as in float64."""
    import torch
    lib = _lib.lib()
    rows, K, N = 130, 2048, 64
    d = _lib.AetherConvDesc(rows, 1, 1, K, N, 1, 1, 1, 1, 0, 0, _lib.MATH_MODES["bf16"])
    g = torch.Generator(device="cuda").manual_seed(4)
    x, w, b = torch.randn((rows, K), generator=g, device="cuda").bfloat16().float(), torch.randn((K, N), generator=g, device="cuda").bfloat16().float(), torch.randn((N,), generator=g, device="cuda")
    x[3, 7], x[4, K - 1], x[5, 1000], x[6, 0], x[6, K - 2], x[129, 512] = float("inf"), -float("inf"), float("nan"), float("inf"), -float("inf"), float("inf")
    n = lib.aether_conv2d_workspace_bytes(ctypes.byref(d))
    ws, y = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.empty((rows, N), device="cuda")
    P = lambda t: t.data_ptr()
    assert lib.aether_conv2d_fwd(ctypes.byref(d), P(x), P(w), P(b), P(y), P(ws), n, torch.cuda.current_stream().cuda_stream) == 0
    want = x.double() @ w.double() + b.double()
    finite = want.isfinite()
    assert int((~finite).any(1).sum()) == 5 and torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isposinf(), want.isposinf()) and torch.equal(y.isneginf(), want.isneginf())
    size = (x.double().abs() @ w.double().abs() + b.double().abs())[finite]
    assert bool(((y.double() - want)[finite].abs() <= (K + 8) * 2.0**-23 * size).all()) and _lib.device_status() == 0
