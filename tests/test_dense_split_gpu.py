"""Dense layers of few tiles, whose K chunks two, four or eight CTAs share: K that divides evenly and not, rows and columns that overhang a tile, one tile, with
and without the activation, against float64 on operands that bf16 represents.  The same bits with and without it, and on a second call.  Sums of K products in
fp32, which tcgen05 truncates: (K + 8) * 2^-23 of the sum of absolute values."""
import ctypes

import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,K,N", [(100, 3136, 128), (256, 2048, 256), (300, 1800, 320), (500, 2600, 416), (1, 5000, 32), (129, 1028, 36), (40, 1024, 64), (128, 960, 512)])
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
