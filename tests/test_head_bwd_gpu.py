"""The backward pass of classifier heads (Dense layers with few outputs): dX, dW and dB of one launch against float64, at the edges
of its row chunks, channel blocks and of the rule that sends many rows to sums of parts."""
import numpy as np
import pytest

from aether_ml_b200 import _lib

pytestmark = pytest.mark.gpu


def _ptr(t):
    return t.data_ptr() if t is not None else None


def _close(got, want, size, terms, what):
    # a sum of `terms` fp32 products by FMAs in any order: at most terms roundings of 2^-24 of the sum of absolute values
    err = np.abs(got.cpu().numpy().astype(np.float64) - want)
    assert (err <= terms * 2.0**-24 * size + 1e-30).all(), (what, float((err / (size + 1e-30)).max()))


@pytest.mark.parametrize("rows,n_in,classes", [(1, 128, 10), (63, 132, 2), (64, 256, 10), (65, 144, 15), (256, 256, 1), (300, 6000, 2), (257, 1028, 15), (1000, 128, 7),
                                               (512, 128, 3), (1024, 1024, 10), (1025, 132, 10), (3000, 260, 3), (40000, 128, 2)])
@pytest.mark.parametrize("wanted", ["all", "dx", "dw", "db", "dw db"])
def test_head_backward(rows, n_in, classes, wanted):
    import torch
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(rows + n_in)
    x, dy = torch.randn((rows, n_in), generator=g, device="cuda"), torch.randn((rows, classes), generator=g, device="cuda")
    w = torch.randn((n_in, classes), generator=g, device="cuda")
    d = _lib.AetherConvDesc(rows, 1, 1, n_in, classes, 1, 1, 1, 1, 0, 0, 0)
    ws = torch.empty(lib.aether_conv2d_workspace_bytes(d), dtype=torch.uint8, device="cuda")
    new = lambda name, *shape: torch.full(shape, float("nan"), device="cuda") if wanted == "all" or name in wanted.split() else None
    dx, dw, db = new("dx", rows, n_in), new("dw", n_in, classes), new("db", classes)
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.aether_conv2d_bwd(d, _ptr(x), _ptr(dy), _ptr(w), _ptr(dx), _ptr(dw), _ptr(db), _ptr(ws), ws.numel(), 0, stream) == 0
    X, DY, W = (t.cpu().numpy().astype(np.float64) for t in (x, dy, w))
    if dx is not None:
        _close(dx, DY @ W.T, np.abs(DY) @ np.abs(W).T, classes, "dx")
    if dw is not None:
        _close(dw, X.T @ DY, np.abs(X).T @ np.abs(DY), rows, "dw")
    if db is not None:
        _close(db, DY.sum(0), np.abs(DY).sum(0), rows, "db")
    if wanted == "all":                                     # without x: the same dX, nothing of the filter's
        other = torch.full_like(dx, float("nan"))
        assert lib.aether_conv2d_bwd(d, None, _ptr(dy), _ptr(w), _ptr(other), None, None, None, 0, 0, stream) == 0
        assert torch.equal(other, dx)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("rows,n_in,classes", [(1, 128, 10), (65, 144, 15), (256, 256, 1), (257, 1028, 3), (1024, 512, 10), (1025, 132, 10), (3000, 260, 7)])
@pytest.mark.parametrize("kind", ["int32", "int64", "targets"])
@pytest.mark.parametrize("wanted", ["all", "dw", "db", ""])
def test_head_loss_gradient(rows, n_in, classes, kind, wanted):
    """The same with the combined softmax / cross-entropy gradient, which every block computes for itself."""
    import torch
    lib, smooth = _lib.lib(), 0.1
    g = torch.Generator(device="cuda").manual_seed(rows + n_in)
    x, w = torch.randn((rows, n_in), generator=g, device="cuda"), torch.randn((n_in, classes), generator=g, device="cuda")
    prob = torch.softmax(torch.randn((rows, classes), generator=g, device="cuda"), 1)
    if kind == "targets":
        labels = torch.softmax(torch.randn((rows, classes), generator=g, device="cuda"), 1)
        onehot = labels.double()
    else:
        labels = torch.randint(0, classes, (rows,), generator=g, device="cuda").to(getattr(torch, kind))
        onehot = torch.nn.functional.one_hot(labels.long(), classes).double()
    given = [_ptr(labels) if kind == k else None for k in ("int32", "int64", "targets")]
    d = _lib.AetherConvDesc(rows, 1, 1, n_in, classes, 1, 1, 1, 1, 0, 0, 0)
    assert lib.aether_head_supported(d)
    ws = torch.empty(lib.aether_conv2d_workspace_bytes(d), dtype=torch.uint8, device="cuda")
    new = lambda *shape: torch.full(shape, float("nan"), device="cuda")
    dz, dx = new(rows, classes), new(rows, n_in)
    dw, db = new(n_in, classes) if wanted in ("all", "dw") else None, new(classes) if wanted in ("all", "db") else None
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.aether_head_cce_bwd_ex(d, _ptr(prob), *given, smooth, _ptr(x), _ptr(w), _ptr(dz), _ptr(dx), _ptr(dw), _ptr(db), _ptr(ws), ws.numel(), stream) == 0
    want = (prob.double() - (onehot * (1 - smooth) + smooth / classes)) / rows
    # a few roundings of numbers of at most 1, times 1 / rows
    assert float((dz.double() - want).abs().max()) <= 4 * 2.0**-24 / rows
    X, DZ, W = (t.cpu().numpy().astype(np.float64) for t in (x, dz, w))
    _close(dx, DZ @ W.T, np.abs(DZ) @ np.abs(W).T, classes, "dx")
    if dw is not None:
        _close(dw, X.T @ DZ, np.abs(X).T @ np.abs(DZ), rows, "dw")
    if db is not None:
        _close(db, DZ.sum(0), np.abs(DZ).sum(0), rows, "db")
    assert _lib.device_status() == 0
