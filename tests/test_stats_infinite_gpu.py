"""An infinite value in a convolution's output: the batch mean from the epilogue's statistics is infinite with its sign, the variance
not a number, as sums over the output give them; other channels are not touched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,H,Cin,Cout,f", [(4, 16, 16, 32, 1), (4, 64, 16, 32, 1), (3, 16, 4, 32, 1), (2, 16, 3, 32, 1)])
def test_mean_stays_infinite(S, H, Cin, Cout, f):
    import torch
    from aether_ml_b200 import layers as L
    np.random.seed(1)
    conv, bn = L.Conv_Layer((H, H, Cin), Cout, (f, f)), L.Batch_Norm(n_features=Cout)
    conv.emit_bn_stats, bn.stats_from = True, conv
    w = conv.filter_weights.clone()
    w[:, :, :, : Cout // 2] = w[:, :, :, : Cout // 2].sign() * 0.5       # (as large as a bf16 rounding keeps)
    w[0, 0, 0, Cout // 2:] = 0.0
    x = torch.rand((S, H, H, Cin), device="cuda")
    x[S - 1, H - 1, 5, 0] = 3e38
    w[0, 0, 0, : Cout // 2] *= 8.0                                         # 1.2e39: beyond fp32
    conv.set_parameters(w, torch.zeros(Cout, device="cuda"))
    y = conv.forward(x, True)
    assert conv.bn_partials is not None
    bn.forward(y, True)
    sums = y.double().sum((0, 1, 2))
    assert bool(torch.isinf(sums[: Cout // 2]).all()) and bool(torch.isfinite(sums[Cout // 2:]).all())
    mean, var = bn.batch_mean.flatten(), bn.batch_var.flatten()
    assert torch.equal(mean[: Cout // 2].double(), sums[: Cout // 2]) and bool(torch.isnan(var[: Cout // 2]).all())
    want = y.double()[..., Cout // 2:]
    assert float((mean[Cout // 2:].double() - want.mean((0, 1, 2))).abs().max()) <= 1e-6
    assert float((var[Cout // 2:].double() / want.var((0, 1, 2), unbiased=False) - 1).abs().max()) <= 1e-5
