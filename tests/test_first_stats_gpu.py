"""Batch_Norm statistics from the epilogue of first layers, for channels whose mean is far from zero compared with their
spread.  Sums are fp32 about a pivot close to the mean, in chains of at most 4 rows per tile and a tree of 3 additions: the relative
error of the variance is at most (4 T + 3 + 4) * 2^-24 for CTAs of T tiles (the last 4: pivot, product and output), whatever
the mean is; the mean is rounded once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias", [0.0, 30.0, -300.0])
@pytest.mark.parametrize("S,H,Cin,Cout", [(1, 5, 1, 16), (16, 28, 1, 32), (3, 11, 3, 20), (256, 28, 1, 32), (64, 32, 3, 128), (9, 32, 3, 160), (200, 17, 2, 256)])
def test_mean_far_from_zero(S, H, Cin, Cout, bias):
    import torch
    from aether_ml_b200 import layers as L
    np.random.seed(1)
    g = torch.Generator(device="cuda").manual_seed(2)
    conv, bn = L.Conv_Layer((H, H, Cin), Cout), L.Batch_Norm(n_features=Cout)
    conv.emit_bn_stats, bn.stats_from = True, conv
    conv.biases.copy_(torch.randn(Cout, generator=g, device="cuda") + bias)
    y = conv.forward(torch.rand((S, H, H, Cin), generator=g, device="cuda"), True)
    assert conv.bn_partials is not None
    bn.forward(y, True)
    mean, var = y.double().mean((0, 1, 2)), y.double().var((0, 1, 2), unbiased=False)
    tiles = -(-(-(-S * H * H // 128)) // torch.cuda.get_device_properties(0).multi_processor_count)
    bound = (4 * tiles + 7) * 2.0 ** -24
    assert float(((bn.batch_var.flatten().double() - var).abs() / var).max()) <= bound
    assert bool(((bn.batch_mean.flatten().double() - mean).abs() <= 2.0 ** -23 * mean.abs() + bound * var.sqrt()).all())
