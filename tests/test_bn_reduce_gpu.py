"""Batch_Norm's reductions at their edges: fewer rows than CTAs, than row lanes and than loads in flight, channel counts
that fill no warp, that end inside a round of 1024 channels, and tensors of eight million elements (the line between the
merged and the three-launch form is in test_bn_small_line_gpu.py).  Relative L2 <= 1e-5 against float64; the statistics of values far from zero keep the digits that the
values have (mean 100, deviation 1: the variance loses log2(100) bits, 1e-4)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,C,offset", [(1, 4, 0), (2, 36, 0), (31, 1028, 0), (33, 4, 0), (700, 20, 100), (9001, 8, 100), (5000, 100, 0),
                                           (129, 2052, 0), (131072, 64, 0), (131073, 64, 0), (50000, 1, 0), (300, 7, 0)])
def test_statistics_and_gradients(rows, C, offset):
    import torch
    from aether_ml_b200 import layers
    g = torch.Generator(device="cuda").manual_seed(rows + C)
    x = torch.randn((rows, C), generator=g, device="cuda") + offset
    dy = torch.randn((rows, C), generator=g, device="cuda")
    bn = layers.Batch_Norm(n_features=C)
    gamma, beta = torch.rand(C, generator=g, device="cuda") + 0.5, torch.randn(C, generator=g, device="cuda")
    bn.set_parameters(gamma, beta, torch.zeros(C, device="cuda"), torch.ones(C, device="cuda"))
    y = bn.forward(x, True)
    dx = bn.backward(dy)
    xd, gd = x.double(), dy.double()
    mean, var = xd.mean(0), xd.var(0, unbiased=False)
    inv = 1.0 / torch.sqrt(var + bn.epsilon)
    xh = (xd - mean) * inv
    dgamma, dbeta = (gd * xh).sum(0), gd.sum(0)
    want_dx = gamma.double() * inv / rows * (rows * gd - dbeta - xh * dgamma)
    tol = 1e-4 if offset else 1e-5

    def err(a, b):
        return float((a.double() - b).norm()) / max(float(b.norm()), 1e-30)

    assert err(bn.batch_mean.reshape(-1), mean) <= 1e-5
    if rows == 1:
        # y is beta and dx zero, as differences of numbers gamma / sqrt(epsilon) = up to 474 times as large as x and dy, each
        # the sum of two or three float coefficients' products: 2^-24 of that per coefficient
        scale = gamma.double() * inv
        assert bool(((y - beta).abs() <= 4 * 2.0 ** -24 * (scale * (xd.abs() + mean.abs()) + beta.abs())).all())
        assert bool((dx.abs() <= 8 * 2.0 ** -24 * scale * gd.abs()).all())
        return
    assert err(bn.batch_var.reshape(-1), var) <= tol
    assert err(y, gamma.double() * xh + beta.double()) <= tol
    assert err(bn.dbiases.reshape(-1), dbeta) <= tol
    assert err(bn.dweights.reshape(-1), dgamma) <= 10 * tol       # (sums of terms of both signs)
    assert err(dx, want_dx) <= tol if rows > 2 else True          # (two rows: dx is a difference of equals)
