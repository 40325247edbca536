"""Which tensors take Batch_Norm's one-pass form: rows times channels in whole blocks of 32, on both sides of the line (one launch
less each way below it), with the results of float64 on both: relative L2 <= 1e-5, as the reductions' other tests."""
import pytest

pytestmark = pytest.mark.gpu

M = 1 << 20


@pytest.mark.parametrize("C,filled", [(4, 32), (8, 32), (32, 32), (36, 64), (64, 64), (260, 288)])
@pytest.mark.parametrize("beyond", [0, 1])
@pytest.mark.parametrize("form", ["alone", "chain"])
def test_line(C, filled, beyond, form):
    import torch
    from aether_ml_b200 import _lib, layers as L
    from aether_ml_b200.model import _Chain
    rows = (4 if form == "alone" else 7) * M // filled + beyond
    g = torch.Generator(device="cuda").manual_seed(C)
    x, dy = torch.randn((rows, C), generator=g, device="cuda"), torch.randn((rows, C), generator=g, device="cuda")
    bn, act = L.Batch_Norm(n_features=C), L.ReLU()
    bn.gamma.copy_(torch.rand(C, generator=g, device="cuda") + 0.5)
    bn.beta.copy_(torch.randn(C, generator=g, device="cuda"))
    chain = _Chain.find([bn, act], 0)
    counts = [_lib.launch_count()]
    if form == "alone":
        y = bn.forward(x, True)
        counts.append(_lib.launch_count())
        bn.backward(dy)
    else:
        assert chain.forward([bn, act], 0, x, True)
        y = act.output
        counts.append(_lib.launch_count())
        assert chain.backward([bn, act], 0, dy)
    counts.append(_lib.launch_count())
    assert [b - a for a, b in zip(counts, counts[1:])] == [2 + beyond] * 2
    xd, gd, ga = x.double(), dy.double(), bn.gamma.double()
    mean, var = xd.mean(0), xd.var(0, unbiased=False)
    inv = 1.0 / torch.sqrt(var + bn.epsilon)
    xh = (xd - mean) * inv
    want = xh * ga + bn.beta.double()
    if form == "chain":
        gd = gd * (want >= 0)
        want = want.clamp(min=0)
    dgamma, dbeta = (gd * xh).sum(0), gd.sum(0)
    want_dx = ga * inv / rows * (rows * gd - dbeta - xh * dgamma)

    def err(a, b):
        return float((a.double() - b).norm() / b.norm())
    # (a cell within a rounding of zero may pass its gradient on one side only: a few of millions, each a whole value)
    tol = 1e-5 if form == "alone" else 1e-3
    assert err(y, want) <= 1e-5 and err(bn.dinputs, want_dx) <= tol and err(bn.dbiases, dbeta) <= tol and err(bn.dweights, dgamma) <= tol
