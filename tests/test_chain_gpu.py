"""Batch_Norm, activation, spatial dropout and max pooling that a model runs in one pass each way while every layer keeps
its own arrays: the same arrays as the layers produce one by one.  Forward values are the same operations (equal bits);
backward, the Batch_Norm sums are grouped differently: fp32 sums, relative L2 <= 1e-5."""
import numpy as np
import pytest

from oracle import aether_oracle as O

pytestmark = pytest.mark.gpu

# (S, H, W, C, alpha, dropout, window or None): whole and ragged windows, 3x3 windows, no pooling, C / 4 no power of two, 2-D
CASES = [(3, 8, 6, 16, 0.0, True, 2), (2, 7, 9, 20, 0.1, True, 2), (2, 7, 8, 12, 0.0, False, 3), (5, 5, 5, 64, 0.2, True, None),
         (37, None, None, 36, 0.01, False, None), (2, 2, 2, 1028, 0.0, True, 2), (150, 28, 28, 32, 0.0, False, 2), (1, 3, 3, 4, 0.0, True, 3)]


@pytest.mark.parametrize("case", CASES)
def test_chain_equals_the_layers_one_by_one(case):
    import torch
    from aether_ml_b200 import layers as Ly, model as M
    S, H, W, C, alpha, with_drop, window = case
    g = torch.Generator(device="cuda").manual_seed(4)
    shape = (S, C) if H is None else (S, H, W, C)
    x = torch.randn(shape, generator=g, device="cuda") + 0.3

    def build():
        m = M.Model()
        m.add(Ly.Batch_Norm(n_features=C))
        m.add(Ly.Leaky_ReLU(alpha) if alpha else Ly.ReLU())
        if with_drop:
            d = Ly.Layer_Dropout_Spatial(0.3)
            d.fixed_mask = np.where(np.arange(C) % 3 == 0, 0.0, 1.0 / 0.7)
            m.add(d)
        if window:
            m.add(Ly.Pooling((window, window), (window, window), "valid", "max"))
        gg = torch.Generator(device="cuda").manual_seed(5)
        m.layers[0].gamma.copy_(torch.rand(C, generator=gg, device="cuda") + 0.5)
        m.layers[0].beta.copy_(torch.randn(C, generator=gg, device="cuda") * 0.2)
        m.set(loss=Ly.Loss_CategoricalCrossEntropy())
        m.finalize()
        return m

    one, ref = build(), build()
    assert 0 in one._chains
    ref._chains, ref._chain_ends = {}, {}
    for training in (True, False, True):
        a, b = one.forward(x, training), ref.forward(x, training)
        assert torch.equal(a, b)
        for p, q in zip(one.layers, ref.layers):
            assert torch.equal(p.inputs, q.inputs) and torch.equal(p.output, q.output)
        assert torch.equal(one.layers[0].running_var, ref.layers[0].running_var)
    if window:
        assert torch.equal(one.layers[-1]._argmax, ref.layers[-1]._argmax)
    dy = torch.randn(a.shape, generator=g, device="cuda")
    for m in (one, ref):                        # the loss layer's gradient is what Model.backward starts from
        m.loss.backward = lambda output, y, m=m: setattr(m.loss, "dinputs", dy)
        m.backward(a, None)
    torch.cuda.synchronize()
    assert one._chains[0].live is None          # it ran, and its state was used up
    for p, q in zip(one.layers[1:], ref.layers[1:]):
        assert torch.equal(p.dinputs, q.dinputs)
    bn, bq = one.layers[0], ref.layers[0]
    for u, v in ((bn.dinputs, bq.dinputs), (bn.dweights, bq.dweights), (bn.dbiases, bq.dbiases)):
        assert O.rel_l2(u.cpu().numpy(), v.cpu().numpy()) <= 1e-5
