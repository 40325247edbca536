"""Up to how many rows the activation behind a Dense layer goes back in one pass with its operand copy and column sums: 384 more
than columns, 1408 at most; one launch less below the line, the same gradients (fp32 sums of dB in another order) on both sides."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns,most", [(32, 416), (128, 512), (260, 644), (1024, 1408), (1100, 1408)])
def test_line(columns, most):
    import torch
    from aether_ml_b200 import _lib, layers as L
    from aether_ml_b200.model import _DenseAct
    launches = []
    for rows in (most, most + 1):
        dense, act = L.Layer_Dense(64, columns), L.ReLU()
        pair = _DenseAct.find([dense, act], 0)
        g = torch.Generator(device="cuda").manual_seed(columns)
        x, dy = torch.randn((rows, 64), generator=g, device="cuda"), torch.randn((rows, columns), generator=g, device="cuda")
        assert pair.forward([dense, act], 0, x, True)
        n0 = _lib.launch_count()
        assert pair.backward([dense, act], 0, dy) == (rows == most)
        if rows > most:
            act.backward(dy)
            dense.backward(act.dinputs)
        launches.append(_lib.launch_count() - n0)
        got = [dense.dinputs.clone(), dense.dweights.clone(), dense.dbiases.clone(), act.dinputs.clone()]
        act.backward(dy)
        dense.backward(act.dinputs)
        for a, b in zip(got, (dense.dinputs, dense.dweights, dense.dbiases, act.dinputs)):
            assert float((a - b).norm() / b.norm()) <= 1e-6
    assert launches[0] < launches[1]
