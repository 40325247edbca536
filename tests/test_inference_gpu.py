"""Inference over several batches at once: predictions and accumulated loss / accuracy equal those of the batches one by
one, whatever number of them a pass takes, and the layers are left as the last batch leaves them.  The products are the
same, only their tiles differ: fp32 sums of bf16 products in another order, relative L2 <= 1e-4."""
import numpy as np
import pytest

from oracle import aether_oracle as O

pytestmark = pytest.mark.gpu


def network():
    from aether_ml_b200 import layers as L
    from aether_ml_b200.model import Accuracy_Categorical, Model
    np.random.seed(5)
    m = Model()
    m.add(L.Conv_Layer((9, 8, 3), 16, (3, 3), (1, 1), "same"))
    m.add(L.Batch_Norm(n_features=16))
    m.add(L.ReLU())
    m.add(L.Layer_Dropout_Spatial(0.2))
    m.add(L.Conv_Layer((9, 8, 16), 32, (3, 3), (1, 1), "valid"))
    m.add(L.Batch_Norm(n_features=32))
    m.add(L.Leaky_ReLU(0.01))
    m.add(L.Pooling((2, 2), (2, 2), "valid", "max"))
    m.add(L.Flatten())
    m.add(L.Layer_Dense(3 * 3 * 32, 10))
    m.add(L.SoftMax())
    m.set(loss=L.Loss_CategoricalCrossEntropy(label_smoothing=0.01), optimizer=L.Optimizer_Adam(), accuracy=Accuracy_Categorical())
    m.finalize()
    return m


@pytest.mark.parametrize("batch,images,limit", [(7, 61, None), (7, 61, 1), (7, 61, 400000), (16, 33, None), (16, 32, None), (16, 9, None), (None, 20, None)])
def test_batches_at_once(batch, images, limit):
    import torch
    m = network()
    if limit is not None:
        m.INFERENCE_PASS_BYTES = limit
    rng = np.random.default_rng(images)
    X = rng.random((images, 9, 8, 3)).astype(np.float32)
    y = rng.integers(0, 10, images)
    got = m.predict(X, batch_size=batch)
    last = [(l.output, getattr(l, "inputs", None)) for l in m.layers]
    step = batch or images
    outs = [m.forward(X[k:k + step], training=False).clone() for k in range(0, images, step)]
    assert O.rel_l2(got.cpu().numpy(), torch.vstack(outs).cpu().numpy()) <= 1e-4
    for (out, inp), l in zip(last, m.layers):
        assert O.rel_l2(out.cpu().numpy(), l.output.cpu().numpy()) <= 1e-4
        assert inp is None or O.rel_l2(inp.cpu().numpy(), l.inputs.cpu().numpy()) <= 1e-4
    acc, loss = m.evaluate(X, y, batch_size=batch)
    m.loss.new_pass()
    m.accuracy.new_pass()
    for k, out in enumerate(outs):
        m.loss.calculate(out, y[k * step:(k + 1) * step], training=False)
        m.accuracy.calculate(m.output_layer_activation.predictions(out), y[k * step:(k + 1) * step])
    assert abs(float(m.loss.calculate_accumulated()) - loss) <= 1e-4 * abs(loss)
    assert float(m.accuracy.calculate_accumulated()) == acc
