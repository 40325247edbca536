"""A captured train step addresses the layers' workspaces: they stay where they are for as long as the graph exists, also
when a larger batch has since given a layer a larger workspace."""
import weakref

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def captured(X, y):
    from aether_ml_b200 import layers as L
    from aether_ml_b200.model import Accuracy_Categorical, Model
    np.random.seed(5)
    m = Model()
    m.add(L.Conv_Layer((12, 12, 3), 16, (3, 3), (1, 1), "same"))
    m.add(L.Batch_Norm(n_features=16))
    m.add(L.ReLU())
    m.add(L.Pooling((2, 2), (2, 2), "valid", "max"))
    m.add(L.Conv_Layer((6, 6, 16), 32, (3, 3), (1, 1), "same"))
    m.add(L.Batch_Norm(n_features=32))
    m.add(L.ReLU())
    m.add(L.Pooling((2, 2), (2, 2), "valid", "max"))
    m.add(L.Flatten())
    m.add(L.Layer_Dense(3 * 3 * 32, 64))
    m.add(L.ReLU())
    m.add(L.Layer_Dense(64, 10))
    m.add(L.SoftMax())
    m.set(loss=L.Loss_CategoricalCrossEntropy(), optimizer=L.Optimizer_Adam(), accuracy=Accuracy_Categorical())
    m.finalize(flat=True, fuse=True, lean=True)
    m.capture_train_step(X, y)
    return m


def test_replay_after_a_larger_batch():
    import torch
    rng = np.random.default_rng(1)
    X, y = torch.as_tensor(rng.random((16, 12, 12, 3)).astype(np.float32)).cuda(), torch.as_tensor(rng.integers(0, 10, 16)).cuda()
    larger = torch.as_tensor(rng.random((300, 12, 12, 3)).astype(np.float32)).cuda()
    alone, m = captured(X, y), captured(X, y)
    spaces = [w for _, w, buf, _ in m._workspaces() if buf is not None]
    held = [(weakref.ref(w.buf), w.buf.data_ptr(), w.buf.numel()) for w in spaces]
    m.forward(larger, training=False)
    replaced = [(p, n) for (_, p, n), w in zip(held, spaces) if w.buf.data_ptr() != p]
    assert replaced and all(ref() is not None for ref, _, _ in held)
    others = [torch.full((n,), 0x5A, dtype=torch.uint8, device="cuda") for _, n in replaced for _ in range(3)]
    for _ in range(3):
        alone.train_step_graph(X, y)
        m.train_step_graph(X, y)
    torch.cuda.synchronize()
    assert all(bool((o == 0x5A).all()) for o in others)
    assert torch.equal(alone.flat_params, m.flat_params) and torch.equal(alone.flat_grads, m.flat_grads)
    m.release_graphs()
    torch.cuda.synchronize()
    assert m._graph_memory is None and any(ref() is None for ref, _, _ in held)
