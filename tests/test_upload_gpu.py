"""Channel masks from the host travel as kernel arguments, 512 values a launch: every value arrives, whatever their number."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 255, 511, 512, 513, 1024, 1537])
def test_mask(C):
    import torch
    from aether_ml_b200 import layers as L
    rng = np.random.default_rng(C)
    drop = L.Layer_Dropout_Spatial(0.25)
    drop.fixed_mask = rng.standard_normal(C).astype(np.float32)
    x = torch.rand((2, 3, 1, C), device="cuda")
    y = drop.forward(x, True)
    want = torch.as_tensor(drop.fixed_mask).cuda()
    assert torch.equal(drop.channel_mask, want.view(1, 1, 1, C)) and torch.equal(y, x * want)
