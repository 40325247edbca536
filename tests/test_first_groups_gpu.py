"""First layers' forward kernel: the groups of warps that build tiles in turn, at numbers of tiles per CTA that are no multiple of the groups
and at the longest windows (K up to 64).  With and without statistics it is launched with different groups: the outputs are the same bits."""
import numpy as np
import pytest

from oracle import aether_oracle as O

pytestmark = pytest.mark.gpu


# 148 CTAs: (pixels, window) for one tile in some; 1 and 2; 2 and 3; 4 and 5; 3 and 4 tiles each
@pytest.mark.parametrize("H,W,Cin,f", [(30, 31, 3, 3), (137, 139, 3, 3), (195, 195, 1, 7), (275, 276, 1, 3), (240, 239, 2, 5), (138, 138, 4, 4), (300, 260, 3, 4)])
@pytest.mark.parametrize("Cout", [32, 100])
def test_forward(H, W, Cin, f, Cout):
    import torch
    from aether_ml_b200 import _lib, layers
    rng = np.random.default_rng(H)
    x = rng.random((1, H, W, Cin)).astype(np.float32)
    conv = layers.Conv_Layer((H, W, Cin), Cout, (f, f), (1, 1), "same" if f % 2 else "valid", math_mode="bf16")
    b = rng.standard_normal(Cout).astype(np.float32)
    w = conv.filter_weights.cpu().numpy()
    conv.set_parameters(w, b)
    y = conv.forward(x, True)
    conv.emit_bn_stats = True
    with_stats = conv.forward(x, True)
    assert conv.bn_partials is not None and torch.equal(y, with_stats)
    assert O.rel_l2(y.cpu().numpy(), O.conv_forward_blas(x, w, b, (1, 1), conv.padding)) <= 1e-2       # (bf16 operands)
    assert _lib.device_status() == 0
