"""The update of many tensors in one call against the update of each by itself, bit for bit (the same operations per element):
tensors that share memory, whose updates have to follow each other, and more tensors than one launch takes (32)."""
import pytest

pytestmark = pytest.mark.gpu


def layers(sizes, tie):
    """Objects with what an optimizer needs of a layer; `tie` lists (layer, layer it shares weights and moments with)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    out = []
    for n in sizes:
        l = type("Layer", (), {})()
        for name in ("weights", "dweights", "weight_momentums", "weight_cache"):
            setattr(l, name, torch.rand(n, generator=g, device="cuda"))
        for name in ("biases", "dbiases", "bias_momentums", "bias_cache"):
            setattr(l, name, torch.rand(3 + n % 5, generator=g, device="cuda"))
        out.append(l)
    for a, b, what in tie:
        for name in what:
            setattr(out[a], name, getattr(out[b], name)[:out[a].weights.numel()])
    return out


def both_ways(sizes, tie, steps=3):
    import torch
    from aether_ml_b200.layers import Optimizer_Adam
    res = []
    for together in (True, False):
        ls, opt = layers(sizes, tie), Optimizer_Adam(learning_rate=0.01, decay=1e-3)
        for _ in range(steps):
            opt.pre_update_parameters()
            if together:
                opt.update_layers(ls)
            else:
                for l in ls:
                    opt.update_parameters(l)
            opt.post_update_parameters()
        res.append([getattr(l, n) for l in ls for n in ("weights", "biases", "weight_momentums", "weight_cache", "bias_momentums", "bias_cache")])
    torch.cuda.synchronize()
    return res


@pytest.mark.parametrize("sizes,tie", [((5000, 5000), [(1, 0, ("weights",))]),                              # tied weights, moments of their own
                                       ((5000, 70, 5000), [(2, 0, ("weights", "weight_momentums", "weight_cache"))]),
                                       ((300000, 1000, 40, 250), [(1, 0, ("weights",)), (3, 1, ("weights",))]),    # parts of a larger array
                                       ((4096, 4096), [])])
def test_shared_memory(sizes, tie):
    import torch
    a, b = both_ways(sizes, tie)
    assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("count", [1, 15, 16, 17, 32, 33])                  # two tensors each
def test_more_than_one_launch(count):
    import torch
    from aether_ml_b200 import _lib
    n0 = _lib.launch_count()
    a, b = both_ways([1 + 977 * k for k in range(count)], [], steps=1)
    assert _lib.launch_count() - n0 == -(-2 * count // 32) + 2 * count
    assert all(torch.equal(x, y) for x, y in zip(a, b))
