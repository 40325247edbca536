"""Errors of torch inside the native host path arrive as Python exceptions (run in a process of its own: an exception that
leaves a C callback ends the process)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CALLS = {
    "tag of a tensor of inference mode": "with torch.inference_mode():\n    t = torch.zeros(3)\nh.tag(t)",
    "same of a tensor of inference mode": "with torch.inference_mode():\n    t = torch.zeros(3)\nh.same(t, (0, 3, 0, 3))",
    "empty_like of a nested tensor": "h.empty_like(torch.nested.nested_tensor([torch.zeros(2), torch.zeros(3)]))",
    "tag of a sparse tensor": "h.tag(torch.zeros(3, 3).to_sparse())",
    "empty without a device or of too many dimensions": "h.empty((1,) * 9)",
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_exception(name):
    code = ("import sys\nsys.path.insert(0, %r)\nimport torch\nfrom aether_ml_b200._lib import host\nh = host()\n"
            "def call():\n    %s\ntry:\n    call()\nexcept (RuntimeError, TypeError) as e:\n    print('caught', type(e).__name__)\n"
            % (ROOT, CALLS[name].replace("\n", "\n    ")))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("caught"), (r.returncode, r.stdout, r.stderr[-2000:])


@pytest.mark.gpu
def test_layer_under_inference_mode():
    """Arrays of inference mode carry no record of in-place changes, which the operand copies need: refused as an exception."""
    import torch
    from aether_ml_b200 import layers as L
    conv, x = L.Conv_Layer((8, 8, 16), 16), torch.rand(2, 8, 8, 16, device="cuda")
    with torch.inference_mode():
        with pytest.raises(RuntimeError):
            conv.forward(x.clone(), False)
    assert conv.forward(x, False).shape == (2, 8, 8, 16)
    torch.cuda.synchronize()
