"""Workspaces of layers where the memory for the one that is asked for is not there, without a device."""
import pytest


@pytest.fixture
def workspace(monkeypatch):
    """A workspace and the sizes that were allocated or refused for it, on a device with room for 1000 bytes at a time."""
    import torch
    from aether_ml_b200 import layers
    asked = []

    class Host:
        @staticmethod
        def empty_u8(shape):
            asked.append(shape[0])
            if shape[0] > 1000:
                raise torch.OutOfMemoryError("no room")
            return bytearray(shape[0])
    monkeypatch.setattr(layers, "host", lambda: Host)
    return layers._Workspace(), asked


class Plan:
    def __init__(self, least):
        self.least_ws_bytes = lambda: least


def test_the_least_instead(workspace):
    ws, asked = workspace
    buf = ws.get(5000, Plan(600))
    assert ws.buf is buf and len(buf) == ws.size == 600 and asked == [5000, 600]
    assert ws.get(5000, Plan(600)) is buf and ws.get(6000, Plan(300)) is buf and asked == [5000, 600]      # (a refusal is not asked for on every pass)
    assert len(ws.get(7000, Plan(800))) == 800 and asked == [5000, 600, 800]
    assert len(ws.get(900, Plan(600))) == 900 and asked[-1] == 900                             # what there is room for is taken


def test_no_less_to_be_had(workspace):
    import torch
    ws, asked = workspace
    for plan in (None, Plan(5000), Plan(2000)):
        with pytest.raises(torch.OutOfMemoryError):
            ws.get(5000, plan)
    assert ws.buf is None and ws.size == 0
    assert len(ws.get(10)) == 256
