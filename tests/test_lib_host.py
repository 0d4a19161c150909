"""Host-side helpers of the call path, with a fake of the CUDA runtime's per-device state."""

import torch

from betterrobot_b200 import _lib


def test_capturing_asks_about_the_given_device(monkeypatch):
    """A plan for one device is laid out while another one is current: the capture state that matters is
    that of the plan's device (a copy that a capture records must not be taken for one that has run)."""
    state = {"current": 0, "captured": {1}}

    class Switch:
        def __init__(self, device):
            self.to = torch.device(device).index

        def __enter__(self):
            self.back, state["current"] = state["current"], self.to

        def __exit__(self, *exc):
            state["current"] = self.back

    monkeypatch.setattr(torch.cuda, "current_device", lambda: state["current"])
    monkeypatch.setattr(torch.cuda, "device", Switch)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["current"] in state["captured"])
    assert _lib.capturing(torch.device("cuda", 1)) and not _lib.capturing(torch.device("cuda", 0))
    state["current"] = 1
    assert _lib.capturing(torch.device("cuda", 1)) and not _lib.capturing(torch.device("cuda", 0))
    assert state["current"] == 1
