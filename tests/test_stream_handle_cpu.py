"""Which stream a call is launched on: that of the tensor's device, whatever form the device has."""
import torch

from ojasx_b200 import ops


def test_stream_of_a_device_with_and_without_index(monkeypatch):
    monkeypatch.setattr(ops, "_raw_stream", lambda index: 1000 + index)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    assert ops._stream_ptr(torch.device("cuda", 1)) == 1001
    assert ops._stream_ptr(torch.device("cuda", 0)) == 1000
    assert ops._stream_ptr(torch.device("cuda")) == 1003
