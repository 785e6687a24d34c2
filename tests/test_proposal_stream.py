"""Which stream the proposal calls run on when none is given: torch's current one, by its raw handle where torch
has a name for that."""
from types import SimpleNamespace


def test_current_stream_with_and_without_the_raw_handle(vf, monkeypatch):
    import torch

    from vfwater import proposal

    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: SimpleNamespace(cuda_stream=77))
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 1000 + device, raising=False)
    assert proposal._current_stream() == 1003
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    assert proposal._current_stream() == 77
