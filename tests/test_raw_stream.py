"""The handle of torch's current stream is found with and without torch's private
short cut for it (no GPU needed: torch.cuda.current_stream is a stand-in)."""
import importlib
import types

from conftest import pkg


def test_handle_without_the_private_function(monkeypatch):
    import torch

    pkg()
    spmlutil = importlib.import_module("dennou-ogcm_b200.spmlutil")
    asked = []

    def current_stream(dev):
        asked.append(dev)
        return types.SimpleNamespace(cuda_stream=4711)

    monkeypatch.setattr(torch.cuda, "current_stream", current_stream)
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert spmlutil._raw_stream()(3) == 4711 and asked == [3]
    short = lambda dev: 100 + dev  # noqa: E731
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", short, raising=False)
    assert spmlutil._raw_stream()(3) == 103 and asked == [3]
