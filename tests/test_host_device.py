"""Device and stream of an operator call by torch's public names alone, as on a
torch release without the private ones (no device needed)."""

import importlib.util
from types import SimpleNamespace

import torch

from scico_gb300 import _device


def test_public_names_serve_where_the_private_ones_are_gone(monkeypatch):
    for name in ("_cuda_getDevice", "_cuda_getCurrentRawStream"):
        monkeypatch.delattr(torch._C, name, raising=False)
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda index: SimpleNamespace(cuda_stream=70 + index))
    spec = importlib.util.spec_from_file_location("scico_gb300._device_public", _device.__file__)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    assert module.require_cuda() == torch.device("cuda", 3)
    assert module.stream() == 73
