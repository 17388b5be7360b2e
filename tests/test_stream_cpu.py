"""The stream a call runs on: the one given, else the current one, also on a torch without the raw handle."""
from types import SimpleNamespace

import torch

from daxtoolkit_gb300 import cont


def test_given_stream(monkeypatch):
    monkeypatch.setattr(cont, "_raw_stream", None)
    assert cont._stream(SimpleNamespace(cuda_stream=17)).value == 17


def test_raw_handle_of_the_current_device(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(cont, "_raw_stream", lambda device: 100 + device)
    assert cont._stream().value == 103
    assert cont._stream(SimpleNamespace(cuda_stream=5)).value == 5


def test_without_the_raw_handle(monkeypatch):
    monkeypatch.setattr(cont, "_raw_stream", None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: SimpleNamespace(cuda_stream=29))
    assert cont._stream().value == 29
