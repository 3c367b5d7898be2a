"""CPU: the binding takes torch's current stream by its public call where the
raw-handle entry is missing."""
import types

import gbfft
import torch


def test_current_stream_without_the_raw_entry(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=77))
    monkeypatch.setattr(torch, "_C", types.SimpleNamespace())
    assert gbfft._stream(None) == 77
    monkeypatch.setattr(torch, "_C", types.SimpleNamespace(_cuda_getCurrentRawStream=lambda d: 100 + d))
    assert gbfft._stream(None) == 103


def test_given_streams():
    assert gbfft._stream(5) == 5
    assert gbfft._stream(types.SimpleNamespace(cuda_stream=9)) == 9
