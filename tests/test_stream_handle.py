"""The handle of torch's current stream, with and without torch's functions that give it as a
number (no GPU needed)."""
from types import SimpleNamespace

import pytest
import torch


@pytest.mark.parametrize("raw", [True, False])
def test_current_stream_handle(monkeypatch, raw):
    from apbf_gb300 import api

    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: SimpleNamespace(cuda_stream=77))
    monkeypatch.setattr(api, "_raw_device", (lambda: 3) if raw else None)
    monkeypatch.setattr(api, "_raw_stream", (lambda device: 70 + device) if raw else None)
    assert api._stream_handle(None).value == (73 if raw else 77)
    assert api._stream_handle(SimpleNamespace(cuda_stream=5)).value == 5
